"""Backward sweep of multi-source passes over rows around the lengths at which they
are split over CTAs (1,024 arcs; 2,048 from cores of 2^18 vertices on): BC of a
pass's sources against the oracle's."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delta,tol", [("fp64", 1e-12), ("fp32c", 1e-6)])
@pytest.mark.parametrize("core", [(1 << 18) - 1, 1 << 18])
def test_bc_of_a_pass(core, delta, tol):
    P, G = pkg(), graphs()
    rng = np.random.default_rng(core)
    ids = np.arange(core)
    u, v = [ids, ids], [(ids + 1) % core, rng.integers(0, core, core)]
    for hub, deg in enumerate([1000, 1024, 1025, 2000, 2048, 2049, 5000]):
        u.append(np.full(deg - 2, hub * 1000))
        v.append(rng.choice(core, deg - 2, replace=False))
    u, v = G.simple_edges(core, np.concatenate(u), np.concatenate(v))
    d = P.Decomposition(P.Graph.from_edges(core, u, v))
    a = d.arrays()
    assert a["n_bcc"] == 1
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, batch_width=32,
                    delta=P.DELTA_FP64 if delta == "fp64" else P.DELTA_FP32C)
    plan = ctx.plan(d)
    k = plan.n_units // 2
    plan.run(k, k + 1)
    got = plan.read()[a["orig"]]
    want = oracle().bcc_sources(a, 0, plan.unit_sources(k, k + 1).astype(np.int32))
    assert rel_err(got, want) < tol
    plan.close()
    ctx.close()
