"""Rows around the lengths at which a multi-source pass splits a row over CTAs, on
cores just below and at the size where that length changes: the rows of a pass
against the oracle's, bit for bit."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core", [(1 << 18) - 1, 1 << 18])
def test_hub_rows_bit_exact(core):
    P, G = pkg(), graphs()
    rng = np.random.default_rng(core)
    ids = np.arange(core)
    u, v = [ids, ids], [(ids + 1) % core, rng.integers(0, core, core)]
    for hub, deg in enumerate([1000, 1024, 1025, 2000, 2048, 2049, 5000]):
        u.append(np.full(deg - 2, hub * 1000))
        v.append(rng.choice(core, deg - 2, replace=False))
    u, v = G.simple_edges(core, np.concatenate(u), np.concatenate(v))
    d = P.Decomposition(P.Graph.from_edges(core, u, v))
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, batch_width=32, delta=P.DELTA_FP64)
    plan = ctx.plan(d)
    src, dd, ss = plan.pass_rows(plan.n_units // 2)
    a = d.arrays()
    for i in (0, len(src) - 1):
        do, so = oracle().bcc_source_rows(a, 0, int(src[i]))
        nc = dd.shape[1]
        assert np.array_equal(dd[i], do[:nc]) and np.array_equal(ss[i], so[:nc])
    plan.close()
    ctx.close()
