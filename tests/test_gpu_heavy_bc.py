"""Multi-source passes over rows around the lengths at which they are split over
CTAs: 1,024 arcs, and 2,048 where at least 4,096 rows lie between the two. Levels
and path counts of a pass against the oracle's bit for bit, BC of its sources."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

CORE = 24000


def many_rows(count):
    """`count` rows of 1,025 to 1,100 arcs, and a few around and past 2,048."""
    rng = np.random.default_rng(count)
    ids = np.arange(CORE)
    u, v = [ids], [(ids + 1) % CORE]
    lengths = [1000, 1024, 2047, 2048, 2049, 5000] + list(rng.integers(1025, 1101, count - 2))
    for k, deg in enumerate(lengths):  # every second vertex of the ring a hub
        u.append(np.full(deg - 2, 2 * k))
        v.append(2 * len(lengths) + rng.choice(CORE - 2 * len(lengths), deg - 2, replace=False))
    return (CORE,) + graphs().simple_edges(CORE, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("count", [4095, 4096])
def test_rows_and_bc_of_a_pass(count):
    P = pkg()
    d = P.Decomposition(P.Graph.from_edges(*many_rows(count)))
    a = d.arrays()
    deg = np.diff(a["row"])
    assert a["n_bcc"] == 1 and a["n_plain"][0] >= 16384 and int(((deg > 1024) & (deg <= 2048)).sum()) == count
    for delta, tol in ((P.DELTA_FP64, 1e-12), (P.DELTA_FP32C, 1e-6)):
        ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, batch_width=32, delta=delta)
        plan = ctx.plan(d)
        k = plan.n_units // 2
        src, dd, ss = plan.pass_rows(k)  # runs the pass
        for i in (0, len(src) - 1):
            do, so = oracle().bcc_source_rows(a, 0, int(src[i]))
            assert np.array_equal(dd[i], do[:dd.shape[1]]) and np.array_equal(ss[i], so[:dd.shape[1]])
        got = plan.read()[a["orig"]]
        assert rel_err(got, oracle().bcc_sources(a, 0, plan.unit_sources(k, k + 1).astype(np.int32))) < tol
        plan.close()
        ctx.close()
