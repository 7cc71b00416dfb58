"""The contracted per-source kernel with more rows for the whole CTA on one
level than it takes that way (rows of over 1,024 arcs, over 64 of them): which
ones a warp sums instead depends on the order in which they were queued, BC must
not. Runs give the same bits, with and without a rescale forced on almost every
level, and the oracle's BC."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def many_hubs(hubs, others, seed):
    """Hubs over random subsets of 1,050-1,400 of the same vertices, leaves on
    random vertices: from a hub, all other hubs are on level 2."""
    rng = np.random.default_rng(seed)
    u, v = [], []
    for h in range(hubs):
        k = int(rng.integers(1050, 1400))
        u.append(np.full(k, h))
        v.append(hubs + rng.permutation(others)[:k])
    n, leaves = hubs + others, 500
    u.append(rng.integers(0, n, leaves))
    v.append(n + np.arange(leaves))
    return (n + leaves,) + graphs().simple_edges(n + leaves, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("ctas", [0, 4, 16])
def test_same_bits_on_every_run(ctas):
    P = pkg()
    n, u, v = many_hubs(99, 2400, 11)
    O = oracle()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    outs = []
    for rescale in (0, 2):
        ctx = P.Context(mode=P.MODE_BATCHED, plain_core=1 << 30, tile_max=-1, plain_ctas_per_sm=ctas,
                        rescale_exp=rescale)
        plan = ctx.plan(d)
        for _ in range(5):
            plan.reset()
            plan.run()
            outs.append(plan.read())
        plan.close()
        ctx.close()
    assert all(np.array_equal(x, outs[0]) for x in outs)
    assert rel_err(outs[0], O.brandes(n, *O.csr(n, u, v))) < TOL
