"""The contracted per-source kernel's rows by length -- a thread's, a warp's, the
whole CTA's, and more of either on one level than its queues hold -- on BCCs with
enough chains to be contracted. Which of a level's long rows come first depends on
timing, BC must not: runs give the same bits, with and without a rescale forced
on almost every level, and the oracle's BC."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def with_chains(n, u, v, ends, count, length, seed):
    """`count` chains of `length` between random vertices of `ends`, and leaves."""
    rng = np.random.default_rng(seed)
    us, vs = [u], [v]
    for _ in range(count):
        a, b = rng.choice(ends, 2, replace=False)
        path = np.concatenate([[a], n + np.arange(length), [b]])
        us.append(path[:-1])
        vs.append(path[1:])
        n += length
    us.append(rng.integers(0, n, 300))
    vs.append(n + np.arange(300))
    n += 300
    return (n,) + graphs().simple_edges(n, np.concatenate(us), np.concatenate(vs))


def many_hubs(hubs, others, seed):
    """Hubs over random subsets of 1,050-1,400 of the same vertices: from a hub, all
    other hubs are on level 2."""
    rng = np.random.default_rng(seed)
    u, v = [], []
    for h in range(hubs):
        k = int(rng.integers(1050, 1400))
        u.append(np.full(k, h))
        v.append(hubs + rng.permutation(others)[:k])
    n = hubs + others
    return with_chains(n, np.concatenate(u), np.concatenate(v), np.arange(hubs, n), 500, 3, seed)


def two_hubs():
    """Two hubs over the same 2,300 vertices, which form a ring, and a clique of 60."""
    ring = np.arange(2, 2302)
    cl = np.arange(2302, 2362)
    cu, cv = np.triu_indices(60, 1)
    u = np.concatenate([np.zeros(2300, int), np.ones(2300, int), ring, cl[cu], ring[:60]])
    v = np.concatenate([ring, ring, np.roll(ring, 1), cl[cv], cl])
    return with_chains(2362, u, v, np.arange(2362), 500, 4, 3)


def wide_level():
    """700 vertices of degree 12 and more on one level."""
    mid = np.arange(1, 701)
    u = np.concatenate([np.zeros(700, int)] + [mid] * 11)
    v = np.concatenate([mid] + [1 + (mid + 13 * j) % 700 for j in range(11)])
    return with_chains(701, u, v, np.arange(701), 150, 4, 4)


CASES = {"many-hubs": lambda: many_hubs(99, 2400, 11), "two-hubs": two_hubs, "wide-level": wide_level}


@pytest.mark.parametrize("name,ctas", [(name, ctas) for name in CASES for ctas in (0, 4, 16)])
def test_same_bits_on_every_run(name, ctas):
    P = pkg()
    n, u, v = CASES[name]()
    O = oracle()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    outs = []
    for rescale in (0, 2):
        ctx = P.Context(mode=P.MODE_BATCHED, plain_core=1 << 30, tile_max=-1, plain_ctas_per_sm=ctas,
                        rescale_exp=rescale)
        plan = ctx.plan(d)
        for _ in range(5):
            plan.reset()
            st = plan.run()
            assert st["bfs_sources"] == st["sources"]  # none is merged: the contracted kernel's
            outs.append(plan.read())
        plan.close()
        ctx.close()
    assert all(np.array_equal(x, outs[0]) for x in outs)
    assert rel_err(outs[0], O.brandes(n, *O.csr(n, u, v))) < TOL
