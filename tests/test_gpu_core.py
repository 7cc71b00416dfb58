"""The contracted per-source kernel (every BCC that neither multi-source passes
nor shared memory take): BC against the oracle's Brandes on shapes that reach
its edges -- chains of every length up to its ring's limit and past it, chains
with reach, chains meeting on a vertex and between two, parallel chains, rows
handled by a thread, a warp and the whole CTA, more long rows on a level than
its queue holds, every CTA size -- and bit-identical BC under a rescale forced
on almost every level."""
import numpy as np
import pytest

from helpers import GOLDEN_CASES, graphs, load_case, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def subdivided(n, u, v, lengths, leaves, seed):
    """The first len(lengths) edges (in random order) become chains of those
    lengths; leaves hang off random vertices, chain vertices among them."""
    G = graphs()
    rng = np.random.default_rng(seed)
    order = rng.permutation(len(u))
    u, v = np.asarray(u)[order].astype(np.int64), np.asarray(v)[order].astype(np.int64)
    eu, ev = [u[len(lengths):]], [v[len(lengths):]]
    for a, b, k in zip(u, v, lengths):
        path = np.concatenate([[a], np.arange(n, n + k), [b]])
        eu.append(path[:-1])
        ev.append(path[1:])
        n += int(k)
    at = rng.integers(0, n, leaves)
    eu.append(at)
    ev.append(n + np.arange(leaves))
    n += leaves
    return (n,) + G.simple_edges(n, np.concatenate(eu), np.concatenate(ev))


def random_core(n, m, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    return graphs().simple_edges(n, np.concatenate([i, rng.integers(0, n, m)]), np.concatenate([(i + 1) % n, rng.integers(0, n, m)]))


def hubs():
    """Two hubs over the same 2,300 vertices (rows for the whole CTA), a clique
    (long rows, all on one level), chains between hub and clique."""
    G = graphs()
    ring = np.arange(2, 2302)
    cl = np.arange(2302, 2362)
    cu, cv = np.triu_indices(60, 1)
    u = np.concatenate([np.zeros(2300, int), np.ones(2300, int), ring, cl[cu], ring[:60]])
    v = np.concatenate([ring, ring, np.roll(ring, 1), cl[cv], cl])
    u, v = G.simple_edges(2362, u, v)
    return subdivided(2362, u, v, [1, 2, 3, 4, 5] * 40, 30, 3)


def wide_level():
    """700 vertices of degree 12 on one level: more than the queue of long rows holds."""
    G = graphs()
    mid = np.arange(1, 701)
    u = np.concatenate([np.zeros(700, int)] + [mid] * 11)
    v = np.concatenate([mid] + [1 + (mid + 13 * j) % 700 for j in range(11)])
    return (701,) + G.simple_edges(701, u, v)


CASES = {
    "lengths": lambda: subdivided(60, *random_core(60, 60, 1), list(range(1, 62)), 0, 1),
    "lengths-reach": lambda: subdivided(60, *random_core(60, 60, 2), list(range(1, 62)), 400, 2),
    "past-ring": lambda: subdivided(40, *random_core(40, 30, 3), [62, 61, 5], 20, 3),
    "single-chains": lambda: subdivided(300, *random_core(300, 200, 4), [1] * 200, 50, 4),
    "parallel": lambda: (lambda n, u, v: (n, u, v))(*subdivided(
        4, np.array([0, 1, 2, 3, 0, 1]), np.array([1, 2, 3, 0, 2, 3]), [3, 4, 5, 6, 7, 8], 10, 5)),
    "no-chains": lambda: (257,) + random_core(257, 600, 6),
    "hubs": hubs,
    "wide-level": wide_level,
    "grid": lambda: graphs().gen_grid(40, leaves=200, seed=2),
    "rmat": lambda: graphs().gen_rmat(10, 16, chain_frac=0.3, chain_hi=8, seed=7),
    "ba": lambda: graphs().pack_graphs(graphs().gen_ba_batch(8, 30, 1500, seed=9))[:3],
}
CASES.update({name: (lambda name=name: load_case(name)[:3]) for name in GOLDEN_CASES})


def run(n, u, v, **opts):
    P = pkg()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=1 << 30, tile_max=-1, **opts)
    bc, st = ctx.run(d)
    ctx.close()
    return bc, st


@pytest.mark.parametrize("name", list(CASES))
def test_bc_and_forced_rescaling(name):
    n, u, v = CASES[name]()
    O = oracle()
    row, col = O.csr(n, u, v)
    bc, _ = run(n, u, v)
    assert rel_err(bc, O.brandes(n, row, col)) < TOL
    forced, _ = run(n, u, v, rescale_exp=2)
    assert np.array_equal(bc, forced)


@pytest.mark.parametrize("ctas", [4, 8, 16])
def test_cta_sizes_give_the_oracles_bc(ctas):
    n, u, v = CASES["lengths-reach"]()
    O = oracle()
    row, col = O.csr(n, u, v)
    bc, _ = run(n, u, v, plain_ctas_per_sm=ctas)
    assert rel_err(bc, O.brandes(n, row, col)) < TOL


def test_ranges_add_up():
    """Any split of the units gives the whole run's BC to rounding, and the
    same split the same bits twice."""
    P = pkg()
    n, u, v = CASES["rmat"]()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=1 << 30, tile_max=-1)
    plan = ctx.plan(d)
    k = plan.n_units
    outs = []
    for cuts in ([0, k], [0, 1, k // 3, k - 1, k], [0, 1, k // 3, k - 1, k]):
        plan.reset()
        for a, b in zip(cuts, cuts[1:]):
            plan.run(a, b)
        outs.append(plan.read())
    plan.close()
    ctx.close()
    assert np.array_equal(outs[1], outs[2])
    assert rel_err(outs[1], outs[0]) < TOL
