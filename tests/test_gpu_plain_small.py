"""PLAIN plans whose BCCs fit shared memory run them on the small-BCC kernels:
whole runs against the oracle, unit ranges against the contracted per-source
kernel (a BATCHED plan without small-BCC items has the same units), over the
classes of those kernels and the edges of their queues, level tables and slice
forms; the same bits again on a second run."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def cycle_with_chords(n, chords, seed):
    """A cycle of n vertices plus random chords: one BCC."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    u = np.concatenate([i, rng.integers(0, n, chords)])
    v = np.concatenate([(i + 1) % n, rng.integers(0, n, chords)])
    return (n,) + graphs().simple_edges(n, u, v)


def ladder(rungs):
    i = np.arange(rungs)
    return (2 * rungs,) + graphs().simple_edges(2 * rungs, np.concatenate([i[:-1], rungs + i[:-1], i]),
                                                np.concatenate([i[1:], rungs + i[1:], rungs + i]))


def star_and_grid():
    """A hub row far longer than a warp next to a BCC of many levels (too deep
    for the classes with short level tables) and one-cycle BCCs."""
    G = graphs()
    hub = np.arange(1, 400)
    wheel = (400,) + G.simple_edges(400, np.concatenate([np.zeros(399, int), hub]),
                                    np.concatenate([hub, np.roll(hub, 1)]))
    ring = (700,) + G.simple_edges(700, np.arange(700), (np.arange(700) + 1) % 700)
    return G.pack_graphs([wheel, ring, ladder(600), (3,) + G.simple_edges(3, [0, 1, 2], [1, 2, 0])])[:3]


CASES = {
    "triangle": lambda: cycle_with_chords(3, 0, 1),
    "warp-class": lambda: cycle_with_chords(640, 500, 2),
    "cta-class": lambda: cycle_with_chords(641, 500, 3),
    "wide-rows": lambda: cycle_with_chords(300, 12000, 4),
    "int32-offsets": lambda: cycle_with_chords(800, 40000, 5),
    "groups-of-64": lambda: cycle_with_chords(1200, 1500, 9),
    "groups-of-128": lambda: cycle_with_chords(1201, 1500, 10),
    "deep-small": lambda: ladder(300),
    "mid": lambda: cycle_with_chords(2900, 5000, 6),
    "large": lambda: cycle_with_chords(6500, 9000, 7),
    "too-large": lambda: cycle_with_chords(17000, 6000, 8),
    "shapes": star_and_grid,
    "ba": lambda: graphs().pack_graphs(graphs().gen_ba_batch(10, 30, 3000, seed=5))[:3],
}


@pytest.mark.parametrize("name", list(CASES))
def test_plain_routes(name):
    P = pkg()
    n, u, v = CASES[name]()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    got = []
    for opts in (dict(mode=P.MODE_PLAIN), dict(mode=P.MODE_BATCHED, plain_core=1 << 30, tile_max=-1), dict(mode=P.MODE_PLAIN)):
        ctx = P.Context(**opts)
        plan = ctx.plan(d)
        k = plan.n_units
        parts = [(0, min(k, 600))] if name == "too-large" else [(0, k), (k // 3, 2 * k // 3), (k - 1, k), (0, 0)]
        got.append([])
        for a, b in parts:
            plan.reset()
            plan.run(a, b)
            got[-1].append(plan.read())
        plan.close()
        ctx.close()
    for x, y, z in zip(*got):
        assert np.array_equal(x, z)
        assert rel_err(x, y) < TOL
    if name != "too-large":
        O = oracle()
        row, col = O.csr(n, u, v)
        assert rel_err(got[0][0], O.brandes(n, row, col)) < TOL


@pytest.mark.parametrize("repeat", [1, 3])
def test_begin_free_repeated_and_partial_sources(repeat):
    """Sources in any order, some of them several times: each occurrence counts."""
    P = pkg()
    n, u, v = cycle_with_chords(900, 900, 11)
    row, col = oracle().csr(n, u, v)
    R, Cc = row.astype(np.int32), col.astype(np.int32)
    rng = np.random.default_rng(3)
    reach = rng.integers(0, 4, n).astype(np.int32)
    src = np.repeat(rng.permutation(n)[:133], repeat).astype(np.int32)
    out = []
    for rx in (0, 900):
        ctx = P.Context(mode=P.MODE_PLAIN, rescale_exp=rx)
        bc = np.full(n, -1.0, dtype=np.float32)
        P.begin_gpu_free(ctx, R, Cc, n, len(Cc), src, reach, bc)
        out.append(bc)
        ctx.close()
    assert np.array_equal(out[0], out[1])


def test_inputs_the_bounds_do_not_cover_stay_per_source():
    """A CSR whose arcs are not mirrored (a path count of zero, refused as out
    of range), and one that is not connected, take the per-source kernel and
    end as they did."""
    P = pkg()
    n = 700
    i = np.arange(n)
    oneway = (np.concatenate([[0], 2 * (i + 1)]).astype(np.int32), np.stack([(i + 1) % n, (i + 7) % n], 1).ravel().astype(np.int32))
    two = (np.concatenate([[0], 2 * (i + 1)]).astype(np.int32),
           np.stack([np.where(i < 350, (i + 1) % 350, 350 + (i - 349) % 350),
                     np.where(i < 350, (i - 1) % 350, 350 + (i - 351) % 350)], 1).ravel().astype(np.int32))
    src = np.arange(0, n, 9, dtype=np.int32)
    reach = np.zeros(n, np.int32)
    for R, Cc, code in ((*oneway, P.EOVERFLOW), (*two, P.OK)):
        out = []
        for rx in (0, 900):
            ctx = P.Context(mode=P.MODE_PLAIN, rescale_exp=rx)
            bc = np.zeros(n, dtype=np.float32)
            try:
                P.begin_gpu_free(ctx, R, Cc, n, len(Cc), src, reach, bc)
                assert code == P.OK and bc.max() > 0
            except P.BcError as e:
                assert e.code == code
            out.append(bc)
            ctx.close()
        assert np.array_equal(out[0], out[1])
