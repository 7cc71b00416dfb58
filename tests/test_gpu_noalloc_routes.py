"""bc_begin_free_noalloc over the sizes that change its kernel: the small-BCC
classes, BCCs beyond shared memory (per-source kernel, its fixed array shared by
as many rows as fit), BCCs too deep for the small-BCC kernels' level tables and
with path counts past 2^1000 (run again on the per-source kernel), each against
the oracle, one after another on one device so that every change of layout is
met; and malformed input on both routes."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def chorded(n, chords, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    return (n,) + graphs().simple_edges(n, np.concatenate([i, rng.integers(0, n, chords)]),
                                        np.concatenate([(i + 1) % n, rng.integers(0, n, chords)]))


def ladder(rungs):
    i = np.arange(rungs)
    return (2 * rungs,) + graphs().simple_edges(2 * rungs, np.concatenate([i[:-1], rungs + i[:-1], i]),
                                                np.concatenate([i[1:], rungs + i[1:], rungs + i]))


def layered(width, layers):
    """Complete bipartite layers in a row: width^l shortest paths on level l."""
    a, b = np.meshgrid(np.arange(width), np.arange(width))
    u = np.concatenate([width * l + a.ravel() for l in range(layers - 1)])
    v = np.concatenate([width * (l + 1) + b.ravel() for l in range(layers - 1)])
    return (width * layers,) + graphs().simple_edges(width * layers, u, v)


CASES = [
    ("triangle", lambda: chorded(3, 0, 1), 3),
    ("warp class", lambda: chorded(640, 700, 2), 640),
    ("beyond shared memory", lambda: chorded(14000, 9000, 3), 40),
    ("cta class", lambda: chorded(641, 700, 4), 300),
    ("largest", lambda: chorded(16384, 3000, 5), 20),
    ("groups of four", lambda: chorded(2900, 5000, 6), 64),
    ("past the level tables", lambda: ladder(1100), 48),
    ("one cta per SM", lambda: chorded(8500, 4000, 7), 40),
    ("past the groups' level tables", lambda: ladder(700), 48),
    ("counts past 2^1000", lambda: layered(11, 292), 64),
    ("two groups", lambda: chorded(5200, 6000, 8), 40),
]


def call(P, ctx, dev, n, m, nsrc, out):
    import torch

    torch.cuda.synchronize()
    return P.begin_gpu_free_noalloc(ctx, dev[0].data_ptr(), dev[1].data_ptr(), n, m, dev[2].data_ptr(), nsrc,
                                    dev[3].data_ptr(), out.data_ptr())


def test_every_route_gives_the_oracles_bc():
    import torch

    P = pkg()
    ctx = P.Context(mode=P.MODE_PLAIN)
    for seed, (name, make, nsrc) in enumerate(CASES):
        d = P.Decomposition(P.Graph.from_edges(*make()))
        a = d.arrays()
        n = int(a["vtx_off"][1])
        assert a["n_bcc"] == 1, name
        src = np.random.default_rng(seed).permutation(n)[:nsrc].astype(np.int32)
        arrs = [a["row"].astype(np.int32), a["col"].astype(np.int32), src, a["reach"].astype(np.int32)]
        dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in arrs]
        outs = []
        for _ in range(2):
            out = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
            call(P, ctx, dev, n, len(arrs[1]), nsrc, out)
            outs.append(out.cpu().numpy())
        assert np.array_equal(outs[0], outs[1]), name
        assert rel_err(outs[0], oracle().bcc_sources(a, 0, src)) < TOL, name
    ctx.close()


@pytest.mark.parametrize("n", [100, 2000, 12000])
def test_malformed_input_is_refused(n):
    import torch

    P = pkg()
    ctx = P.Context(mode=P.MODE_PLAIN)
    d = P.Decomposition(P.Graph.from_edges(*chorded(n, 2 * n // 3, 9)))
    a = d.arrays()
    good = [a["row"].astype(np.int32), a["col"].astype(np.int32), np.arange(8, dtype=np.int32), a["reach"].astype(np.int32)]
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    for which, at, value in ((0, 5, 1 << 29), (1, 7, n), (1, 7, -1), (2, 3, n), (2, 3, -1)):
        bad = [x.copy() for x in good]
        bad[which][at] = value
        dev = [torch.from_numpy(x).cuda() for x in bad]
        with pytest.raises(P.BcError) as e:
            call(P, ctx, dev, n, len(good[1]), 8, out)
        assert e.value.code == P.EINVAL and "malformed" in str(e.value)
    dev = [torch.from_numpy(x).cuda() for x in good]  # and the next call is served
    call(P, ctx, dev, n, len(good[1]), 8, out)
    assert rel_err(out.cpu().numpy(), oracle().bcc_sources(a, 0, good[2])) < TOL
    ctx.close()
