"""bc_begin_free_noalloc on each class of the small-BCC kernels that it picks, at
the sizes where one gives way to the next, against the oracle."""
import ctypes as C

import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

TOL = 1e-12
SMEM = 227 * 1024

# vertices, chords, class: 8, 7, 6 eight groups of 32, 64, 128 threads; 1, 2, 3 one
# source per 256, 512, 1,024 threads; 5, 4 four, two groups; -1 no class
CASES = [(3, 0, 8), (640, 700, 8), (641, 700, 7), (1200, 20, 7), (1201, 20, 6), (2200, 20, 1), (1900, 2500, 6),
         (3500, 4500, 5), (4900, 5000, 4), (8500, 4000, 3), (16384, 3000, -1)]


def pad16(x):
    return (x + 15) // 16 * 16


def class_of(n, arcs):
    f = pkg().lib()._ZN3bcg10tile_classEllm
    f.argtypes = [C.c_int64, C.c_int64, C.c_size_t]
    pairs = (arcs + n + 1) // 2
    return f(n, pad16((2 if pairs < 65536 else 4) * (n + 1)) + pad16(4 * pairs), SMEM)


def chorded(n, chords):
    rng = np.random.default_rng(n + chords)
    i = np.arange(n)
    return (n,) + graphs().simple_edges(n, np.concatenate([i, rng.integers(0, n, chords)]),
                                        np.concatenate([(i + 1) % n, rng.integers(0, n, chords)]))


def bcc(n, chords):
    P = pkg()
    a = P.Decomposition(P.Graph.from_edges(*chorded(n, chords))).arrays()
    assert a["n_bcc"] == 1
    return a


@pytest.mark.parametrize("n,chords,cls", CASES)
def test_class(n, chords, cls):
    assert class_of(n, len(bcc(n, chords)["col"])) == cls


def test_no_graph_takes_the_warp_class():
    """Any number of arcs that a simple graph of up to 640 vertices can have."""
    for n in list(range(3, 120)) + list(range(120, 641, 13)) + [640]:
        for arcs in np.linspace(2 * n, n * (n - 1), 60).astype(int):
            assert class_of(n, int(arcs)) != 0, (n, arcs)


@pytest.mark.gpu
@pytest.mark.parametrize("n,chords,cls", CASES)
def test_bc_of_every_class(n, chords, cls):
    import torch

    P = pkg()
    a = bcc(n, chords)
    src = np.random.default_rng(n).permutation(n)[:40].astype(np.int32)
    arrs = [a["row"].astype(np.int32), a["col"].astype(np.int32), src, a["reach"].astype(np.int32)]
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in arrs]
    out = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
    ctx = P.Context(mode=P.MODE_PLAIN)
    torch.cuda.synchronize()
    P.begin_gpu_free_noalloc(ctx, dev[0].data_ptr(), dev[1].data_ptr(), n, len(arrs[1]), dev[2].data_ptr(), len(src),
                             dev[3].data_ptr(), out.data_ptr())
    assert rel_err(out.cpu().numpy(), oracle().bcc_sources(a, 0, src)) < TOL
    ctx.close()
