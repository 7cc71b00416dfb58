"""Multi-source passes where chains decide the result: lengths below, at and above
what a warp keeps in registers (8), leaves on chain vertices or none, two ends that
tie or that the chain connects, sources on every chain, slots that do not fill a
lane's two or four, and level exponents; whole BC against the oracle."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu


def chained(core, lengths, leaves, seed):
    """A cycle of `core` vertices with chords, some chords with chains of the given
    lengths in turn, and leaves on every third chain vertex."""
    rng = np.random.default_rng(seed)
    u = [np.arange(core), rng.integers(0, core, core)]
    v = [(np.arange(core) + 1) % core, rng.integers(0, core, core)]
    n = core
    for i in range(core // 2):
        k = lengths[i % len(lengths)]
        a = int(rng.integers(0, core))
        b = (a + 1 + int(rng.integers(0, core - 1))) % core
        path = np.r_[a, np.arange(n, n + k), b]
        n += k
        u.append(path[:-1])
        v.append(path[1:])
        if leaves:
            hang = path[1:-1:3]
            u.append(hang)
            v.append(np.arange(n, n + len(hang)))
            n += len(hang)
    u, v = graphs().simple_edges(n, np.concatenate(u), np.concatenate(v))
    return n, u, v


@pytest.mark.parametrize("rescale", [0, 1])
@pytest.mark.parametrize("width,delta", [(96, "fp64"), (128, "fp64"), (160, "fp32c"), (256, "fp32c")])
@pytest.mark.parametrize("core,lengths,leaves", [(40, [1], False), (61, [1, 2, 3, 4], True), (90, [7, 8, 9], False),
                                                 (50, [8, 9, 20, 1], True)])
def test_chain_dependencies(core, lengths, leaves, width, delta, rescale):
    P, O = pkg(), oracle()
    n, u, v = chained(core, lengths, leaves, core + width)
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, batch_width=width, rescale_exp=rescale,
                    delta=P.DELTA_FP64 if delta == "fp64" else P.DELTA_FP32C)
    bc, _ = ctx.run(P.Decomposition(P.Graph.from_edges(n, u, v)))
    row, col = O.csr(n, u, v)
    assert rel_err(bc, O.brandes(n, row, col)) < (1e-12 if delta == "fp64" else 1e-6)
    ctx.close()
