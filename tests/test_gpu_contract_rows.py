"""Contracted rows of the multi-source passes: hub rows at the edges of a warp's
strip (31 to 65 arcs), all unit arcs, all chain arcs, or the two mixed in an order
that alternates, against the oracle."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deg", [31, 32, 33, 64, 65])
@pytest.mark.parametrize("every", [1, 2, 0])  # each, every second, no arc of the hub enters a chain
def test_hub_rows(deg, every):
    P, G = pkg(), graphs()
    u, v, n = [], [], 1 + 2 * deg
    rim = 1 + np.arange(deg)  # a wheel whose rim vertices are doubled by a second ring: all of degree >= 3
    for j in range(deg):
        nxt = (j + 1) % deg
        u += [rim[j], rim[j], rim[j] + deg]
        v += [rim[nxt], rim[j] + deg, rim[nxt] + deg]
        if every and j % every == 0:  # a spoke of two inner vertices
            u += [0, n, n + 1]
            v += [n, n + 1, rim[j]]
            n += 2
        else:
            u.append(0)
            v.append(rim[j])
    u, v = G.simple_edges(n, np.array(u), np.array(v))
    perm = np.random.default_rng(deg).permutation(n)  # unit and chain neighbours interleave in the hub's row
    u, v = G.simple_edges(n, perm[u], perm[v])
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, delta=P.DELTA_FP64)
    bc, _ = ctx.run(P.Decomposition(P.Graph.from_edges(n, u, v)))
    ctx.close()
    row, col = oracle().csr(n, u, v)
    assert rel_err(bc, oracle().brandes(n, row, col)) < 1e-12
