"""The read-back of a plan adds a vertex's terms (one per BCC it is in) in packed
order, whatever the number of host threads: the same bits for every team, below
and above the size from which a team is used, and the closed form of a chain of
triangles."""
import ctypes

import numpy as np
import pytest

from helpers import graphs, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("triangles", [1, 2, 16383, 16384, 20000])
def test_teams_agree(triangles):
    P = pkg()
    n = 2 * triangles + 1  # triangles (2i, 2i + 1, 2i + 2), each sharing a vertex with the next
    i = 2 * np.arange(triangles)
    u, v = graphs().simple_edges(n, np.concatenate([i, i, i + 1]), np.concatenate([i + 1, i + 2, i + 2]))
    gomp = ctypes.CDLL("libgomp.so.1")
    had = gomp.omp_get_max_threads()
    ctx = P.Context(mode=P.MODE_BATCHED, delta=P.DELTA_FP64)
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    out = []
    for team in (1, 3, 7):
        gomp.omp_set_num_threads(team)
        out.append(ctx.run(d)[0].copy())
    gomp.omp_set_num_threads(had)
    ctx.close()
    assert all(x.tobytes() == out[0].tobytes() for x in out)
    want = np.zeros(n)  # a shared vertex: every pair of its two sides, both ways
    k = np.arange(1, triangles)
    want[2 * k] = 2.0 * (2 * k) * (n - 1 - 2 * k)
    # whole numbers below 2^53, one rounding per BCC of the vertex at most
    assert np.max(np.abs(out[0] - want) / np.maximum(want, 1.0)) <= 1e-14
