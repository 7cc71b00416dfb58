"""Calls of several host threads at once, each with a context of its own and BCCs
that need different amounts of shared memory of the same kernels: every call gives
what it gives alone."""
import threading

import numpy as np
import pytest

from helpers import graphs, pkg

pytestmark = pytest.mark.gpu


def bcc(n, seed):
    """A ring with chords; chains on a third of its edges when n is odd."""
    G = graphs()
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    u, v = G.simple_edges(n, np.concatenate([i, rng.integers(0, n, n)]), np.concatenate([(i + 1) % n, rng.integers(0, n, n)]))
    if n % 2:
        n, u, v = G.subdivide(n, u, v, 0.33, 1, 4, rng)
    return (n, u, v)


def test_contexts_of_four_threads():
    P = pkg()
    sizes = [[60, 2401, 900], [3000, 301, 150], [12001, 640, 60], [1301, 5000, 9001]]
    work = [[P.Decomposition(P.Graph.from_edges(*bcc(n, n))) for n in row] for row in sizes]
    modes = [dict(mode=P.MODE_PLAIN), dict(mode=P.MODE_BATCHED), dict(mode=P.MODE_PLAIN),
             dict(mode=P.MODE_BATCHED, plain_core=1000, delta=P.DELTA_FP64)]
    alone = []
    for row, opts in zip(work, modes):
        ctx = P.Context(**opts)
        alone.append([ctx.run(d)[0] for d in row])
        ctx.close()
    bad = []

    def go(k):
        try:
            ctx = P.Context(**modes[k])
            for rep in range(6):
                for d, want in zip(work[k], alone[k]):
                    if not np.array_equal(ctx.run(d)[0], want):
                        bad.append((k, rep, "differs"))
            ctx.close()
        except Exception as e:  # noqa: BLE001
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=go, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert bad == []
