"""The whole-BCC per-source kernel on BCCs beyond shared memory that the contracted
kernel does not take: without chains, and with chains too long for it (merged
from their ends). Rescaling forced on almost every level leaves BC bit for bit,
and it is the oracle's."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def dense(n, m, chains, seed):
    """A random graph too dense for shared memory, chains of 62 to 70, leaves."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    us, vs = [i, rng.integers(0, n, m)], [(i + 1) % n, rng.integers(0, n, m)]
    for k in chains:
        a, b = rng.choice(n, 2, replace=False)
        path = np.concatenate([[a], n + np.arange(k), [b]])
        us.append(path[:-1])
        vs.append(path[1:])
        n += k
    us.append(rng.integers(0, n, 200))
    vs.append(n + np.arange(200))
    n += 200
    return (n,) + graphs().simple_edges(n, np.concatenate(us), np.concatenate(vs))


@pytest.mark.parametrize("chains", [[], [62, 70, 65, 62]], ids=["no-chains", "long-chains"])
@pytest.mark.parametrize("ctas", [0, 16])
def test_bc_and_forced_rescaling(chains, ctas):
    P, O = pkg(), oracle()
    n, u, v = dense(1500, 60000, chains, 5)
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    outs = []
    for rescale in (0, 2):
        ctx = P.Context(mode=P.MODE_PLAIN, plain_ctas_per_sm=ctas, rescale_exp=rescale)
        plan = ctx.plan(d)
        for _ in range(2):
            plan.reset()
            st = plan.run()
            assert plan.tile_launches() == [] and (st["bfs_sources"] < st["sources"]) == bool(chains)
            outs.append(plan.read())
        plan.close()
        ctx.close()
    assert all(np.array_equal(x, outs[0]) for x in outs)
    assert rel_err(outs[0], O.brandes(n, *O.csr(n, u, v))) < TOL
