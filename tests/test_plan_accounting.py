"""What a plan says of its per-source work, on the stand-in runtime: the BFS runs
of each kernel that items go to, and the CTAs of it that are resident."""
import pytest

from test_host_plumbing import run_stub, stub_dir  # noqa: F401

RING = """
def ring(n, m, chains, length, seed):
    # a ring with m random chords, and chains of `length` between its vertices
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    us, vs = [i, rng.integers(0, n, m)], [(i + 1) % n, rng.integers(0, n, m)]
    for c in range(chains):
        path = np.concatenate([[c], n + np.arange(length), [n // 2]])
        us.append(path[:-1])
        vs.append(path[1:])
        n += length
    return (n,) + G.simple_edges(n, np.concatenate(us), np.concatenate(vs))
"""


@pytest.mark.parametrize("size,length,merged", [(300, 9, False), (14000, 9, False), (14000, 70, True)])
def test_bfs_runs_by_kernel(stub_dir, size, length, merged):  # noqa: F811
    """A BCC in shared memory, one on the contracted kernel, and one with chains too
    long for that: only the last merges its chain sources."""
    res = run_stub(stub_dir, RING + f"""
d = decomp(*ring({size}, {size}, 4, {length}, 1))
a = d.arrays()
ctx = P.Context(mode=P.MODE_PLAIN)
plan = ctx.plan(d)
st = plan.run()
out["st"] = [st[k] for k in ("sources", "bfs_sources", "aux_bfs")]
first = plan.run(0, 10)
out["first"] = [first[k] for k in ("sources", "bfs_sources", "aux_bfs")]
out["own"] = int(a["n_plain"].sum())
plan.close()
ctx.close()
""")
    sources, bfs, aux = res["st"]
    assert sources > res["own"]
    assert (bfs, aux > 0) == ((res["own"], True) if merged else (sources, False))
    assert (res["first"][1] == res["first"][0]) == (not merged)


def test_concurrency_is_of_the_kernel_that_runs(stub_dir):  # noqa: F811
    """With 16 CTAs an SM asked for (the stand-in device has 148, and says that four
    CTAs of any kernel fit): the contracted kernel's own, or the whole-BCC kernel's."""
    res = run_stub(stub_dir, RING + """
for name, size, chains, length in (("contracted", 14000, 4, 9), ("whole", 14000, 4, 70)):
    d = decomp(*ring(size, size, chains, length, 1))
    ctx = P.Context(mode=P.MODE_PLAIN, plain_ctas_per_sm=16)
    plan = ctx.plan(d)
    out[name] = plan.concurrency
    plan.close()
    ctx.close()
""")
    assert res == {"contracted": 148 * 4, "whole": 148 * 16}
