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
d = decomp(*ring({size}, {size}, {400 if size > 1000 else 4}, {length}, 1))
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
    CTAs of any kernel fit): the contracted kernel's own, or the whole-BCC kernel's, which
    takes the BCCs with chains too long for that one and those with few chains: a
    seventh of a ring's vertices have no chord."""
    res = run_stub(stub_dir, RING + """
for name, chains, length in (("contracted", 400, 9), ("long chains", 80, 70), ("few chains", 10, 9)):
    d = decomp(*ring(14000, 14000, chains, length, 1))
    ctx = P.Context(mode=P.MODE_PLAIN, plain_ctas_per_sm=16)
    plan = ctx.plan(d)
    out[name] = plan.concurrency
    plan.close()
    ctx.close()
""")
    assert res == {"contracted": 148 * 4, "long chains": 148 * 16, "few chains": 148 * 16}


@pytest.mark.parametrize("sub_p,contracted", [(0.0, False), (0.02, True)])
def test_deep_bccs_with_any_chains_are_contracted(stub_dir, sub_p, contracted):  # noqa: F811
    """A grid of 130 x 130 with no vertex on a chain, and with one in eleven."""
    res = run_stub(stub_dir, f"""
d = decomp(*G.gen_grid(130, delete_frac=0.0, sub_p={sub_p}, leaves=0, seed=3))
a = d.arrays()
out["share"] = int(a["n_plain"][0]) / int(a["n_packed"])
ctx = P.Context(mode=P.MODE_PLAIN, plain_ctas_per_sm=16)
plan = ctx.plan(d)
out["concurrency"] = plan.concurrency
plan.close()
ctx.close()
""")
    assert (res["share"] > 0.97) == (not contracted) and res["share"] > 0.8
    assert res["concurrency"] == 148 * (4 if contracted else 16)


@pytest.mark.parametrize("sources,contracted", [(256, True), (257, False)])
def test_few_sources_of_a_bcc_with_hubs_are_contracted(stub_dir, sources, contracted):  # noqa: F811
    """A free-source call has no chains: only up to 256 sources of a BCC with a row
    of more than 1,024 arcs go to the contracted kernel, which allocates tables."""
    res = run_stub(stub_dir, f"""
L.stub_cudart_mallocs.restype = C.c_longlong
rng = np.random.default_rng(3)
n = 16000
i = np.arange(n)
counts = []
for hub in (1500, 1000):
    a = decomp(n, *G.simple_edges(n, np.concatenate([i, rng.integers(0, n, n), np.zeros(hub, int)]),
                                  np.concatenate([(i + 1) % n, rng.integers(0, n, n), rng.permutation(n)[:hub]]))).arrays()
    assert a["n_bcc"] == 1 and int(a["n_packed"]) == n
    src = np.arange({sources}, dtype=np.int32)
    ctx = P.Context(mode=P.MODE_PLAIN)
    m0 = L.stub_cudart_mallocs()
    P.begin_gpu_free(ctx, a["row"].astype(np.int32), a["col"].astype(np.int32), n, len(a["col"]), src,
                     a["reach"].astype(np.int32), np.zeros(n, np.float32))
    counts.append(L.stub_cudart_mallocs() - m0)
    ctx.close()
out["more"] = counts[0] - counts[1]
""")
    assert (res["more"] > 0) == contracted
