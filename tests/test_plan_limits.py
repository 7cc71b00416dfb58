"""bc_opts.workspace_limit on the stand-in runtime: a plan that is accepted holds
no more device memory than the limit, whichever kernels its items run on, and the
least limit that is accepted depends on the rows of the largest BCC alone (two
slots beside the graph, the counters and the items)."""
import pytest

from test_host_plumbing import run_stub, stub_dir  # noqa: F401

GRAPHS = {
    # one BCC on the contracted kernel
    "rmat": "G.gen_rmat(13, 16, chain_frac=0.2, chain_hi=8, seed=2)",
    "grid": "G.gen_grid(120, leaves=100, seed=3)",
    # BCCs that fit shared memory
    "small": "G.pack_graphs(G.gen_ba_batch(30, 100, 900, seed=7))[:3]",
    # those and larger ones; a BCC with a chain too long for the contracted kernel and
    # one without, both beyond shared memory
    "mixed": "G.pack_graphs(G.gen_ba_batch(4, 100, 900, seed=7) + G.gen_ba_batch(2, 9000, 12000, seed=8))[:3]",
    "both": "two_kernels()",
}
TWO_KERNELS = """
def two_kernels():
    rng = np.random.default_rng(5)
    n, us, vs = 0, [], []
    for size, chain in ((14000, 0), (14000, 70)):
        i = np.arange(size)
        u, v = np.concatenate([i, rng.integers(0, size, size)]), np.concatenate([(i + 1) % size, rng.integers(0, size, size)])
        size, u, v = G.subdivide(size, u, v, 0.2, 1, 4, rng)
        path = np.concatenate([[0], size + np.arange(chain), [size // 2]])
        us += [n + u, n + path[:-1]]
        vs += [n + v, n + path[1:]]
        n += size + chain
    return (n,) + G.simple_edges(n, np.concatenate(us), np.concatenate(vs))
"""


@pytest.mark.parametrize("name", list(GRAPHS))
def test_plain_plans_stay_within_the_limit(stub_dir, name):  # noqa: F811
    res = run_stub(stub_dir, TWO_KERNELS + f"""
d = decomp(*{GRAPHS[name]})
a = d.arrays()
n, nb, m, nch = int(a["n_packed"]), int(a["n_bcc"]), len(a["col"]), len(a["chain_l"])
graph = 8 * (n + 1) + 8 * (nb + 1) + 4 * m + 4 * n + 4 * 4 * max(nch, 1) + 8 * n + 4 + 8
ctx = P.Context(mode=P.MODE_PLAIN)
plan = ctx.plan(d)
items = plan.n_units
plan.close()
ctx.close()
rows = 76 * (int(np.diff(a["vtx_off"]).max()) + 2)
least = graph + 32 * n + 20 * items + 2 * rows + 64 * 148
out["least"] = least
for extra in (-1, 0, rows, 3 * rows, 10 * rows, 40 * rows, 150 * rows, 600 * rows):
    ctx = P.Context(mode=P.MODE_PLAIN, workspace_limit=least + extra)
    got = []
    def build():
        plan = ctx.plan(d)
        got.append(int(L.bc_plan_device_bytes(plan._h)))
        plan.close()
    r = raises(build)
    out[str(extra)] = r[0] if r else got[0] - (least + extra)
    ctx.close()
""")
    least = res.pop("least")
    assert res.pop("-1") == 3, least  # BCGPU_ENOMEM
    assert all(v <= 0 for v in res.values()), (least, res)


@pytest.mark.parametrize("width,delta", [(128, "P.DELTA_FP32C"), (256, "P.DELTA_FP64")])
def test_merged_passes_give_way_to_the_rest_of_the_plan(stub_dir, width, delta):  # noqa: F811
    """Multi-source passes (an R-MAT BCC) beside per-source items (a grid too deep
    for them) and small BCCs: once a limit is accepted, every larger one is, and
    what passes run as one take stays within it."""
    res = run_stub(stub_dir, f"""
n, us, vs = 0, [], []
for k, u, v in (G.gen_rmat(12, 16, chain_frac=0.2, chain_hi=8, seed=2), G.gen_grid(90, leaves=50, seed=3),
                G.pack_graphs(G.gen_ba_batch(6, 60, 300, seed=7))[:3]):
    us.append(n + u)
    vs.append(n + v)
    n += k
d = decomp(n, np.concatenate(us), np.concatenate(vs))
got = []
for i in range(28):
    limit = int(4e6 * 1.2 ** i)
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=1500, batch_width={width}, delta={delta}, workspace_limit=limit)
    held = []
    def build():
        plan = ctx.plan(d)
        held.append(plan.device_bytes)
        plan.close()
    r = raises(build)
    got.append([limit, r[0] if r else 0, held[0] if held else 0])
    ctx.close()
out["got"] = got
""")["got"]
    first = next(i for i, g in enumerate(res) if g[1] == 0)
    assert 0 < first < 20 and all(code == 3 for _, code, _ in res[:first])
    assert all(code == 0 for _, code, _ in res[first:]), res
    least = res[first][2]
    assert all(held <= max(limit, least) for limit, _, held in res[first:]), res
    assert res[-1][2] > 2 * least  # with room, passes run as one and more sources are in flight
