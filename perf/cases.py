"""What this framework is used for, as timed calls through its public entry points.

Exact betweenness centrality is asked for in four ways, and each has its cases:

* one BCC at a time through the calls that stand in for the reference's
  ``begin_gpu`` (host buffers, device buffers, chain endpoints with their ears);
* a whole graph in one call, host edges or a decomposition in, host BC out;
* a plan that stays on the device and is run again, whole or over a unit range
  (a sampled estimate, or one shard of a job over several GPUs);
* the one-shot form of such a range, with its uploads.

The graphs are the ones the repository's benchmark and tests are built on: a
small core with pendants and chains, R-MAT, a road-like grid, batches of
Barabasi-Albert graphs. They are made here with torch on the GPU, since the
largest ones take seconds otherwise.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

_ROOT = Path(__file__).resolve().parents[1]


def _pkg():
    """The package under the current tree, whose folder name is not an identifier."""
    name = "centrality_gpu_b200"
    if name not in sys.modules:
        d = Path.cwd() / "centrality-gpu_b200"
        d = d if d.is_dir() else _ROOT / "centrality-gpu_b200"
        spec = importlib.util.spec_from_file_location(name, d / "__init__.py", submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ------------------------------------------------------------------ cases ----


def listed():
    return [
        # The smallest call: one little BCC out of a decomposition that the
        # caller made, every vertex a free source. A caller makes thousands of
        # these, so what counts is the call's own cost.
        dict(name="free_64", kind="free", n=64, deg=3.0, sources=64),
        # The same for a caller whose buffers are on the device already (a
        # framework's tensors), with a part of the sources: the largest BCCs
        # that this entry point takes are four times this one.
        dict(name="free_device_4001", kind="free_device", n=4001, deg=4.0, sources=1500),
        # Chain endpoints and their ears, the second half of the reference's
        # pair of calls, on an ordinary BCC.
        dict(name="active_ears_1500", kind="active", core=700, deg=3.2, ears=200, ear_lo=1, ear_hi=7),
        # The 2,000-vertex configuration as a Python user meets it: edges in,
        # BC out, the default options (FP64, one source at a time).
        dict(name="betweenness_2000", kind="betweenness", core=1000),
        # The same graph kept on the device and replayed from a captured graph.
        dict(name="small_replay", kind="plan", graph="small", core=1000, mode="batched", delta="fp64", width=0,
             capture=True, at=0.0, units=0),
        # Many uneven graphs in one launch, a sixteenth of the 4,096-graph batch.
        dict(name="ba_batch_256", kind="plan", graph="ba", count=256, n_lo=50, n_hi=5000, mode="batched",
             delta="fp32c", width=0, capture=False, at=0.0, units=0),
        # A whole road-like graph of high diameter in one call.
        dict(name="grid_80_run", kind="run", graph="grid", side=80, mode="batched", delta="fp32c", width=0),
        # The road-like configuration at full size; all its sources take about
        # a minute, so a shard of them.
        dict(name="grid_512_shard", kind="plan", graph="grid", side=512, mode="batched", delta="fp32c", width=0,
             capture=False, at=0.5, units=1184),
        # What the command line does after reading the file: edges,
        # decomposition on the GPU, every source of every BCC.
        dict(name="rmat_14_pipeline", kind="pipeline", graph="rmat", scale=14, factor=16, chains=0.1, hi=4,
             mode="batched", delta="fp32c", width=0),
        # R-MAT 16 with 20% chains, double precision, one-shot over a few
        # passes: a sampled estimate from host buffers, uploads included.
        dict(name="rmat_16_sample_fp64", kind="run_units", graph="rmat", scale=16, factor=16, chains=0.2, hi=8,
             mode="batched", delta="fp64", width=256, at=0.4, units=6),
        # The headline configuration: R-MAT 20 on the device, two passes of 512.
        dict(name="rmat_20_passes", kind="plan", graph="rmat", scale=20, factor=16, chains=0.1, hi=4, mode="batched",
             delta="fp32c", width=512, capture=False, at=0.5, units=2),
        # The per-source FP64 schedule on R-MAT: the form a caller picks for
        # full precision on a graph that no small-BCC form fits.
        dict(name="rmat_14_plain", kind="plan", graph="rmat", scale=14, factor=16, chains=0.2, hi=8, mode="plain",
             delta="fp64", width=0, capture=False, at=0.25, units=592),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["free", "free_device", "active", "betweenness", "small", "ba", "grid_run", "grid_shard",
                       "pipeline", "sample", "passes", "plain"])
    if kind == "free":
        n = _log(rng, 24, 1500)
        return dict(kind="free", n=n, deg=round(rng.uniform(2.3, 6.0), 2), sources=max(1, int(n * rng.choice([1.0, 0.5]))))
    if kind == "free_device":
        n = _log(rng, 150, 16000)
        return dict(kind="free_device", n=n, deg=round(rng.uniform(2.3, 6.0), 2), sources=min(n, _log(rng, 100, 1500)))
    if kind == "active":
        core = _log(rng, 30, 1500)
        return dict(kind="active", core=core, deg=round(rng.uniform(2.6, 5.0), 2), ears=max(2, core // rng.randint(3, 8)),
                    ear_lo=1, ear_hi=rng.randint(1, 9))
    if kind == "betweenness":
        return dict(kind="betweenness", core=_log(rng, 40, 2000))
    if kind == "small":
        return dict(kind="plan", graph="small", core=_log(rng, 60, 2500), mode="batched",
                    delta=rng.choice(["fp64", "fp32c"]), width=0, capture=rng.random() < 0.7, at=0.0, units=0)
    if kind == "ba":
        return dict(kind="plan", graph="ba", count=_log(rng, 16, 256), n_lo=50, n_hi=_log(rng, 400, 5000),
                    mode="batched", delta="fp32c", width=0, capture=rng.random() < 0.5, at=0.0, units=0)
    if kind == "grid_run":
        return dict(kind="run", graph="grid", side=_log(rng, 20, 88), mode=rng.choice(["batched", "batched", "plain"]),
                    delta="fp32c", width=0)
    if kind == "grid_shard":
        return dict(kind="plan", graph="grid", side=_log(rng, 128, 512), mode="batched", delta="fp32c", width=0,
                    capture=False, at=round(rng.uniform(0.1, 0.8), 3), units=rng.randint(592, 1184))
    if kind == "pipeline":
        return dict(kind="pipeline", graph="rmat", scale=rng.randint(9, 14), factor=rng.randint(6, 16),
                    chains=round(rng.uniform(0.05, 0.1), 3), hi=rng.randint(1, 4), mode="batched",
                    delta=rng.choice(["fp32c", "fp64"]), width=0)
    if kind == "sample":
        return dict(kind="run_units", graph="rmat", scale=rng.randint(15, 17), factor=16,
                    chains=round(rng.uniform(0.05, 0.2), 3), hi=rng.randint(2, 8), mode="batched",
                    delta=rng.choice(["fp64", "fp32c"]), width=rng.choice([128, 256, 512]),
                    at=round(rng.uniform(0.05, 0.8), 3), units=rng.randint(1, 6))
    if kind == "passes":
        return dict(kind="plan", graph="rmat", scale=rng.randint(15, 19), factor=16,
                    chains=round(rng.uniform(0.05, 0.2), 3), hi=rng.randint(2, 8), mode="batched",
                    delta=rng.choice(["fp32c", "fp32c", "fp64"]), width=rng.choice([128, 256, 384, 512, 1024]),
                    capture=rng.random() < 0.5, at=round(rng.uniform(0.05, 0.8), 3), units=rng.randint(1, 3))
    return dict(kind="plan", graph="rmat", scale=rng.randint(12, 14), factor=rng.randint(8, 16),
                chains=round(rng.uniform(0.05, 0.2), 3), hi=rng.randint(2, 8), mode="plain", delta="fp64", width=0,
                capture=False, at=round(rng.uniform(0.05, 0.7), 3), units=rng.randint(296, 592))


# ----------------------------------------------------------------- graphs ----
# Each returns (n, u, v), every undirected edge once, as int64 tensors on the GPU.


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + 17)
    return g


def _ints(g, lo, hi, count):
    return torch.randint(lo, hi, (count,), generator=g, device="cuda", dtype=torch.int64)


def _unit(g, count):
    return torch.rand(count, generator=g, device="cuda", dtype=torch.float32)


def _range(count, start=0):
    return torch.arange(start, start + count, device="cuda", dtype=torch.int64)


def _simple(n, u, v):
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.minimum(u, v) * n + torch.maximum(u, v))
    return key // n, key % n


def _some(g, size, count):
    """A random `count` of `size` places, as a mask."""
    mask = torch.zeros(size, dtype=torch.bool, device="cuda")
    mask[torch.argsort(_unit(g, size))[:count]] = True
    return mask


def _subdivide(g, n, u, v, pick, lo, hi):
    """The picked edges become paths through lo..hi new vertices each (every
    length equally often, in random order: another seed gives a graph of the
    same size), numbered path by path; also returns how many each got."""
    su, sv = u[pick], v[pick]
    k = (lo + _range(len(su)) % (hi - lo + 1))[torch.argsort(_unit(g, len(su)))]
    first = n + torch.cumsum(k, 0) - k
    owner = torch.repeat_interleave(_range(len(su)), k)
    new = _range(int(k.sum()), n)
    prev = torch.where(new == first[owner], su[owner], new - 1)
    return n + len(new), torch.cat([u[~pick], prev, first + k - 1]), torch.cat([v[~pick], new, sv]), k


def _leaves(g, n, u, v, count, targets):
    return n + count, torch.cat([u, _ints(g, 0, targets, count)]), torch.cat([v, _range(count, n)])


def _small(g, core):
    """A random core of degree about 6, a pendant for every second core vertex,
    and core / 10 chains of five."""
    a = _range(core).repeat_interleave(3)
    u, v = _simple(core, a, _ints(g, 0, core, 3 * core))
    n, u, v = _leaves(g, core, u, v, core // 2, core)
    c = max(1, core // 10)
    x = _ints(g, 0, core, c)
    y = (x + 1 + _ints(g, 0, core - 1, c)) % core
    eu, ev = torch.cat([u, x]), torch.cat([v, y])
    pick = torch.zeros(len(eu), dtype=torch.bool, device="cuda")
    pick[len(u):] = True
    return _subdivide(g, n, eu, ev, pick, 5, 5)[:3]


# The share of an R-MAT's edges that is left without loops and repeats, a little
# below what 16 edges a vertex give.
_KEPT = {9: 0.6, 10: 0.64, 11: 0.69, 12: 0.73, 13: 0.77, 14: 0.81, 15: 0.84, 16: 0.87, 17: 0.89, 18: 0.91, 19: 0.92,
         20: 0.93}


def _rmat(g, scale, factor, chains, hi):
    m = factor << scale
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros_like(u)
    a, ab, abc = 0.57, 0.76, 0.95
    for bit in range(scale):
        r = _unit(g, m)
        u |= (r >= ab).long() << bit
        v |= (((r >= a) & (r < ab)) | (r >= abc)).long() << bit
    n = 1 << scale
    u, v = _simple(n, u, v)
    return _subdivide(g, n, u, v, _some(g, len(u), int(chains * _KEPT[scale] * m)), 1, hi)[:3]


def _grid(g, side):
    """A grid with 10% of its edges gone, 30% of the rest subdivided by one to
    four vertices, and leaves on about 6% of its vertices."""
    idx = _range(side * side).reshape(side, side)
    u = torch.cat([idx[:, :-1].reshape(-1), idx[:-1].reshape(-1)])
    v = torch.cat([idx[:, 1:].reshape(-1), idx[1:].reshape(-1)])
    keep = ~_some(g, len(u), len(u) // 10)
    u, v = u[keep], v[keep]
    n, u, v, _ = _subdivide(g, side * side, u, v, _some(g, len(u), 3 * len(u) // 10), 1, 4)
    return _leaves(g, n, u, v, side * side * 15 // 262, side * side)


def _ba(g, count, n_lo, n_hi):
    """Preferential attachment with two edges a vertex, sizes log-uniform, about
    10% of the edges subdivided by one to three vertices, leaves on 10%."""
    cpu = np.random.default_rng(int(_ints(g, 0, 1 << 40, 1)))
    us, vs, base = [], [], 0
    # sizes are laid out over the range, not drawn, so that another seed is
    # another batch of the same amount of work
    sizes = np.exp(np.log(n_lo) + (np.arange(count) + 0.5) / count * (np.log(n_hi) - np.log(n_lo))).astype(np.int64)
    for n0 in cpu.permutation(sizes):
        # the list of edge ends so far: 0 and 1, then for edge e its chosen end
        # and its new vertex 2 + e // 2; a choice is a uniform earlier place of
        # the list, and a chosen end stands for what was chosen there
        e = np.arange(2 * int(n0 - 2))
        choice = (cpu.random(len(e)) * (2 + 4 * (e // 2))).astype(np.int64)
        at = choice.copy()
        while True:
            again = (at >= 2) & (at % 2 == 0)
            if not again.any():
                break
            at[again] = choice[(at[again] - 2) // 2]
        us += [base + 2 + e // 2, [base]]
        vs += [base + np.where(at < 2, at, 2 + (at - 3) // 2 // 2), [base + 1]]
        base += int(n0)
    u = torch.from_numpy(np.concatenate(us)).cuda()
    v = torch.from_numpy(np.concatenate(vs)).cuda()
    u, v = _simple(base, u, v)
    n, u, v, _ = _subdivide(g, base, u, v, _some(g, len(u), base // 6), 1, 3)
    return _leaves(g, n, u, v, base // 10, base)


def _graph(case, seed):
    g = _gen(seed)
    kind = case.get("graph", "small")
    if kind == "rmat":
        n, u, v = _rmat(g, case["scale"], case["factor"], case["chains"], case["hi"])
    elif kind == "grid":
        n, u, v = _grid(g, case["side"])
    elif kind == "ba":
        n, u, v = _ba(g, case["count"], case["n_lo"], case["n_hi"])
    else:
        n, u, v = _small(g, case["core"])
    return (n,) + _simple(n, u, v)


def _host(t):
    return t.to(torch.int32).cpu().numpy()


def _csr(n, u, v):
    """Symmetric CSR with sorted rows, int32, on the GPU."""
    key = torch.sort(torch.cat([u * n + v, v * n + u])).values
    row = torch.searchsorted(key, torch.arange(n + 1, device="cuda", dtype=torch.int64) * n)
    return row.to(torch.int32), (key % n).to(torch.int32)


def _one_bcc(case, seed):
    """One BCC as its caller holds it: (n, u, v, reach, sources, ears). A cycle
    through a random order of the vertices with random edges on top, so it has
    no cut vertex; about a tenth of the vertices have something hanging off."""
    g = _gen(seed)
    active = case["kind"] == "active"
    n0 = case["core"] if active else case["n"]
    order = torch.argsort(_unit(g, n0))
    extra = int(n0 * (case["deg"] - 2.0) / 2.0)
    u, v = _simple(n0, torch.cat([order, _ints(g, 0, n0, extra)]), torch.cat([order.roll(1), _ints(g, 0, n0, extra)]))
    n, ears = n0, None
    if active:  # some of the edges become chains: the ears
        pick = _some(g, len(u), case["ears"])
        ends = torch.stack([u[pick], v[pick]], 1).tolist()
        n, u, v, lens = _subdivide(g, n0, u, v, pick, case["ear_lo"], case["ear_hi"])
        ears, at = [], n0
        for (a, b), k in zip(ends, lens.tolist()):
            ears.append((a, b, [(j + 1, at + j, k - j) for j in range(k)]))
            at += k
        sources = np.unique(np.array(ends, dtype=np.int32))
    else:
        sources = torch.sort(torch.argsort(_unit(g, n0))[:case["sources"]]).values.to(torch.int32)
    w = _unit(g, n)
    reach = torch.where(w < 0.1, 1.0 + 2000.0 * w * w, torch.zeros_like(w)).to(torch.int32)
    return n, u, v, reach, sources, ears


# -------------------------------------------------------------------- run ----


def _context(P, case, **more):
    return P.Context(mode=P.MODE_PLAIN if case.get("mode") == "plain" else P.MODE_BATCHED,
                     delta=P.DELTA_FP64 if case.get("delta") == "fp64" else P.DELTA_FP32C,
                     batch_width=case.get("width", 0), **more)


def _range_of(case, units):
    """The units of this case: all of them, or `units` of them from a fraction
    `at` of the list (clear of its end)."""
    if not case.get("units"):
        return 0, units
    k = min(case["units"], units)
    b = min(int(case["at"] * units), units - k)
    return b, b + k


def prepare(case, seed):
    P = _pkg()
    s = dict(P=P, kind=case["kind"], case=dict(case))
    if case["kind"] in ("free", "free_device", "active"):
        n, u, v, reach, src, ears = _one_bcc(case, seed)
        row, col = _csr(n, u, v)
        s.update(n=n, m=len(col), ctx=_context(P, case), ears=ears)
        if case["kind"] == "free_device":
            s.update(row=row, col=col, reach=reach, src=src, bc=torch.zeros(n, dtype=torch.float64, device="cuda"))
        else:
            s.update(row=row.cpu().numpy(), col=col.cpu().numpy(), reach=reach.cpu().numpy(),
                     src=src if ears else src.cpu().numpy(), bc=np.zeros(n, dtype=np.float32))
        torch.cuda.synchronize()
        return s
    n, u, v = _graph(case, seed)
    s.update(n=n, u=_host(u), v=_host(v))
    if case["kind"] == "betweenness":
        return s
    if case["kind"] == "pipeline":
        s["ctx"] = _context(P, case)
        return s
    # graphs of thousands of BFS levels decompose faster on the host, as the
    # library's own notes say
    s["decomp"] = P.Decomposition(P.Graph.from_edges(n, s["u"], s["v"]), gpu_device=0 if case["graph"] == "rmat" else None)
    s["ctx"] = _context(P, case, graph=bool(case.get("capture")))
    if case["kind"] == "run_units":
        # the unit count of a multi-source plan follows from the largest BCC
        V = s["decomp"].view.contents
        s["range"] = _range_of(case, -(-int(V.vtx_off[1]) // case["width"]))
    elif case["kind"] == "plan":
        s["plan"] = s["ctx"].plan(s["decomp"])
        s["range"] = _range_of(case, s["plan"].n_units)
        if case.get("capture"):
            s["plan"].record(*s["range"])
    torch.cuda.synchronize()
    return s


def run(s):
    P, kind = s["P"], s["kind"]
    if kind == "free":
        P.begin_gpu_free(s["ctx"], s["row"], s["col"], s["n"], s["m"], s["src"], s["reach"], s["bc"])
        return s["bc"]
    if kind == "free_device":
        P.begin_gpu_free_noalloc(s["ctx"], s["row"].data_ptr(), s["col"].data_ptr(), s["n"], s["m"], s["src"].data_ptr(),
                                 len(s["src"]), s["reach"].data_ptr(), s["bc"].data_ptr())
        return s["bc"]
    if kind == "active":
        bc = np.zeros(s["n"], dtype=np.float32)
        P.begin_gpu_active(s["ctx"], s["row"], s["col"], s["n"], s["m"], s["src"], s["ears"], s["reach"], bc)
        return bc
    if kind == "betweenness":
        return P.betweenness(s["n"], s["u"], s["v"])[0]
    if kind == "pipeline":
        d = P.Decomposition(P.Graph.from_edges(s["n"], s["u"], s["v"]), gpu_device=0)
        return s["ctx"].run(d)[0]
    if kind == "run":
        return s["ctx"].run(s["decomp"])[0]
    if kind == "run_units":
        return s["ctx"].run_units(s["decomp"], *s["range"])[0]
    s["plan"].reset()
    s["plan"].run(*s["range"], stats=False)
    return s["plan"].read()


# ------------------------------------------------------------- work, exact ----


def _sizes(case):
    """(vertices, arcs, sources) of a case, near enough for an account of its
    work: the numbers that the generators give on average."""
    k = case["kind"]
    if k in ("free", "free_device"):
        return case["n"], case["n"] * case["deg"], case["sources"]
    if k == "active":
        z = case["ears"] * (case["ear_lo"] + case["ear_hi"]) / 2
        return case["core"] + z, case["core"] * case["deg"] + 2 * z, z + min(case["core"], 2 * case["ears"])
    g = case.get("graph", "small")
    if g == "small":
        n = 1.45 * case["core"]  # pendants are outside its one BCC
        return n, 7.0 * case["core"], n
    if g == "ba":
        t = (np.arange(case["count"]) + 0.5) / case["count"]
        sizes = np.exp(np.log(case["n_lo"]) + t * (np.log(case["n_hi"]) - np.log(case["n_lo"]))) * 1.4
        # every source scans its own graph: the arcs that reproduce that sum
        return sizes.sum(), 3.1 * (sizes ** 2).sum() / sizes.sum(), sizes.sum()
    if g == "grid":
        n = 2.35 * case["side"] ** 2
        per_unit = 2.3
    else:
        m = _KEPT[case["scale"]] * (case["factor"] << case["scale"])
        z = case["chains"] * m * (1 + case["hi"]) / 2
        n = 0.42 * (1 << case["scale"]) + z
        per_unit = 1 + min(16.0, z / (0.42 * (1 << case["scale"])))
        arcs = 2 * (m + z)
    if g == "grid":
        arcs = 2.68 * n
    if case.get("units"):
        src = case["units"] * (case["width"] if case["width"] else per_unit)
        return n, arcs, min(n, src)
    return n, arcs, n


def work(case):
    """Every source has to look at each arc of its BCC once on the way out and
    once on the way back, with an addition each, and at each vertex for a
    multiplication, a division and two additions. The bytes are those of the
    graph, once, and of the result."""
    n, arcs, src = _sizes(case)
    return {"bytes": 4.0 * arcs + 16.0 * n, "flops": float(src) * (2.0 * arcs + 4.0 * n)}


def _brandes(n, u, v, weight=None, sources=None):
    """Weighted Brandes in 64 bits by sparse products on the GPU: the sum over
    sources s of weight(s) * delta_s(v), delta with targets weighted likewise."""
    row, col = _csr(n, u, v)
    A = torch.sparse_csr_tensor(row.long(), col.long(), torch.ones(len(col), dtype=torch.float64, device="cuda"), (n, n))
    weight = torch.ones(n, dtype=torch.float64, device="cuda") if weight is None else weight.double()
    sources = _range(n) if sources is None else torch.as_tensor(sources, device="cuda").long()
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    step = max(32, min(1024, int(1.5e8 // max(n, 1))))
    for at in range(0, len(sources), step):
        s = sources[at:at + step]
        k = torch.arange(len(s), device="cuda")
        dist = torch.full((n, len(s)), -1, dtype=torch.int16, device="cuda")
        sigma = torch.zeros((n, len(s)), dtype=torch.float64, device="cuda")
        dist[s, k] = 0
        sigma[s, k] = 1.0
        front, lev = sigma.clone(), 0
        while True:
            front = A @ front
            new = (front > 0) & (dist < 0)
            if not bool(new.any()):
                break
            lev += 1
            front = torch.where(new, front, torch.zeros((), dtype=torch.float64, device="cuda"))
            dist[new] = lev
            sigma += front
        delta = torch.zeros_like(sigma)
        zero = torch.zeros((), dtype=torch.float64, device="cuda")
        for l in range(lev, 1, -1):
            q = torch.where(dist == l, (weight[:, None] + delta) / sigma, zero)
            delta += torch.where(dist == l - 1, sigma * (A @ q), zero)
        out += (delta * weight[s][None, :]).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("free", "free_device", "active"):
        n, u, v, reach, src, ears = _one_bcc(case, seed)
        if ears:
            src = np.concatenate([src, [z for e in ears for _, z, _ in e[2]]])
        bc = _brandes(n, u, v, reach.double() + 1.0, src)
        return bc if kind == "free_device" else bc.cpu().numpy()
    # a unit range's sources are the framework's own choice, so nothing but the
    # framework knows them; a whole run needs none of that
    if case.get("units"):
        return None
    if case.get("graph") == "ba":
        if case["count"] * case["n_hi"] > 60_000:
            return None  # the sources of all graphs together: minutes
    elif case.get("graph") == "grid" and case["side"] > 90:
        return None
    n, u, v = _graph(case, seed)
    return _brandes(n, u, v).cpu().numpy()
