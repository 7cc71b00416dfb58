"""A kernel's limit of dynamic shared memory belongs to the function, not to a
call: were it set to what one launch needs, a launch of another thread with a
context of its own could find it lowered. Plans and calls of different sizes set
one value per kernel (stand-in runtime)."""
import os
import subprocess
import sys

from test_host_plumbing import PKG, STUB, run_stub, stub_dir  # noqa: F401


def test_one_limit_per_kernel(stub_dir, tmp_path):  # noqa: F811
    sys.path.insert(0, str(PKG))
    import build as pkg_build
    objs = [str(PKG / "_build" / (s + ".o")) for s in pkg_build.CU_SOURCES + pkg_build.CXX_SOURCES]
    stub_o = tmp_path / "func_attr_log.o"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-I/usr/local/cuda/include", "-I", str(STUB), "-c",
                    str(STUB / "func_attr_log.cpp"), "-o", str(stub_o)], check=True)
    subprocess.run(["g++", "-shared", "-o", str(tmp_path / "libbcgpu.so")] + objs +
                   [str(stub_o), "-lgomp", "-Wl,--no-undefined", "-Wl,-Bsymbolic"], check=True)
    res = run_stub(tmp_path, """
graphs_ = [G.pack_graphs(G.gen_ba_batch(20, lo, hi, seed=7))[:3] for lo, hi in ((40, 90), (300, 900), (1000, 7000))]
graphs_ += [G.gen_grid(k, leaves=20, seed=3) for k in (40, 100, 130)] + [G.gen_rmat(k, 16, 0.2, 1, 8, seed=2) for k in (11, 13)]
for g in graphs_:
    d = decomp(*g)
    for opts in (dict(mode=P.MODE_PLAIN), dict(mode=P.MODE_BATCHED), dict(mode=P.MODE_BATCHED, tile_max=-1),
                 dict(mode=P.MODE_BATCHED, plain_core=200, batch_width=128)):
        ctx = P.Context(**opts)
        ctx.run(d)
        ctx.close()
ctx = P.Context(mode=P.MODE_PLAIN)
for n in (50, 700, 2000, 6000):
    i = np.arange(n)
    a = decomp(n, *G.simple_edges(n, np.concatenate([i, i[:n // 2]]), np.concatenate([(i + 1) % n, (i[:n // 2] + n // 3) % n]))).arrays()
    nb = int(a["vtx_off"][1])
    R, Cc, reach = a["row"].astype(np.int32), a["col"].astype(np.int32), a["reach"].astype(np.int32)
    src = np.arange(nb, dtype=np.int32)
    bc = np.zeros(nb)
    P.begin_gpu_free_noalloc(ctx, R.ctypes.data, Cc.ctypes.data, nb, len(Cc), src.ctypes.data, nb, reach.ctypes.data,
                             bc.ctypes.data)
ctx.close()
out["kernels"] = L.stub_cudart_limited_kernels()
out["values"] = L.stub_cudart_limits_of_one_kernel()
""")
    assert res["kernels"] >= 6 and res["values"] == 1, res
