"""A host allocation that fails on a thread of a plan's routing is an error of the
call, not the end of the process (stand-in runtime, operator new made to fail in
parallel regions)."""
import subprocess
import sys

from test_host_plumbing import PKG, STUB, run_stub, stub_dir  # noqa: F401


def test_routing_out_of_memory_is_an_error(stub_dir, tmp_path, monkeypatch):  # noqa: F811
    sys.path.insert(0, str(PKG))
    import build as pkg_build
    objs = [str(PKG / "_build" / (s + ".o")) for s in pkg_build.CU_SOURCES + pkg_build.CXX_SOURCES]
    stub_o = tmp_path / "host_nomem.o"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-fopenmp", "-I/usr/local/cuda/include", "-I", str(STUB), "-c",
                    str(STUB / "host_nomem.cpp"), "-o", str(stub_o)], check=True)
    subprocess.run(["g++", "-shared", "-o", str(tmp_path / "libbcgpu.so")] + objs +
                   [str(stub_o), "-lgomp", "-Wl,--no-undefined", "-Wl,-Bsymbolic"], check=True)
    monkeypatch.setenv("OMP_NUM_THREADS", "4")
    res = run_stub(tmp_path, """
# BCCs in shared memory; on the contracted kernel, several and one large; multi-source passes
for name, g, opts in (("small", G.pack_graphs(G.gen_ba_batch(60, 100, 300, seed=7))[:3], dict(mode=P.MODE_PLAIN)),
                      ("several", G.pack_graphs(G.gen_ba_batch(3, 9000, 12000, seed=8))[:3], dict(mode=P.MODE_PLAIN)),
                      ("large", G.gen_rmat(13, 16, chain_frac=0.2, chain_hi=8, seed=2), dict(mode=P.MODE_PLAIN)),
                      ("passes", G.pack_graphs(G.gen_ba_batch(3, 9000, 12000, seed=8))[:3], dict(mode=P.MODE_BATCHED))):
    d = decomp(*g)
    ctx = P.Context(**opts)
    L.stub_cudart_team_nomem(1)
    r = raises(lambda: ctx.plan(d).close())
    L.stub_cudart_team_nomem(0)
    out[name] = [r[0] if r else 0, raises(lambda: ctx.plan(d).close())]
    ctx.close()
""")
    assert {k: v[0] for k, v in res.items()} == {"small": 3, "several": 3, "large": 3, "passes": 3}  # BCGPU_ENOMEM
    assert all(v[1] is None for v in res.values())
