"""Multi-source passes run several at a time on small cores: the whole range in
one call (merged) gives the BC of its passes run one call each (never merged),
and the oracle's; over widths that end on a whole group of words and widths
that do not (not merged), BCCs with a partial last pass, several BCCs in a row,
ranges that start and end inside a BCC, chain sources in every pass, and a
recorded graph. A pass's rows are still its own after a merged run."""
import numpy as np
import pytest

from helpers import graphs, oracle, pkg, rel_err

pytestmark = pytest.mark.gpu


def several():
    G = graphs()
    parts = [G.gen_rmat(8, 8, chain_frac=0.3, chain_hi=6, seed=1), G.gen_rmat(9, 8, chain_frac=0.2, chain_hi=9, seed=2),
             G.gen_small(3)]
    return G.pack_graphs(parts)[:3]


CASES = {
    "rmat": lambda: graphs().gen_rmat(10, 16, chain_frac=0.2, chain_hi=8, seed=5),
    "several": several,
    "grid": lambda: graphs().gen_grid(24, leaves=60, seed=4),
}


@pytest.mark.parametrize("name,width,delta", [("rmat", 128, "fp64"), ("rmat", 256, "fp32c"), ("rmat", 96, "fp64"),
                                              ("several", 128, "fp64"), ("several", 384, "fp32c"), ("grid", 128, "fp64")])
@pytest.mark.parametrize("graph", [False, True])
def test_merged_run_is_the_sum_of_its_passes(name, width, delta, graph):
    P = pkg()
    n, u, v = CASES[name]()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, batch_width=width, graph=graph,
                    delta=P.DELTA_FP64 if delta == "fp64" else P.DELTA_FP32C)
    tol = 1e-12 if delta == "fp64" else 1e-6
    plan = ctx.plan(d)
    k = plan.n_units
    for a, b in [(0, k), (1, k), (k // 3, max(k // 3 + 2, 2 * k // 3))]:
        b = min(b, k)
        outs = []
        for cuts in ([a, b], list(range(a, b + 1)), [a, b]):
            plan.reset()
            for i, j in zip(cuts, cuts[1:]):
                plan.run(i, j)
            outs.append(plan.read())
        assert np.array_equal(outs[0], outs[2])  # the same call, the same bits
        assert rel_err(outs[0], outs[1]) < tol
        one_shot, _ = ctx.run_units(d, a, b, with_art=True)  # its own plan, with the tables of these passes only
        assert np.array_equal(one_shot, outs[0])
        if (a, b) == (0, k):
            O = oracle()
            row, col = O.csr(n, u, v)
            assert rel_err(outs[0], O.brandes(n, row, col)) < tol
    plan.close()
    ctx.close()


def test_pass_rows_after_a_merged_run():
    P = pkg()
    n, u, v = CASES["rmat"]()
    d = P.Decomposition(P.Graph.from_edges(n, u, v))
    a = d.arrays()
    ctx = P.Context(mode=P.MODE_BATCHED, plain_core=-1, batch_width=128, delta=P.DELTA_FP64)
    plan = ctx.plan(d)
    plan.run()
    for unit in (0, plan.n_units // 2, plan.n_units - 1):
        src, dd, ss = plan.pass_rows(unit)
        for i in (0, len(src) - 1):
            do, so = oracle().bcc_source_rows(a, 0, int(src[i]))
            nc = dd.shape[1]
            assert np.array_equal(dd[i], do[:nc]) and np.array_equal(ss[i], so[:nc])
    plan.close()
    ctx.close()
