"""The resident kernels at the limits of their dispatch: hubs on both sides of
the largest number of communities a block's table holds (14,336), rows longer
than the table whose vertices still see few communities (repeated neighbours),
and the class kernels beside them in every precision.  Bar: the oracle's run
bit for bit; the engine's two forms against one another where the precision is
not the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 14336  # communities a vertex may see in the resident kernels


def _same(a, b):
    assert (a["level_sizes"] == b["level_sizes"]).all() and a["iterations"] == b["iterations"]
    assert (a["trace"] == b["trace"]).all() and a["modularity"] == b["modularity"]
    assert (a["assignment"] == b["assignment"]).all()


def _multi(O, n, times, weighted):
    """Vertex 0 joined `times` times to every other one, the others in groups of
    seven whose pairs are joined twice as often: rows hold repeated neighbours
    (symmetric as a multiset)."""
    leaf = np.arange(1, n)
    i, j = np.triu_indices(7, 1)
    i, j = (np.arange(0, n, 7)[:, None] + 1 + np.stack([i, j])[:, None]).reshape(2, -1)
    m = j < n
    u = np.concatenate([np.zeros((n - 1) * times, np.int64), np.repeat(i[m], 2 * times)])
    v = np.concatenate([np.repeat(leaf, times), np.repeat(j[m], 2 * times)])
    row, col = np.concatenate([u, v]), np.concatenate([v, u])
    x = np.arange(len(u)) * 2654435761 % 5 + 1.0
    x = np.concatenate([x, x])
    o = np.argsort(row, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.uint64)
    return O.CSR(n, off, col[o].astype(np.uint32), x[o] if weighted else None)


def _run_both(O, ctx, g, resident):
    """Single runs and a batch of the graph twice against the oracle; whether
    the first level ran in the resident kernel shows in the launches."""
    refs = {v: O.louvain(g, version=v) for v in (1, 2)}
    dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights)
    b = ctx.batch_from_csr([(g.n, g.offsets, g.cols, g.weights)] * 2)
    for v, ref in refs.items():
        a = dg.louvain(version=v, max_phases=1)
        ctx.sweep_options(light_streams=1)
        try:
            c = dg.louvain(version=v, max_phases=1)
            _same(dg.louvain(version=v), ref)
        finally:
            ctx.sweep_options()
        _same(a, c)
        assert (a["kernel_launches"] < c["kernel_launches"]) == resident
        _same(dg.louvain(version=v), ref)
        r = b.run(version=v)
        for i in range(2):
            assert r["graphs"]["modularity"][i] == ref["modularity"]
            assert r["graphs"]["iterations"][i] == ref["iterations"]
            assert (r["assignments"][i] == ref["assignment"]).all()
    dg.close()
    b.close()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("degree", [CAP - 1, CAP, CAP + 1])
def test_hub_at_the_tables_limit(O, ctx, degree, weighted):
    _run_both(O, ctx, _multi(O, degree + 1, 1, weighted), degree <= CAP)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,times", [(20, 9), (20, 2000), (33, 40), (130, 70), (CAP, 2), (CAP + 1, 2)])
def test_rows_longer_than_the_table(O, ctx, n, times, weighted):
    _run_both(O, ctx, _multi(O, n, times, weighted), n <= CAP)


@pytest.mark.parametrize("version", [1, 2])
@pytest.mark.parametrize("precision", ["fp64", "int64", "fp32"])
@pytest.mark.parametrize("name", ["rmat", "sbm", "weights"])
def test_class_kernels_in_every_precision(O, ctx, name, precision, version):
    """Full runs of the class kernels (which every level too large for the
    resident one takes), with the table-free first sweep and without it, equal
    the resident kernel's."""
    g = {"rmat": lambda: O.gen_rmat(13, seed=5), "sbm": lambda: O.gen_sbm(9001, 24, 17.0, 0.8, seed=4),
         "weights": lambda: _multi(O, 900, 3, True)}[name]()
    dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights)
    a = dg.louvain(version=version, precision=precision)
    for table_first in (False, True):
        ctx.sweep_options(light_streams=1, table_first_sweep=table_first)
        try:
            _same(dg.louvain(version=version, precision=precision), a)
        finally:
            ctx.sweep_options()
    ref = O.louvain(g, version=version)
    assert abs(a["modularity"] - ref["modularity"]) <= 1e-3
    if precision == "fp64":
        _same(a, ref)
    dg.close()


@pytest.mark.parametrize("graphs", [False, True])
def test_batch_launch_modes_of_the_class_kernels(O, mg, ctx, graphs):
    """Batches of small graphs run resident by default, whatever launch mode is
    asked for; with the shapes fixed, both modes of the class kernels run."""
    from test_gpu_batch import _check_graph, _mixed_graphs, _pack

    gs = _mixed_graphs(O)
    b = _pack(ctx, gs)
    ctx.tune_mode(mg.TUNE_OFF)
    try:
        res = b.run(graphs=graphs)
    finally:
        ctx.tune_mode(mg.TUNE_ON)
    assert res["kernel_launches"] > b.run()["kernel_launches"]
    for i, g in enumerate(gs):
        if g.nnz:
            _check_graph(res, i, O.louvain(g))
    b.close()
