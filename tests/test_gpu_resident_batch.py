"""Batches whose graphs each run on a cluster of blocks (the resident batch
kernel) against the same graphs alone and against the class kernels (used when
the caller fixes the shapes), bit for bit: graph counts and sizes that take
clusters of one to eight blocks, more graphs than clusters, empty and tiny
graphs, weights, both versions, many iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(ctx, gs, **kw):
    b = ctx.batch_from_csr([(g.n, g.offsets, g.cols, g.weights) for g in gs])
    r = b.run(**kw)
    b.close()
    return r


def _same(r, refs):
    for i, ref in enumerate(refs):
        assert r["graphs"]["modularity"][i] == ref["modularity"], i
        assert r["graphs"]["iterations"][i] == ref["iterations"], i
        assert (r["assignments"][i] == ref["assignment"]).all(), i


def _alone(O, g, **kw):
    if g.nnz == 0:  # no edges: the identity, Q = 0 (the oracle's Q is 0 / 0)
        return dict(modularity=0.0, iterations=0, assignment=np.arange(g.n))
    return O.louvain(g, **kw)


def _weighted(O, g, seed):
    row = np.repeat(np.arange(g.n), np.diff(g.offsets).astype(np.int64))
    m = row < g.cols
    return O.csr_from_pairs(g.n, row[m], g.cols[m], np.random.default_rng(seed).integers(1, 9, m.sum()).astype(float))


@pytest.mark.parametrize("version", [1, 2])
@pytest.mark.parametrize("sizes", [(1,), (2, 1, 3), (33,) * 5, (1000,) * 200, (30011, 500, 17), (3000, 9000, 40) * 9])
def test_graph_counts_and_sizes(O, mg, ctx, sizes, version):
    gs = [O.gen_sbm(n, min(n, 4 + i % 13), 6.0 + i % 19, 0.75, seed=i + 1) for i, n in enumerate(sizes)]
    refs = [_alone(O, g, version=version) for g in gs]
    _same(_batch(ctx, gs, version=version), refs)
    ctx.tune_mode(mg.TUNE_OFF)
    try:
        for graphs in (True, False):
            _same(_batch(ctx, gs, version=version, graphs=graphs), refs)
    finally:
        ctx.tune_mode(mg.TUNE_ON)


def test_weights_hubs_and_empty_graphs(O, ctx):
    empty = O.CSR(5, np.zeros(6, np.uint64), np.zeros(0, np.uint32), None)
    hub = O.csr_from_pairs(3001, np.zeros(3000, np.int64), np.arange(1, 3001))
    gs = [O.gen_rmat(12, seed=3), empty, hub, O.gen_sbm(4001, 30, 20.0, 0.8, seed=6), O.gen_rmat(10, seed=8)]
    gs = [g if g is empty else _weighted(O, g, i) for i, g in enumerate(gs)]
    _same(_batch(ctx, gs), [_alone(O, g) for g in gs])


def test_real_weights(O, ctx):
    gs = [O.gen_chunglu(1 << 12, max_degree=500.0, seed=s) for s in range(1, 7)]
    r = _batch(ctx, gs)
    for i, g in enumerate(gs):
        assert abs(r["graphs"]["modularity"][i] - O.louvain(g)["modularity"]) < 1e-3
        assert abs(O.modularity(g, r["assignments"][i]) - r["graphs"]["modularity"][i]) < 1e-9
