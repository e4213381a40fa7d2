"""The resident level kernel (all iterations of a small level in one launch):
hubs on both sides of every degree at which a vertex changes hands (lanes of a
warp, a warp, 128 or 256 threads, the CTA, too large for the kernel), levels
that need more iterations than one launch holds, tiny levels.  Bar: the
oracle's run bit for bit on integral weights, which the class kernels (forced
with sweep_options) give as well; real weights within the engine's bounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hubs(O, degrees, weighted, seed=1):
    """Hubs of the given degrees joined to random leaves, leaves in a ring."""
    rng = np.random.default_rng(seed)
    h, leaves = len(degrees), max(max(degrees), 64) + 11
    u, v = [np.arange(leaves) + h], [(np.arange(leaves) + 1) % leaves + h]
    for i, d in enumerate(degrees):
        u.append(np.full(d, i))
        v.append(h + rng.choice(leaves, d, replace=False))
    u, v = np.concatenate(u), np.concatenate(v)
    w = rng.integers(1, 9, len(u)).astype(np.float64) if weighted else None
    return O.csr_from_pairs(h + leaves, u, v, w)


def _same(a, b):
    assert (a["level_sizes"] == b["level_sizes"]).all() and a["iterations"] == b["iterations"]
    assert (a["trace"] == b["trace"]).all() and a["modularity"] == b["modularity"]
    assert (a["assignment"] == b["assignment"]).all()


def _check(O, ctx, g, versions=(1, 2)):
    dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights)
    for version in versions:
        ref = O.louvain(g, version=version)
        _same(dg.louvain(version=version), ref)
        ctx.sweep_options(light_streams=1)
        try:
            _same(dg.louvain(version=version), ref)
        finally:
            ctx.sweep_options()
    dg.close()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("degrees", [(1, 2, 3, 4, 5, 8, 9), (16, 17, 31, 32, 33, 34), (63, 64, 65, 66, 127, 128, 129),
                                     (255, 256, 257, 511, 512, 513), (1023, 1024, 1025, 2047, 2048, 2049),
                                     (4095, 4096, 4097, 8191, 8193), (10921, 10922, 10923), (16385, 300)])
def test_degrees(O, ctx, degrees, weighted):
    _check(O, ctx, _hubs(O, degrees, weighted))


@pytest.mark.parametrize("n,blocks", [(2, 1), (3, 1), (33, 2), (1013, 4), (20011, 40)])
def test_sizes(O, ctx, n, blocks):
    # (20,011 vertices: more iterations in a level than one launch holds)
    _check(O, ctx, O.gen_sbm(n, blocks, 12.0, 0.7, seed=5))


def test_thresholds(O, ctx):
    g = O.gen_sbm(5000, 16, 14.0, 0.8, seed=2)
    dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, None)
    for thr in (0.0, 1e-9, 1e-2, 10.0):
        _same(dg.louvain(threshold=thr), O.louvain(g, threshold=thr))


@pytest.mark.parametrize("f32", [False, True])
def test_real_weights(O, ctx, f32):
    g = O.gen_chunglu(1 << 14, max_degree=3000.0, seed=3)
    w = g.weights.astype(np.float32) if f32 else g.weights
    a = ctx.graph_from_csr(g.n, g.offsets, g.cols, w).louvain()
    assert abs(a["modularity"] - O.louvain(g)["modularity"]) < 1e-3
    assert abs(O.modularity(g, a["assignment"]) - a["modularity"]) < 1e-9
