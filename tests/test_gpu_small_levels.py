"""Sizes at which the device scan and sort change their launch form (one block,
a sum per tile, scanned tile sums; one-block sort, tiled sort): bins and
coarsening around them against the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 8191, 8192, 8193, 441343, 441344, 1048577])
def test_bins_sizes(O, ctx, n):
    deg = np.random.default_rng(n).integers(0, 70, n)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    for scheme in (0, 1, 2):
        a, b = ctx.bins_offsets(scheme, off), O.bins(scheme, off)
        for key in ("sizes", "offsets", "perm"):
            assert (a[key] == b[key]).all(), (n, scheme, key)
        assert a["max_degree"] == b["max_degree"]


@pytest.mark.parametrize("kind", ["unit", "int", "real"])
@pytest.mark.parametrize("pairs", [1, 2047, 4095, 4096, 4097, 9000, 40000])
def test_coarsen_sizes(O, ctx, pairs, kind):
    rng = np.random.default_rng(pairs)
    n = max(3, pairs // 3)
    u = rng.integers(0, n, pairs)
    v = (u + rng.integers(1, n, pairs)) % n
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    key = np.unique(lo.astype(np.int64) * n + hi)
    w = None if kind == "unit" else rng.integers(1, 9, len(key)).astype(np.float64) if kind == "int" else rng.random(len(key)) + 0.5
    g = O.csr_from_pairs(n, key // n, key % n, w)
    C = rng.integers(0, max(1, n // 4), n).astype(np.uint32)
    cd, g2 = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights).coarsen(C)
    cd_o, h, _ = O.coarsen(g, C)
    off, cols, wts = g2.csr()
    assert (cd == cd_o).all() and (off == h.offsets).all() and (cols == h.cols).all()
    if kind == "real":  # sums of at most a few thousand doubles
        np.testing.assert_allclose(wts, h.weight_array(), rtol=1e-12)
    else:
        assert (wts == h.weight_array()).all()


@pytest.mark.parametrize("kind", ["unit", "int", "real"])
@pytest.mark.parametrize("n,pairs", [(2, 1), (5, 6), (300, 1000), (1500, 4095), (1500, 4096), (1500, 4097),
                                     (8191, 2000), (8192, 2000), (8193, 2000), (90, 3900)])
def test_small_runs(O, ctx, n, pairs, kind):
    """Runs whose levels lie on both sides of the one-block step from level to
    level (8,192 vertices or entries): the oracle's run, and every level's
    graph the oracle's coarsening of the level before."""
    rng = np.random.default_rng(n + pairs)
    key = np.unique(rng.integers(0, n * (n - 1) // 2, 4 * pairs))[:]
    key = rng.permutation(key)[:pairs]
    hi = ((1 + np.sqrt(1 + 8 * key.astype(np.float64))) // 2).astype(np.int64)
    hi -= hi * (hi - 1) // 2 > key
    lo = key - hi * (hi - 1) // 2
    w = None if kind == "unit" else rng.integers(1, 9, len(key)).astype(np.float64) if kind == "int" else rng.random(len(key)) + 0.5
    g = O.csr_from_pairs(n, lo, hi, w)
    a = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights).louvain(keep_levels=2)
    cur = g
    for lvl, (off, cols, wts) in enumerate(a["level_csr"]):
        assert (off == cur.offsets).all() and (cols == cur.cols).all()
        if kind == "real":  # sums of at most a few thousand doubles a level
            np.testing.assert_allclose(wts, cur.weight_array(), rtol=1e-11)
        else:
            assert (wts == cur.weight_array()).all()
        if lvl + 1 < len(a["level_csr"]):
            _, cur, _ = O.coarsen(cur, a["level_maps"][lvl])
    b = O.louvain(g)
    if kind == "real":
        assert abs(a["modularity"] - b["modularity"]) < 1e-3
        assert abs(O.modularity(g, a["assignment"]) - a["modularity"]) < 1e-9
    else:
        assert (a["level_sizes"] == b["level_sizes"]).all() and (a["trace"] == b["trace"]).all()
        assert (a["assignment"] == b["assignment"]).all()
