"""Sizes at which the device scan changes its launch form: bins on both sides
of 8,192 counts (one block up to there; a bin scheme has bins * ceil(n / 1024)
of them), relabelling on both sides of 512 tiles (1,048,576 items: the tiles'
sums are scanned above), with odd tails.  Bar: the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,bins", [(0, 10), (1, 11), (2, 9)])
def test_bins_around_one_block(O, ctx, scheme, bins):
    blocks = 8192 // bins
    assert blocks * bins <= 8192 < (blocks + 1) * bins
    for n in (blocks * 1024 - 1, blocks * 1024, blocks * 1024 + 1, (blocks + 1) * 1024 + 7):
        deg = np.random.default_rng(n).integers(0, 40, n)
        off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
        a, b = ctx.bins_offsets(scheme, off), O.bins(scheme, off)
        for key in ("sizes", "offsets", "perm"):
            assert (a[key] == b[key]).all(), (n, key)
        assert a["max_degree"] == b["max_degree"]


@pytest.mark.parametrize("n", [1048575, 1048576, 1048577, 1050625, 2097153, 3000001])
def test_relabel_around_the_scanned_sums(O, ctx, n):
    rng = np.random.default_rng(n)
    u = rng.integers(0, n, 5000)
    v = (u + rng.integers(1, n, 5000)) % n
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    g = O.csr_from_pairs(n, key // n, key % n, None)
    C = rng.choice(n, n // 3, replace=False)[rng.integers(0, n // 3, n)].astype(np.uint32)
    cd, g2 = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights).coarsen(C)
    cd_o, h, _ = O.coarsen(g, C)
    off, cols, wts = g2.csr()
    assert (cd == cd_o).all() and (off == h.offsets).all() and (cols == h.cols).all()
    assert (wts == h.weight_array()).all()
    g2.close()
