"""Modularity of assignments on graphs of mostly empty rows, on both sides of the
number of rows per tile of edges at which edges search their rows one by one:
the oracle's value, bit for bit on integral weights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["unit", "int", "real", "f32"])
@pytest.mark.parametrize("n,pairs", [(65535, 50), (65536, 50), (65537, 1), (70001, 2047), (131073, 2500), (131071, 2500),
                                     (1000003, 20), (1000003, 9000), (5000011, 40000), (5000011, 200000)])
def test_modularity_of_sparse_graphs(O, ctx, n, pairs, kind):
    rng = np.random.default_rng(n + pairs)
    u = rng.integers(0, n, pairs)
    u[: pairs // 2] = n - 1  # a hub at the end, empty rows before it
    v = (u + rng.integers(1, n, pairs)) % n
    key = np.unique(np.minimum(u, v) * n + np.maximum(u, v))
    w = None if kind == "unit" else rng.integers(1, 9, len(key)).astype(np.float64)
    if kind in ("real", "f32"):
        w = (rng.random(len(key)) + 0.5).astype(np.float32).astype(np.float64)
    g = O.csr_from_pairs(n, key // n, key % n, w)
    dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights.astype(np.float32) if kind == "f32" else g.weights)
    for C in (np.arange(n), np.zeros(n, np.int64), rng.integers(0, n, n), np.arange(n) % 7):
        C = C.astype(np.uint32)
        q, ref = dg.modularity(C), O.modularity(g, C)
        assert q == ref if kind in ("unit", "int") else abs(q - ref) < 1e-12
    dg.close()
