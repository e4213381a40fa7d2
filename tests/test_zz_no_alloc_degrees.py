"""mg_local_move_noalloc at the degrees where its kernels take over from one
another (8 lanes, a warp, 256 threads, a CTA, the scratch tables): bit-exact
against the oracle for unit and integer weights, both versions and
directions, from the level's start and from a later assignment."""
import numpy as np
import pytest

from test_zz_no_alloc import _dev, _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("degrees", [(1, 7, 8, 9, 15, 16, 17), (31, 32, 33, 63, 64, 65), (255, 256, 257, 300),
                                     (2047, 2048, 2049, 5000), (10921, 10922, 10923, 16384, 16385)])
def test_degrees(O, mg, degrees, weighted):
    import torch

    f = _noalloc(mg)
    rng = np.random.default_rng(sum(degrees))
    h, leaves = len(degrees), max(degrees) + 37
    u = [np.arange(leaves) + h] + [np.full(d, i) for i, d in enumerate(degrees)]
    v = [(np.arange(leaves) + 1) % leaves + h] + [h + rng.choice(leaves, d, replace=False) for d in degrees]
    u, v = np.concatenate(u), np.concatenate(v)
    name = rng.permutation(h + leaves)
    w = rng.integers(1, 7, len(u)).astype(np.float64) if weighted else None
    g = O.csr_from_pairs(h + leaves, name[u], name[v], w)
    k, mass = O.vertex_weights(g), O.mass(g)
    d_off, d_col, d_k = _dev(torch, g.offsets, np.int32), _dev(torch, g.cols, np.int32), _dev(torch, k, np.float64)
    d_w = _dev(torch, g.weights, np.float64) if weighted else None
    C = np.arange(g.n, dtype=np.uint32)
    for start in range(2):
        sig = np.zeros(g.n)
        np.add.at(sig, C, k)
        d_C, d_s = _dev(torch, C, np.int32), _dev(torch, sig, np.float64)
        for version, up in ((2, True), (2, False), (1, True), (1, False)):
            d_out = torch.full((g.n,), -1, dtype=torch.int32, device="cuda")
            st = f(g.n, d_off.data_ptr(), d_col.data_ptr(), d_w.data_ptr() if weighted else None, mass, d_C.data_ptr(),
                   d_s.data_ptr(), d_k.data_ptr(), d_out.data_ptr(), version, int(up), None)
            assert st == 0
            torch.cuda.synchronize()
            want, _ = O.local_move(g, C, sig, k, mass, version, up)
            got = d_out.cpu().numpy().view(np.uint32)
            assert (got == want).all(), (start, version, up, np.nonzero(got != want)[0][:10])
        C = rng.integers(0, max(1, g.n // 9), g.n).astype(np.uint32)
