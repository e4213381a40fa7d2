"""What a context keeps of the graphs and results that ended: the newest buffers
within the limits, given back by mg_trim and when another context's allocation
finds no memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 256 << 20


def _ring(n):
    """CSR of a ring with four neighbours per vertex."""
    v = np.arange(n, dtype=np.int64)
    cols = np.sort(np.stack([(v - 2) % n, (v - 1) % n, (v + 1) % n, (v + 2) % n], 1), 1).ravel()
    return np.arange(n + 1, dtype=np.uint64) * 4, cols.astype(np.uint32)


def test_the_newest_buffers_are_kept(mg):
    c = mg.Context(0)
    for i in range(40):  # more sizes than places
        n = int(50 * 1.25**i)
        c.graph_from_csr(n, *_ring(n)).close()
        assert c.graph_from_csr(9, *_ring(9)).info()["nnz"] == 36
    n = 6 << 20
    c.graph_from_csr(n, *_ring(n)).close()
    device, _ = c.trim()
    assert 16 * n <= device <= LIMIT  # its columns are among them
    assert c.trim()[0] == 0
    c.close()


def test_limits(mg):
    c = mg.Context(0)
    for n in (5 << 20, 7 << 20, 11 << 20, 13 << 20):
        c.graph_from_csr(n, *_ring(n)).close()
    assert 0 < c.trim()[0] <= LIMIT
    c.close()


def test_trim_of_a_used_context(O, mg):
    c = mg.Context(0)
    g = O.gen_sbm(300000, 50, 8.0, 0.8, seed=3)
    dg = c.graph_from_csr(g.n, g.offsets, g.cols, None)
    a = dg.louvain()
    device, host = c.trim()
    assert host >= 4 * g.n
    b = dg.louvain()
    assert b["modularity"] == a["modularity"] and (b["assignment"] == a["assignment"]).all()
    dg.close()
    c.close()


def test_another_contexts_allocation_gets_the_memory(mg):
    import torch

    n = 4 << 20
    off, cols = _ring(n)
    a, b = mg.Context(0), mg.Context(0)
    for c in (a, b):
        c.graph_from_csr(n, off, cols).close()
    b.trim()
    torch.cuda.synchronize()
    left = 24 << 20  # less than the columns of the graph
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 16 * n
        g = b.graph_from_csr(n, off, cols)
        assert g.info()["nnz"] == 4 * n
        assert a.trim()[0] == 0
        g.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    a.close()
    b.close()


def test_a_failed_call_leaves_no_copy_in_flight(mg):
    """The third allocation of an upload fails while the offsets (240 MB of
    page-locked memory, 4 ms on the link) are being copied: they are the
    caller's again when the call returns, so the device is idle then."""
    import time

    import torch

    n = 30_000_000
    off = torch.zeros(n + 1, dtype=torch.int64).pin_memory().numpy().view(np.uint64)
    c = mg.Context(0)
    c.graph_from_csr(n, off, np.zeros(0, np.uint32)).close()
    torch.cuda.synchronize()
    for _ in range(3):
        c.trim()
        mg.fail_allocation(3)
        try:
            with pytest.raises(mg.MGError) as e:
                c.graph_from_csr(n, off, np.zeros(0, np.uint32))
            t0 = time.perf_counter()
            torch.cuda.synchronize()
            waited = time.perf_counter() - t0
        finally:
            assert mg.fail_allocation(0) == 0
        assert e.value.status == 3 and waited < 1e-3, waited
    assert c.graph_from_csr(9, *_ring(9)).info()["nnz"] == 36
    c.close()


def test_a_workspace_grows_without_slack_on_a_full_device(mg):
    """A workspace that grows for a slightly larger graph takes no more memory
    than a new one when little of the device's memory is left."""
    import torch

    def used(sizes):
        c = mg.Context(0)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        for n in sizes:
            g = c.generate_sbm(n, 64, 16.0, 0.8, seed=1)
            g.louvain()
            g.close()
            c.trim()
        after = torch.cuda.mem_get_info()[0]
        c.close()
        return before - after

    used([100000])
    free, total = torch.cuda.mem_get_info()
    hold = torch.empty(free - (total // 16 - (1 << 30)), dtype=torch.uint8, device="cuda")
    try:
        assert used([3000000, 3300000]) < used([3300000]) + (64 << 20)
    finally:
        del hold
        torch.cuda.empty_cache()
