"""The rules that choose between the resident and the class kernels, on the
CPU.  The measured times (ms of a phase on a B200, by CTAs per graph, 0 = the
class kernels) are of SBM batches whose graphs' sizes are log-uniform: the
choice is never more than 3 % slower than the class kernels, which served every
batch before there was a choice."""
import ctypes as ct

import numpy as np
import pytest

UNIT, INTEGER, REAL = 0, 1, 2


def _team(mg, loads, weights, sms=148):
    a, out = np.ascontiguousarray(loads, np.uint64), ct.c_int(-1)
    assert mg.lib().mg_test_batch_team(len(a), a.ctypes.data_as(ct.c_void_p), int(weights != REAL), sms,
                                       ct.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("graphs,lo,hi,weights,ms", [
    (200, 1000, 8000, UNIT, {0: 9.28, 1: 17.85, 2: 4.24, 4: 4.33, 8: 5.79}),
    (200, 1000, 8000, INTEGER, {0: 10.78, 1: 16.73, 2: 6.71, 4: 6.11, 8: 7.60}),
    (200, 1000, 8000, REAL, {0: 13.41, 1: 30.11, 2: 15.17, 4: 8.99, 8: 11.39}),
    (48, 8000, 50000, UNIT, {0: 17.33, 1: 72.91, 2: 37.36, 4: 19.64, 8: 13.08}),
    (48, 8000, 50000, REAL, {0: 30.86, 1: 413.69, 2: 210.41, 4: 109.75, 8: 57.66}),
    (24, 30000, 60000, UNIT, {0: 17.31, 1: 92.17, 2: 47.67, 4: 24.45, 8: 14.96}),
    (24, 30000, 60000, REAL, {0: 19.03, 1: 209.57, 2: 106.51, 4: 54.19, 8: 27.89}),
    (96, 8000, 100000, REAL, {0: 73.7, 1: 643.85, 2: 326.41, 4: 167.25, 8: 88.23}),
    (256, 1000, 100000, REAL, {0: 119.43, 1: 1296.2, 2: 660.74, 4: 337.21, 8: 174.54}),
])
def test_batch_team(mg, graphs, lo, hi, weights, ms):
    loads = np.geomspace(lo, hi, graphs) * 24  # 20 entries per vertex, and 4 per vertex
    assert ms[_team(mg, loads, weights)] <= 1.03 * ms[0]


def test_batch_team_bounds(mg):
    assert _team(mg, [], UNIT) in (0, 1, 2, 4, 8)
    for weights in (UNIT, INTEGER, REAL):
        assert _team(mg, [2**40], weights) == 0  # one graph too large for a cluster
        assert _team(mg, [20000] * 500, weights) in (1, 2, 4, 8)
        for sms in (1, 7, 8, 20, 148):
            assert _team(mg, [20000] * 50, weights, sms) in (0, 1, 2, 4, 8)
    out = ct.c_int()
    assert mg.lib().mg_test_batch_team(1, None, 1, 148, ct.byref(out)) != 0
    assert mg.lib().mg_test_batch_team(0, None, 1, 0, ct.byref(out)) != 0


def _resident(mg, n, nnz, max_degree, integral):
    out = ct.c_int(-1)
    assert mg.lib().mg_test_level_resident(n, nnz, max_degree, int(integral), ct.byref(out)) == 0
    return out.value


# ms of whole runs on a B200: resident kernels, class kernels (Chung-Lu graphs)
@pytest.mark.parametrize("n,nnz,max_degree,integral,res,cls", [
    (50000, 913494, 8000, False, 4.25, 7.09), (400000, 7806736, 8000, False, 11.07, 14.41),
    (600000, 11672752, 12000, False, 24.88, 29.09), (600000, 11672752, 12000, False, 23.00, 24.48),
    (800000, 15774034, 8000, False, 22.64, 22.24), (800000, 15774034, 8000, False, 15.32, 14.85),
    (900000, 17630442, 12000, False, 42.33, 40.94), (900000, 17630442, 12000, False, 28.41, 26.68),
    (1000000, 19764904, 8000, False, 31.00, 29.79),  # (class kernels: an earlier form of them)
    (900000, 17630442, 12000, True, 44.97, 55.60), (900000, 17630442, 12000, True, 29.66, 35.93),
])
def test_level_resident(mg, n, nnz, max_degree, integral, res, cls):
    assert _resident(mg, n, nnz, max_degree, integral) == (res < cls)


def test_level_resident_bounds(mg):
    for integral, most in ((True, 20 << 20), (False, 14 << 20)):
        assert _resident(mg, 10**6, most, 500, integral) == 1
        assert _resident(mg, 10**6, most + 1, 500, integral) == 0
    assert _resident(mg, 0, 0, 0, True) == 0
    assert _resident(mg, 10**6, 10**6, 14336, True) == 1 and _resident(mg, 10**6, 10**6, 14337, True) == 0
    assert _resident(mg, 14336, 10**6, 10**6, True) == 1


def test_batch_team_of_the_large_batch(mg):
    # 4,096 unit-weight graphs of 1,000 to 200,000 vertices: 2.535 s with four CTAs a graph, 2.735 s with eight
    assert _team(mg, np.geomspace(1000, 200000, 4096) * 24, UNIT) == 4
