"""Drop-in calls on both sides of the sizes where their buffers change (mapped memory, one copy
each way, the caller's arrays directly), with and without strain: every receiver and source
gets bitwise what a small call gives it, and a call without strain the stress of one with it."""
import ctypes

import numpy as np
import pytest

from pyquake3d_b200 import _lib

pytestmark = pytest.mark.gpu
MU = LAM = 32e9
DP = ctypes.POINTER(ctypes.c_double)


def _p(a):
    return None if a is None else a.ctypes.data_as(DP)


def _out(n, strain):
    return np.full((n, 6), np.nan), np.full((n, 6), np.nan) if strain else None


def _same(whole, part, lo, hi):
    for w, p in zip(whole, part):
        assert (w is None) == (p is None)
        if w is not None:
            assert np.array_equal(w[lo:hi], p)


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n", [5999, 6000, 6001, 7500, 8738, 8739, 14563, 14564])
def test_receivers(n, half):
    L = _lib.load()
    r = np.random.default_rng(n)
    x = [np.ascontiguousarray(v) for v in (r.uniform(-5e3, 5e3, n), r.uniform(-5e3, 5e3, n), r.uniform(-4e3, -50, n))]
    P = [np.array(v) for v in ([-300.0, 10.0, -2500.0], [400.0, -20.0, -2300.0], [0.0, 200.0, -1500.0])]

    def call(lo, hi, strain):
        y = [np.ascontiguousarray(v[lo:hi]) for v in x]
        s, e = _out(hi - lo, strain)
        L.TDstressFS_C(_p(y[0]), _p(y[1]), _p(y[2]), hi - lo, _p(P[0]), _p(P[1]), _p(P[2]), 1.0, -0.5, 0.25, MU, LAM,
                       half, _p(s), _p(e))
        return s, e
    both, one = call(0, n, True), call(0, n, False)
    assert np.isfinite(both[0]).all() and np.isfinite(both[1]).all() and np.array_equal(both[0], one[0])
    for lo in (0, n // 2, n - 130):
        _same(both, call(lo, lo + 130, True), lo, lo + 130)


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n", [1, 129, 6000, 6001, 6241, 6242])
def test_sources(n, half):
    L = _lib.load()
    r = np.random.default_rng(n)
    c = r.uniform(-1, 1, (n, 3)) * [5e3, 5e3, 1e3] - [0, 0, 3e3]
    P = [np.ascontiguousarray(c + r.uniform(-200, 200, (n, 3))) for _ in range(3)]

    def call(lo, hi, strain):
        Q = [np.ascontiguousarray(p[lo:hi]) for p in P]
        s, e = _out(hi - lo, strain)
        L.TDstressEachSourceAtReceiver_C(100.0, -50.0, -900.0, _p(Q[0]), _p(Q[1]), _p(Q[2]), hi - lo, 1.0, -0.5, 0.25,
                                         MU, LAM, half, _p(s), _p(e))
        return s, e
    both, one = call(0, n, True), call(0, n, False)
    assert np.isfinite(both[0]).all() and np.isfinite(both[1]).all() and np.array_equal(both[0], one[0])
    if n > 130:
        for lo in (0, n - 130):
            _same(both, call(lo, lo + 130, True), lo, lo + 130)
