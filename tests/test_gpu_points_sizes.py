"""The drop-ins at the sizes where they change: CTAs of 128 receivers with ragged ends, the
mapped buffer (up to 1 MB, growing and reused by smaller calls) and direct copies above it, one
source or several, with and without strain.  The references are the device form of the same
entry point one source at a time (a source's records made once per CTA against once per
thread) and, at every size, the results of single-receiver calls: the same arithmetic, so
within 1e-12 of each receiver's largest component."""
import ctypes

import numpy as np
import pytest

from pyquake3d_b200 import _lib

pytestmark = pytest.mark.gpu
MU = LAM = 32e9
DP = ctypes.POINTER(ctypes.c_double)


def _p(a):
    return a.ctypes.data_as(DP)


def _points(n, seed):
    r = np.random.default_rng(seed)
    return [np.ascontiguousarray(v) for v in (r.uniform(-5e3, 5e3, n), r.uniform(-5e3, 5e3, n), r.uniform(-4e3, -50, n))]


def _call(L, x, P, half):
    n = len(x[0])
    s, e = np.full((n, 6), np.nan), np.full((n, 6), np.nan)
    L.TDstressFS_C(_p(x[0]), _p(x[1]), _p(x[2]), n, _p(P[0]), _p(P[1]), _p(P[2]), 1.0, -0.5, 0.25, MU, LAM, half,
                   _p(s), _p(e))
    return s, e


def _close(a, b):
    assert (np.abs(a - b) <= 1e-12 * np.abs(b).max(axis=1, keepdims=True)).all()


@pytest.mark.parametrize("half", [False, True])
def test_receiver_counts(half):
    L = _lib.load()
    P = [np.array(v) for v in ([-300.0, 10.0, -2500.0], [400.0, -20.0, -2300.0], [0.0, 200.0, -1500.0])]
    x = _points(9000, 3)
    big = _call(L, x, P, half)                       # above 1 MB
    for n in (1, 2, 127, 128, 129, 1000, 8700, 8738, 8739, 5):
        s, e = _call(L, [np.ascontiguousarray(v[:n]) for v in x], P, half)
        _close(s, big[0][:n])
        _close(e, big[1][:n])
    for i in (0, 4321, 8999):
        s, e = _call(L, [v[i:i + 1].copy() for v in x], P, half)
        _close(s, big[0][i:i + 1])


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n", [1, 2, 130, 5000])
def test_source_counts(half, n):
    L = _lib.load()
    r = np.random.default_rng(n)
    c = np.stack([r.uniform(-4e3, 4e3, n), r.uniform(-4e3, 4e3, n), r.uniform(-6e3, -1500, n)], 1)
    P = [np.ascontiguousarray(c + r.uniform(-400, 400, (n, 3))) for _ in range(3)]
    s, e = np.full((n, 6), np.nan), np.full((n, 6), np.nan)
    L.TDstressEachSourceAtReceiver_C(10.0, 20.0, -700.0, _p(P[0]), _p(P[1]), _p(P[2]), n, 1.0, -0.5, 0.25, MU, LAM,
                                     half, _p(s), _p(e))
    x = [np.array([v]) for v in (10.0, 20.0, -700.0)]
    for i in range(0, n, max(1, n // 7)):
        s1, e1 = _call(L, x, [q[i].copy() for q in P], half)
        _close(s[i:i + 1], s1)
        _close(e[i:i + 1], e1)
