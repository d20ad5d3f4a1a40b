"""Work items hold slot numbers, t positions, scale positions and row counts in 32 bits.  A plan
beyond that is refused with OverflowError before any item is made, and one that just fits is
not.  The structures are stand-ins: blocks with index ranges of the sizes in question."""
from types import SimpleNamespace as NS

import numpy as np
import pytest

from pyquake3d_b200 import _lib
from pyquake3d_b200.hmatrix import _dense_items, build_plan_arrays, build_plan_arrays_mixed

LIM = 2 ** 31 - 1


def _struct(m, n, nblocks):
    """Low-rank blocks of m x n, all on the same rows; one leaf."""
    rows, cols = NS(indices=range(m), start=0), NS(indices=range(n), start=0)
    return NS(n=max(m, 8), blocks=[NS(aca=True, row=rows, col=cols) for _ in range(nblocks)],
              leaves=[NS(start=0, leaf_id=0, indices=range(8))])


def _no_dense():
    return np.zeros(0, dtype=_lib.DENSE_BLOCK)


@pytest.mark.parametrize("code", [0, 1, 2])
def test_slots(code):
    s = _struct(2 ** 30, 8, 3)
    one = np.ones(3, np.int64)
    with pytest.raises(OverflowError):
        build_plan_arrays(s, _no_dense(), one, one, code, u_rows=2 ** 30)


def test_slots_mixed():
    s = _struct(2 ** 30, 8, 3)
    counts = np.ones((3, 2, 3), np.int64)
    with pytest.raises(OverflowError):
        build_plan_arrays_mixed(s, _no_dense(), None, u_rows=2 ** 30, counts=counts)


@pytest.mark.parametrize("code", [0, 1, 2])
def test_t_positions(code):
    # 4 blocks of 2^15 terms and 2^16 columns in chunks of one column group: 2^31 and more
    s = _struct(8, 2 ** 16, 4)
    k = np.full(4, 2 ** 14)
    with pytest.raises(OverflowError):
        build_plan_arrays(s, _no_dense(), k, k, code, v_chunk=1)


def test_t_positions_mixed():
    # a V class array has four or more entries per t position: its own limit comes first
    s = _struct(8, 2 ** 16, 4)
    with pytest.raises(_lib.Pq3dError):
        build_plan_arrays_mixed(s, _no_dense(), None, v_chunk=1, counts=np.full((4, 2, 3), 2 ** 14))


def test_dense_slots():
    recs = np.zeros(1, dtype=_lib.DENSE_BLOCK)
    recs["m"], recs["n"] = 2 ** 20, 2 ** 13
    with pytest.raises(OverflowError):
        _dense_items(recs, 4, recs["off32"], 1)           # 2^20 rows x 2^11 chunks = 2^31 slots


def test_just_below_the_limit():
    s = _struct(8, 64, 1)
    k = np.array([2 ** 10])
    A = build_plan_arrays(s, _no_dense(), k, k, 1, v_chunk=1)
    assert A["n_tpart"] == 16 * 6 * 2 ** 10 and (A["vitems"]["tp"][:A["n_vitems"]] < A["n_tpart"]).all()
    recs = np.zeros(1, dtype=_lib.DENSE_BLOCK)
    recs["m"], recs["n"] = 33, 64
    items, rows, n = _dense_items(recs, 4, recs["off32"], 1)
    assert n == 16 * 33 and int(items["slot"].max()) == 15 * 33 and n <= LIM
