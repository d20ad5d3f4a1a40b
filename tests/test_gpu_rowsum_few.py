"""The row reduction of few rows with short lists (one thread a row) beside its other splits: list
lengths on both sides of a batch a row, row counts on both sides of 256.  Reference and
tolerance: numpy sums in FP64, 2 K 2^-53 of the sum of magnitudes of a list of K."""
import numpy as np
import pytest

from pyquake3d_b200 import _lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 16, 17, 255, 256, 257, 300])
@pytest.mark.parametrize("length", [1, 7, 8, 9, 20])
@pytest.mark.parametrize("code", [0, 1, 2])
def test_short_lists(n, length, code):
    rng = np.random.default_rng(n + length)
    cuts = np.minimum(np.arange(0, n + 12, 12), n)
    cuts = np.unique(cuts)
    nl = len(cuts) - 1
    row = np.repeat(np.arange(nl), np.diff(cuts)).astype(np.int32)
    ptr = (length * np.arange(nl + 1)).astype(np.int32)
    off = np.concatenate([rng.permutation(length) for _ in range(nl)]).astype(np.int32) * n
    slots = rng.standard_normal((length * n, 3)).astype(np.float64 if code == 0 else np.float32)
    add = rng.standard_normal((3, n))
    d = {k: torch.tensor(v, device="cuda") for k, v in dict(row=row, ptr=ptr, off=off, slots=slots, add=add).items()}
    x = torch.zeros(4 * (n + 24), dtype=d["slots"].dtype, device="cuda")
    y = torch.full((n + 4, 3), -7.0, dtype=torch.float64, device="cuda")
    hp = np.zeros(1, dtype=_lib.HM_PLAN)
    hp["n"], hp["dtype"], hp["n_slots"] = n, code, length * n
    hp["leaf_of_row"], hp["leaf_ptr"], hp["leaf_off"] = d["row"].data_ptr(), d["ptr"].data_ptr(), d["off"].data_ptr()
    _lib.check(_lib.load().pq3d_hmatvec(hp.ctypes.data, x.data_ptr(), d["slots"].data_ptr(), x.data_ptr(),
                                        d["add"][0].data_ptr(), d["add"][1].data_ptr(), None, y.data_ptr(),
                                        _lib.stream_ptr()), "pq3d_hmatvec")
    s = slots.astype(np.float64).reshape(length, n, 3)
    ref, mag = s.sum(0), np.abs(s).sum(0)
    ref[:, :2] += add[:2].T
    got = y.cpu().numpy()
    assert (np.abs(got[:n] - ref) <= 2 * (length + 2) * 2.0 ** -53 * (mag + np.abs(add.T))).all()
    assert (got[n:] == -7.0).all()
