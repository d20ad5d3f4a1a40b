"""Row sums take leaves in any numbering: the lists of consecutive rows need not be consecutive
(nor lie in the range that the CTA stages).  Reference and tolerance as for lists in row order:
numpy sums in FP64, 2 K 2^-53 of the sum of magnitudes of a list of K."""
import numpy as np
import pytest

from pyquake3d_b200 import _lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["reversed", "random", "first_last"])
@pytest.mark.parametrize("n", [40, 700, 5000])
@pytest.mark.parametrize("code", [0, 1])
def test_leaf_numbering(n, order, code):
    rng = np.random.default_rng(n)
    cuts = [0]
    while cuts[-1] < n:
        cuts.append(min(n, cuts[-1] + int(rng.integers(1, 13))))
    nl = len(cuts) - 1
    ids = np.arange(nl)
    if order == "reversed":
        ids = ids[::-1].copy()
    elif order == "random":
        ids = rng.permutation(nl)
    else:                                   # only two leaves exchanged: some CTAs' ranges are far too wide
        ids[[0, nl - 1]] = ids[[nl - 1, 0]]
    row = np.repeat(ids, np.diff(cuts)).astype(np.int32)
    cnt = rng.integers(0, 31, nl)
    ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    off = np.concatenate([rng.permutation(30)[:c] for c in cnt]).astype(np.int32) * n
    nt = np.float64 if code == 0 else np.float32
    slots = rng.standard_normal((30 * n, 3)).astype(nt)
    d = {k: torch.tensor(v, device="cuda") for k, v in dict(row=row, ptr=ptr, off=off, slots=slots).items()}
    x = torch.zeros(4 * (n + 24), dtype=d["slots"].dtype, device="cuda")
    y = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    hp = np.zeros(1, dtype=_lib.HM_PLAN)
    hp["n"], hp["dtype"] = n, code
    hp["leaf_of_row"], hp["leaf_ptr"], hp["leaf_off"] = d["row"].data_ptr(), d["ptr"].data_ptr(), d["off"].data_ptr()
    _lib.check(_lib.load().pq3d_hmatvec(hp.ctypes.data, x.data_ptr(), d["slots"].data_ptr(), x.data_ptr(), None, None,
                                        None, y.data_ptr(), _lib.stream_ptr()), "pq3d_hmatvec")
    s = slots.astype(np.float64)
    got = y.cpu().numpy()
    for i in range(n):
        v = s[off[ptr[row[i]]:ptr[row[i] + 1]] + i]
        assert (np.abs(got[i] - v.sum(0)) <= 2 * (len(v) + 2) * 2.0 ** -53 * np.abs(v).sum(0)).all(), i
