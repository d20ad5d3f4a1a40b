"""The row reduction of the H-matvec's slots at the sizes where its split changes (16-row
CTAs, 80-row CTAs, short last CTA, lists below and above a batch, lists too long to stage),
and inside the step kernel for several grids, against numpy sums in FP64.

Tolerance: sums of K FP64 values in another order differ by at most 2 K 2^-53 of the sum of
magnitudes (the FP32 slots are widened before they are added)."""
import numpy as np
import pytest

from pyquake3d_b200 import _lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _lists(n, leaf, longest, rng):
    """leaf_of_row, leaf_ptr, leaf_off of n rows in leaves of up to `leaf` rows, each owner
    writing n slots (its offset is a multiple of n), lists of 0 to `longest` owners."""
    cuts = [0]
    while cuts[-1] < n:
        cuts.append(min(n, cuts[-1] + int(rng.integers(1, leaf + 1))))
    row = np.repeat(np.arange(len(cuts) - 1), np.diff(cuts)).astype(np.int32)
    cnt = rng.integers(0, longest + 1, len(cuts) - 1)
    cnt[0] = longest
    ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    off = np.concatenate([rng.permutation(longest)[:c] for c in cnt]).astype(np.int32) * n
    return row, ptr, off


@pytest.mark.parametrize("n,longest", [(1, 3), (15, 16), (16, 1), (17, 17), (81, 40), (1000, 130), (9473, 20),
                                       (500, 400)])
@pytest.mark.parametrize("code", [0, 1])
def test_rowsum(n, longest, code):
    rng = np.random.default_rng(n + longest)
    row, ptr, off = _lists(n, 16, longest, rng)
    tt, nt = (torch.float64, np.float64) if code == 0 else (torch.float32, np.float32)
    slots = rng.standard_normal((longest * n, 3)).astype(nt)
    add = rng.standard_normal((3, n))
    d = {k: torch.tensor(v, device="cuda") for k, v in dict(row=row, ptr=ptr, off=off, slots=slots, add=add).items()}
    x = torch.zeros(4 * (n + 24), dtype=tt, device="cuda")
    y = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    hp = np.zeros(1, dtype=_lib.HM_PLAN)
    hp["n"], hp["dtype"] = n, code
    hp["leaf_of_row"], hp["leaf_ptr"], hp["leaf_off"] = d["row"].data_ptr(), d["ptr"].data_ptr(), d["off"].data_ptr()
    L = _lib.load()
    _lib.check(L.pq3d_hmatvec(hp.ctypes.data, x.data_ptr(), d["slots"].data_ptr(), x.data_ptr(),
                              d["add"][0].data_ptr(), None, d["add"][2].data_ptr(), y.data_ptr(), _lib.stream_ptr()),
               "pq3d_hmatvec")
    s = slots.astype(np.float64)
    ref, mag = np.zeros((n, 3)), np.zeros((n, 3))
    for i in range(n):
        rows = off[ptr[row[i]]:ptr[row[i] + 1]] + i
        ref[i], mag[i] = s[rows].sum(0), np.abs(s[rows]).sum(0)
    ref[:, 0] += add[0]
    ref[:, 2] += add[2]
    tol = 2 * (longest + 2) * 2.0 ** -53 * (mag + np.abs(add.T))
    assert (np.abs(y.cpu().numpy() - ref) <= tol).all()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_step_kernel_grids(prec, tmp_path):
    """One step from the same state with 1, 3 and all CTAs: the same step within rounding."""
    from pyquake3d_b200 import QDsim, meshgen, read_mshV2
    msh, para = meshgen.make_case("tiny", str(tmp_path), n_target=700, precision=prec)
    nodes, tris = read_mshV2(msh)
    sim = QDsim(tris, nodes, para)
    op = sim.tree_block.op()
    from pyquake3d_b200.qdsim import DeviceStepper
    got = []
    for grid in (None, 1, 3, 7):
        st = DeviceStepper(sim, op, prec)
        st.grid = st.grid if grid is None else grid
        st.blk = torch.zeros(10 * st.grid + 16, dtype=torch.float64, device="cuda")
        st.args["blk"] = st.blk.data_ptr()
        h = [st.step(1e3)[0] for _ in range(3)]
        got.append((h, st.get("slipv"), st.get("psi"), st.get("slip")))
    for g in got[1:]:
        for a, b in zip(g, got[0]):
            assert np.linalg.norm(np.asarray(a) - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("grid,rows", [(90, 16), (18, 80), (15, 96), (10, 144), (7, 208), (6, 240), (5, 256)])
def test_step_kernel_row_sums(grid, rows, tmp_path):
    """The step kernel's own row sums for CTAs of `rows` rows (threads left over in one and
    several groups) equal the row reduction's, every time: 2 K 2^-53 of the largest product
    for K slots a row."""
    from pyquake3d_b200 import QDsim, meshgen, read_mshV2
    from pyquake3d_b200.qdsim import DeviceStepper
    msh, para = meshgen.make_case("thrust20k", str(tmp_path), n_target=1500, precision="fp64")
    nodes, tris = read_mshV2(msh)
    sim = QDsim(tris, nodes, para)
    op = sim.tree_block.op()
    st = DeviceStepper(sim, op, "fp64")
    st.grid = grid
    st.blk = torch.zeros(10 * st.grid + 16, dtype=torch.float64, device="cuda")
    st.args["blk"] = st.blk.data_ptr()
    assert st.n == 1428 and min(256, 16 * -(-st.n // (16 * grid))) == rows
    for _ in range(40):
        y = op.matvec(st.x, "fp64")
        st.launch(0)
        assert (st.y - y).abs().max() <= 1e-13 * y.abs().max()
