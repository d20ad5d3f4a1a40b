"""The row sums inside the row-range kernels (CTAs of 256 rows) for lists that are staged and
lists that are too long for it (dense blocks cut into chunks of one column group), over the
whole fault and a ragged range, against the row reduction of the same slots.

Tolerance: sums of K FP64 values in another order differ by at most 2 K 2^-53 of the sum of
their magnitudes, here for K and magnitudes of the longest list of all."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("chunk", [64, 1])
def test_row_range_sums(prec, chunk, tmp_path):
    from pyquake3d_b200 import QDsim, _lib, meshgen, read_mshV2
    from pyquake3d_b200.qdsim import DeviceStepper
    msh, para = meshgen.make_case("thrust20k", str(tmp_path), n_target=1500, precision=prec)
    nodes, tris = read_mshV2(msh)
    sim = QDsim(tris, nodes, para)
    op = sim.tree_block.op()
    op.set_shapes(prec, chunk, 256, 512)
    P = op.plan(prec)
    ptr = P["leaf_ptr"].cpu().numpy()
    row = P["leaf_of_row"].cpu().numpy()
    per_cta = ptr[row[255] + 1] - ptr[row[0]]
    assert (per_cta > 2048) == (chunk == 1)
    st = DeviceStepper(sim, op, prec)
    y = op.matvec(st.x, prec)
    slots = P["slots"].view(-1, 3)[:P["n_slots"]].double().abs().sum().item()
    tol = 2 * int(np.diff(ptr).max()) * 2.0 ** -53 * slots
    n = st.n
    for r0, r1 in ((0, n), (100, 1301), (n - 3, n)):
        grid = -(-(r1 - r0) // 256)
        a = st.args.copy()
        blk = torch.zeros(4 * grid + 16, dtype=torch.float64, device="cuda")
        bar = torch.zeros(4, dtype=torch.int32, device="cuda")
        out = torch.zeros(8, dtype=torch.float64, device="cuda")
        a["blk"], a["bar"] = blk.data_ptr(), bar.data_ptr()
        st.y.fill_(float("nan"))
        _lib.check(st.L.pq3d_rk_rows_attempt(a.ctypes.data, grid, r0, r1, 1e3, 1, out.data_ptr(), _lib.stream_ptr()),
                   "pq3d_rk_rows_attempt")
        assert ((st.y - y)[r0:r1].abs() <= tol).all()
        assert torch.isnan(st.y[:r0]).all() and torch.isnan(st.y[r1:]).all()
