"""The ensemble step kernels write their scratch and nothing behind it: 8 doubles of fstate per
fault in lock step, whatever the grid, and the meeting words of pq3d_ens_meet_bytes with a CTA
per task, left cleared."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faults", [1, 4])
def test_scratch_bounds(faults, tmp_path):
    from pyquake3d_b200 import QDsim, _lib, meshgen, read_mshV2
    from pyquake3d_b200.ensemble import Ensemble
    sims = []
    for k in range(faults):
        d = tmp_path / str(k)
        d.mkdir()
        msh, para = meshgen.make_case("tiny", str(d), n_target=200 + 150 * k, precision="fp64")
        nodes, tris = read_mshV2(msh)
        sims.append(QDsim(tris, nodes, para, precision="fp64"))
    E = Ensemble(sims, precision="fp64")
    L, T, M = E.L, E.n_tasks, E.M
    assert E.grid == T
    mark = -7.25
    E.ctrl[:, 0] = torch.tensor([1e3, 1e9, 1e12, 1e3][:M], device="cuda", dtype=torch.float64)
    for grid in (T, 1, max(1, T - 1)):
        fs = torch.full((8 * M + 64,), mark, dtype=torch.float64, device="cuda")
        E.args["fstate"] = fs.data_ptr()
        E.op.matvec(E.x, "fp64", slots_only=True)
        _lib.check(L.pq3d_ens_step(E.args.ctypes.data, grid, _lib.stream_ptr()), "pq3d_ens_step")
        assert (fs[8 * M:] == mark).all()
        assert (E.ctrl[:, 4] == 0).all()
    words = L.pq3d_ens_meet_bytes(M) // 8
    meet = torch.full((words + 64,), 77, dtype=torch.int64, device="cuda")
    meet[:words] = 0
    fs = torch.full((8 * M + 64,), mark, dtype=torch.float64, device="cuda")
    E.args["fstate"] = fs.data_ptr()
    for _ in range(3):
        E.op.matvec(E.x, "fp64", slots_only=True)
        _lib.check(L.pq3d_ens_step_faults(E.args.ctypes.data, meet.data_ptr(), _lib.stream_ptr()), "pq3d_ens_step_faults")
        assert (meet[words:] == 77).all() and (meet[:words] == 0).all() and (fs[8 * M:] == mark).all()
    assert (E.ctrl[:, 8] == 6).all() and np.isfinite(E.ctrl.cpu().numpy()).all()
