"""Error maxima are folded as ordered bits: a NaN anywhere on a fault must reach every CTA that
decides on the step, whichever lane and CTA holds it, and an infinite term must not hide it.
A step with a NaN error term is rejected until it is given up (21 times, as the controller of
the reference does) and the state stays.  In an ensemble the other faults step as they
do beside a sound one, with a CTA per task and in lock step."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
STATE = ("psi", "Tt1o", "Tt2o", "Tno", "slip1", "slipv")


def _sim(tmp_path, n, tag):
    from pyquake3d_b200 import QDsim, meshgen, read_mshV2
    d = tmp_path / tag
    d.mkdir()
    msh, para = meshgen.make_case("tiny", str(d), n_target=n, precision="fp64")
    nodes, tris = read_mshV2(msh)
    return QDsim(tris, nodes, para, precision="fp64")


@pytest.mark.parametrize("where", [0, 37, 255, -1])
@pytest.mark.parametrize("bad", [("psi", float("nan")), ("Tt1o", float("nan")), ("Tno", float("nan"))])
def test_single_fault(where, bad, tmp_path):
    from pyquake3d_b200 import _lib
    from pyquake3d_b200.qdsim import DeviceStepper
    sim = _sim(tmp_path, 800, "a")
    st = DeviceStepper(sim, sim.tree_block.op(), "fp64")
    st.step(1e3)
    st.t[bad[0]][where] = bad[1]
    st.t["Tt2o"][5] = float("inf")
    keep = {k: st.t[k].clone() for k in STATE}
    steps = float(st.ctrl[8])
    with pytest.raises(_lib.Pq3dError, match="rejects=21"):
        st.step(1e3)
    assert float(st.ctrl[8]) == steps
    for k in STATE:
        assert torch.equal(st.t[k].nan_to_num(nan=-1.0), keep[k].nan_to_num(nan=-1.0)), k


@pytest.mark.parametrize("lock_step", [False, True])
def test_ensemble_fault_that_gives_up(lock_step, tmp_path):
    from pyquake3d_b200.ensemble import Ensemble
    sims = [_sim(tmp_path, n, "e%d" % n) for n in (60, 500, 800)]
    got = []
    for nan in (False, True):
        E = Ensemble(sims, precision="fp64")
        assert E.grid == E.n_tasks > 3
        if lock_step:
            E.grid = E.n_tasks - 1
        a, b = int(E.struct.row0[1]), int(E.struct.row0[2])
        if nan:
            E.t["psi"][b - 3] = float("nan")
        keep = {k: E.t[k][a:b].clone() for k in STATE}
        E.ctrl[:, 0] = torch.tensor([1e3, 1e3, 1e12], device="cuda", dtype=torch.float64)
        for _ in range(3):
            E.launch(0)
        got.append((E.ctrl.cpu().numpy().copy(), {k: E.t[k].cpu().numpy() for k in STATE}))
        if nan:
            for k in STATE:
                assert torch.equal(E.t[k][a:b].nan_to_num(nan=-1.0), keep[k].nan_to_num(nan=-1.0)), k
    (c0, s0), (c1, s1) = got
    assert (c0[:, 4] == 0).all() and (c0[:, 8] == 3).all() and c0[2, 9] > 0
    assert c1[1, 4] != 0 and c1[1, 3] == 21 and c1[1, 8] == 0
    for f in (0, 2):
        assert np.array_equal(c1[f, :11], c0[f, :11])
        a, b = int(E.struct.row0[f]), int(E.struct.row0[f + 1])
        for k in STATE:
            assert np.array_equal(s1[k][a:b], s0[k][a:b]), (f, k)
