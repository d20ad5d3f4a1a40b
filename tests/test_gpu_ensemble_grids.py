"""The ensemble step with a CTA per task (each fault on its own) against fewer CTAs than tasks
(lock step): the same element expressions and exact maxima, so the same steps within rounding."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ensemble(tmp_path_factory):
    from pyquake3d_b200 import QDsim, meshgen, read_mshV2
    from pyquake3d_b200.ensemble import Ensemble
    sims = []
    for k, n in enumerate((60, 300, 800)):
        msh, para = meshgen.make_case("tiny", str(tmp_path_factory.mktemp("f%d" % k)), n_target=n, precision="fp64")
        nodes, tris = read_mshV2(msh)
        sims.append(QDsim(tris, nodes, para, precision="fp64"))
    return Ensemble(sims, precision="fp64")


def _steps(E, start, grids, tries):
    for k, v in start[0].items():
        E.t[k].copy_(v)
    E.x.copy_(start[1])
    E.ctrl.zero_()
    E.steps = 0
    hs = []
    for g, h in zip(grids, tries):
        E.grid = g
        hs.append(np.array(E.step(h)))
    return hs, E.ctrl.cpu().numpy().copy(), {k: E.t[k].cpu().numpy() for k in ("psi", "Tt1o", "slip1", "slipv")}


@pytest.mark.parametrize("pattern", ["one", "three", "all_but_one", "alternating"])
def test_lock_step_and_own_steps_agree(ensemble, pattern):
    E = ensemble
    T = E.n_tasks
    start = ({k: v.clone() for k, v in E.t.items()}, E.x.clone())
    # a size that is accepted, and per-fault ones that are rejected a different number of times
    tries = [np.full(E.M, 1e3), np.array([1e3, 1e9, 1e12]), np.full(E.M, 1e3)]
    grids = {"one": [1] * 3, "three": [3] * 3, "all_but_one": [T - 1] * 3, "alternating": [T, 3, T]}[pattern]
    ref = _steps(E, start, [T] * 3, tries)
    got = _steps(E, start, grids, tries)
    for k, v in start[0].items():
        E.t[k].copy_(v)
    E.x.copy_(start[1])
    assert (ref[1][:, 9] > 0).any() and (ref[1][:, 9] != ref[1][0, 9]).any()      # rejections, not the same for all
    assert np.array_equal(got[1][:, 8:11], ref[1][:, 8:11])                       # steps, rejections, attempts
    for a, b in zip(got[0], ref[0]):
        np.testing.assert_allclose(a, b, rtol=1e-11)
    for k in ref[2]:
        assert np.linalg.norm(got[2][k] - ref[2][k]) <= 1e-11 * np.linalg.norm(ref[2][k]), k
