"""An operator without low-rank blocks read back from a checkpoint takes further storages:
its FP32 near field serves the FP32 and BF16 plans, with no factors to pack.  CPU: the
operator object holds host tensors and launches nothing on this path."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyquake3d_b200 import _lib, checkpoint, meshgen
from pyquake3d_b200.hmatrix import DeviceHMatrix, HStructure, dense_layout


def _operator(struct):
    op = DeviceHMatrix.__new__(DeviceHMatrix)
    op.torch, op.L, op.dev, op.s, op.n = torch, _lib.load(), torch.device("cpu"), struct, struct.n
    op.mu = op.lam = 32e9
    op.aca_tol, op.aca_rel, op.aca_seed, op.kcap, op.halfspace = 0.01, False, 0, 96, 0
    op.keep_factors, op.use_plan_cache, op._stream = False, False, None
    op.dense_blocks = [b for b in struct.blocks if not b.aca]
    op.aca_blocks = [b for b in struct.blocks if b.aca]
    op.plans, op.assembled = {}, False
    return op


def test_dense_operator_takes_further_storages_after_load(tmp_path, monkeypatch):
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    P, T = meshgen.planar(16.0, 8.0, 70.0, 10, 5, jitter=0.1, seed=5)
    xg = meshgen.centroids_km(P, T) * 1e3
    ev = np.zeros((len(xg), 9))
    s = HStructure(xg, mini_leaf=100000)
    op = _operator(s)
    assert not op.aca_blocks
    op.dense_recs, n64, n32 = dense_layout(op.dense_blocks)
    op.dense64, op.dense32 = torch.rand(n64, dtype=torch.float64), torch.rand(n32)
    op.aca_ranks = op.aca_flags = np.zeros(0, np.int32)
    empty = lambda dt: torch.zeros(8, dtype=dt)
    op.install_plan("fp64", empty(torch.float64), empty(torch.float64))
    op.assembled = True
    path = str(tmp_path / "op.pq3d")
    checkpoint.save_operator(op, path, xg, ev)
    got = _operator(s)
    checkpoint.load_operator(got, path, xg, ev)
    assert sorted(got.plans) == ["fp64"]
    for d in ("fp32", "bf16"):
        p = got.plan(d)
        assert p["n_ditems"] > 0 and p["n_vitems"] == p["n_utasks"] == 0
        assert torch.equal(p["dense"], op.dense32)
