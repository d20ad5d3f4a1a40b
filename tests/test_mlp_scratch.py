"""Scratch of the MLP gradient: 258 floats a sample for every batch size, and the kernels write
nothing behind it (nor behind the gradient, where a single CTA's share is made)."""
import numpy as np
import pytest

from pyquake3d_b200 import _lib
from pyquake3d_b200.vmode import MLP_NP, _bind

torch = pytest.importorskip("torch")
SIZES = [1, 2, 16, 17, 18, 32, 33, 35, 36, 64, 65, 4096, 9473]


@pytest.mark.parametrize("B", SIZES + [0, 1 << 20, 1 << 24])
def test_scratch_size(B):
    L = _lib.load()
    _bind(L)
    assert L.pq3d_mlp_scratch_floats(B) == 258 * B


@pytest.mark.gpu
@pytest.mark.parametrize("B", SIZES)
def test_scratch_bounds(B):
    from pyquake3d_b200._lib import ptr, stream_ptr
    from pyquake3d_b200.vmode import MLPTrainer
    X = torch.tensor(np.random.default_rng(B).standard_normal((B, 6)).astype(np.float32), device="cuda")
    tr = MLPTrainer(seed=3)
    G, loss = tr.grad(X, X[:, 5:])
    mark = -3.25
    scratch = torch.full((258 * B + 5000,), mark, device="cuda")
    g = torch.full((MLP_NP + 100,), mark, device="cuda")
    ls = torch.zeros(1, device="cuda")
    _lib.check(tr.L.pq3d_mlp_grad(ptr(tr.P), ptr(X), 6, ptr(X[:, 5:]), 6, B, ptr(scratch), ptr(g), ptr(ls), stream_ptr()),
               "pq3d_mlp_grad")
    assert (scratch[258 * B:] == mark).all() and (g[MLP_NP:] == mark).all()
    assert torch.equal(g[:MLP_NP], G) and float(ls) == loss
    # the update: the same gradient, moved parameters
    P, M, V = tr.P.clone(), torch.zeros_like(tr.P), torch.zeros_like(tr.P)
    g2, ls = torch.full((MLP_NP + 100,), mark, device="cuda"), torch.zeros(1, device="cuda")
    scratch.fill_(mark)
    _lib.check(tr.L.pq3d_mlp_train_step(ptr(P), ptr(M), ptr(V), ptr(X), 6, ptr(X[:, 5:]), 6, B, ptr(scratch), ptr(g2), 1e-3,
                                        0.9, 0.999, 1e-8, 1, ptr(ls), stream_ptr()), "pq3d_mlp_train_step")
    assert torch.equal(g2[:MLP_NP], G) and (g2[MLP_NP:] == mark).all() and (scratch[258 * B:] == mark).all()
    assert float(ls) == loss and not torch.equal(P, tr.P)
