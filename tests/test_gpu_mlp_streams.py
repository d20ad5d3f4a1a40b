"""Gradients of several streams may add to one loss: 400 batches on four streams, each with its
own scratch and gradient, sum to the losses of the batches one by one.

Tolerance: 400 FP32 additions of positive terms, 400 2^-24 of the sum, twice for the order."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_shared_loss():
    from pyquake3d_b200 import _lib
    from pyquake3d_b200._lib import ptr
    from pyquake3d_b200.vmode import MLP_NP, MLPTrainer
    tr = MLPTrainer(seed=1)
    B, n, k = 33, 100, 4
    X = torch.tensor(np.random.default_rng(2).standard_normal((k, n, B, 6)).astype(np.float32), device="cuda")
    one = sum(tr.grad(X[s, i], X[s, i][:, 5:])[1] for s in range(k) for i in range(n))
    loss = torch.zeros(1, device="cuda")
    work = [(torch.cuda.Stream(), torch.empty(258 * B, device="cuda"), torch.empty(MLP_NP, device="cuda")) for _ in range(k)]
    torch.cuda.synchronize()
    for i in range(n):
        for s, (st, scratch, g) in enumerate(work):
            x = X[s, i]
            _lib.check(tr.L.pq3d_mlp_grad(ptr(tr.P), ptr(x), 6, ptr(x[:, 5:]), 6, B, ptr(scratch), ptr(g), ptr(loss),
                                          st.cuda_stream), "pq3d_mlp_grad")
    torch.cuda.synchronize()
    assert abs(float(loss) - one) <= 2 * n * k * 2.0 ** -24 * one
