"""Gradient, first Adam step and inference of the MLP at batch sizes around its tiles of 32
samples, the number of CTAs its scratch allows (one below 36 samples) and more tiles than CTAs.

Tolerance of a gradient entry: FP32 sums of at most 32 + 296 partials after layers of 64
terms lose at most (32 + 296 + 2 * 64) 2^-24 < 3e-5 of the sum of the terms' magnitudes, the
FP32 tanh and activations about as much again: 1e-4 of that sum."""
import numpy as np
import pytest

import vmode_oracle as vo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 5, 17, 31, 32, 33, 35, 36, 64, 1000, 4096, 9473])
def test_mlp_batch_sizes(B):
    from pyquake3d_b200.vmode import MLPTrainer, mlp_unflatten
    D = np.random.default_rng(B).standard_normal((B, 6)).astype(np.float32)
    data = torch.tensor(D, device="cuda")
    tr = MLPTrainer(seed=3)
    P = mlp_unflatten(tr.P.double().cpu().numpy())
    G, loss = tr.grad(data, data[:, 5:])
    X, t = D[:, :5].astype(np.float64), D[:, 5].astype(np.float64)
    L, gr = vo.mlp_loss_grad(P, X, t)
    y, (h1, h2) = vo.mlp_forward(P, X)
    d3 = np.abs(y - t) / B
    d2 = d3[:, None] * np.abs(P["W3"]) * (1 - h2 ** 2)
    d1 = (d2 @ np.abs(P["W2"])) * (1 - h1 ** 2)
    mag = dict(W1=d1.T @ np.abs(X), b1=d1.sum(0), W2=d2.T @ np.abs(h1), b2=d2.sum(0), W3=d3[None] @ np.abs(h2),
               b3=np.array([d3.sum()]))
    g = mlp_unflatten(G.cpu().numpy())
    for k in mag:
        assert (np.abs(g[k] - gr[k]) <= 1e-4 * mag[k]).all(), k
    assert abs(loss - L) <= 1e-4 * L
    assert np.abs(tr.predict(data).cpu().numpy() - y).max() <= 1e-5 * (1 + np.abs(y).max())
    before = tr.P.clone()
    tr.fit(data, epochs=1, batch=B, lr=1e-3)
    # Adam's first step moves a parameter by lr against its gradient's sign
    move, gf = (tr.P - before).cpu().numpy(), G.cpu().numpy()
    big = np.abs(gf) > 1e-4
    assert np.allclose(move[big], -1e-3 * np.sign(gf[big]), rtol=0, atol=2e-6)
