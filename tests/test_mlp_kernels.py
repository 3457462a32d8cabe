"""The rank network's kernels at the edges of their passes (16 samples a CTA, 512
partial gradients), against the float64 oracle."""
import numpy as np
import pytest

import mlp_ref
from ahmed_gb300.rank_predictor import RankPredictor, _moments


@pytest.mark.parametrize("n", [1, 2, 7, 64, 65, 5003])
def test_moments_are_numpys(n):
    X = (np.random.default_rng(n).standard_normal((n, 8)) * 3 + 2).astype(np.float32)
    X[:, 5] = 6.0
    mean, std = _moments(X)
    np.testing.assert_allclose(mean, X.mean(axis=0), rtol=1e-6, atol=1e-6)
    np.testing.assert_allclose(std, X.std(axis=0), rtol=1e-6, atol=1e-6)
    assert std[5] == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 1024, 8192, 8193, 20011])
def test_gradient_and_forward(n):
    rng = np.random.default_rng(n)
    p = (rng.standard_normal(mlp_ref.NPARAMS) * 0.2).astype(np.float32)
    X = (rng.standard_normal((n, 8)) * 2 + 1).astype(np.float32)
    y = rng.standard_normal(n).astype(np.float32)
    mean, std = np.full(8, 0.9, np.float32), np.full(8, 1.8, np.float32)
    M = RankPredictor(seed=1)
    M.params = p
    M.set_norm(mean, std)
    g, loss = M.gradients(X, y)
    lo, go = mlp_ref.loss_and_grad(p, X, y, mean.astype(np.float64), std.astype(np.float64))
    # FP32 sums of 64 terms per layer, n samples in pieces: relative error well below 1e-4
    assert abs(loss - lo) <= 1e-4 * lo
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)
    out = M.predict_log(X)
    ref = mlp_ref.forward(p, X, mean.astype(np.float64), std.astype(np.float64))[-1]
    np.testing.assert_allclose(out, ref, rtol=1e-4, atol=1e-4 * np.abs(ref).max())
    g2, loss2 = M.gradients(X, y)
    assert np.array_equal(g, g2) and loss == loss2  # fixed order of every sum
    M.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch,epochs", [(1, 4, 3), (50, 7, 4), (3000, 1024, 5)])
def test_training_is_reproducible(n, batch, epochs):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 8)).astype(np.float32)
    r = rng.integers(1, 20, n).astype(np.float32)
    got = []
    for _ in range(2):
        M = RankPredictor(seed=3)
        losses = M.fit(X, r, epochs=epochs, batch=batch, seed=5)
        got.append((losses, M.params))
        # the reported loss is the mean squared error of the predictions
        assert abs(losses[-1] - np.mean((M.predict_log(X) - np.log1p(r)) ** 2)) <= 1e-4 * losses[-1] + 1e-7
        M.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
