"""The network's gradient kernel at the edges of its tiles of 64 samples and of
its grid (304 CTAs), against the FP64 oracle: FP32 sums of n terms, 2e-5 of
the largest entry as for the whole network."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 19456, 19521])
def test_gradient_tiles(gpu, n):
    rng = np.random.default_rng(n)
    X = rng.normal(0, 1, (n, 32)).astype(np.float32)
    Y = rng.normal(0, 0.3, n).astype(np.float32)
    mlp = gpu.MLP(seed=7)
    nrm = np.concatenate([rng.normal(0, 0.1, 32), rng.uniform(0.5, 1.5, 32)]).astype(np.float32)
    mlp.set(norm=nrm)
    p, _ = mlp.get()
    g, loss = mlp.grad(X, Y)
    gr, lr = MO.grad(p, nrm, X.astype(np.float64), Y.astype(np.float64))
    assert abs(loss - lr) < 1e-5 * max(1.0, lr)
    np.testing.assert_allclose(g, gr, atol=2e-5 * np.abs(gr).max(), rtol=0)
    y = mlp.predict_fp32(X)
    yr, _ = MO.forward(p, nrm, X.astype(np.float64))
    np.testing.assert_allclose(y, yr, atol=2e-5 * max(1.0, np.abs(yr).max()), rtol=0)
