"""Calls on one handle share its device space, from chunk to chunk and thread to thread."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


# one chunk, two, two and a ragged rest; more than the handle keeps (64 MB) at the end
@pytest.mark.parametrize("n", [65535, 65536, 98311, 530000])
def test_chunked_upload(gpu, n):
    """Predictions are the pieces' to the bit; gradients as in FP64, FP32 sums: 2e-5 of the largest entry."""
    rng = np.random.default_rng(n)
    X = rng.normal(0, 1, (n, 32)).astype(np.float32)
    Y = rng.normal(0, 0.3, n).astype(np.float32)
    mlp = gpu.MLP(seed=7)
    mlp.set(norm=np.concatenate([np.zeros(32), np.ones(32)]).astype(np.float32))
    p, nrm = mlp.get()
    y = mlp.predict(X)
    np.testing.assert_array_equal(y, np.concatenate([mlp.predict(X[i:i + 10000]) for i in range(0, n, 10000)]))
    g, loss = mlp.grad(X, Y)
    gr, lr = MO.grad(p, nrm, X.astype(np.float64), Y.astype(np.float64))
    assert abs(loss - lr) < 1e-5 * max(1.0, lr)
    np.testing.assert_allclose(g, gr, atol=2e-5 * np.abs(gr).max(), rtol=0)


def test_threads_share_a_handle(gpu):
    rng = np.random.default_rng(0)
    mlp = gpu.MLP(seed=7)
    mlp.set(norm=np.concatenate([np.zeros(32), np.ones(32)]).astype(np.float32))
    sets = [rng.normal(0, 1, (n, 32)).astype(np.float32) for n in (100, 70000, 5000, 33000)]
    alone = [mlp.predict(x) for x in sets]
    with ThreadPoolExecutor(4) as ex:
        for _ in range(5):
            for a, b in zip(alone, ex.map(mlp.predict, sets)):
                np.testing.assert_array_equal(a, b)
