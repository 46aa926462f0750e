"""Every call on a network handle takes its turn: gradients beside training,
predictions beside a change of weights."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NORM = np.concatenate([np.zeros(32), np.ones(32)]).astype(np.float32)


def test_gradients_beside_training(gpu):
    """Training at a rate that leaves every FP32 weight as it is; gradients are
    sums in any order, 2e-5 of the largest entry."""
    rng = np.random.default_rng(0)
    mlp = gpu.MLP(seed=7)
    mlp.set(norm=NORM)
    sets = [(rng.normal(0, 1, (n, 32)).astype(np.float32), rng.normal(0, 0.3, n).astype(np.float32))
            for n in (300, 5000, 70000)]
    alone = [mlp.grad(*s) for s in sets]
    with ThreadPoolExecutor(4) as ex:
        for _ in range(20):
            train = ex.submit(mlp.train, *sets[1], epochs=2, batch=256, lr=1e-30)
            for (g, loss), f in zip(alone, [ex.submit(mlp.grad, *s) for s in sets]):
                g2, loss2 = f.result()
                np.testing.assert_allclose(g2, g, rtol=0, atol=2e-5 * np.abs(g).max())
                assert abs(loss2 - loss) < 1e-5 * max(1.0, loss)
            train.result()


def test_predictions_beside_new_weights(gpu):
    """A prediction in several chunks is wholly that of one set of weights."""
    rng = np.random.default_rng(1)
    x = rng.normal(0, 1, (200000, 32)).astype(np.float32)
    mlp = gpu.MLP(seed=7)
    mlp.set(norm=NORM)
    w = [mlp.get()[0], gpu.MLP(seed=8).get()[0]]
    ys = []
    for v in w:
        mlp.set(params=v)
        ys.append(mlp.predict(x))
    with ThreadPoolExecutor(2) as ex:
        for i in range(60):
            f = ex.submit(mlp.predict, x)
            for j in range(8):
                mlp.set(params=w[(i + j) & 1])
            y = f.result()
            assert any(np.array_equal(y, v) for v in ys)
