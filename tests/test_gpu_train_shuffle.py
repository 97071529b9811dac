"""The training's seeded Fisher-Yates order: numbers swapped on the host, samples
gathered on the device, against the swaps written out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1


def _order(n, seed):
    s = seed ^ 0x5DEECE66D
    order = list(range(n))
    for i in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & MASK
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & MASK
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & MASK
        j = (z ^ (z >> 31)) % (i + 1)
        order[i], order[j] = order[j], order[i]
    return order


@pytest.mark.parametrize("n", [128, 129, 257, 4096, 65537])
def test_shuffled_order(n):
    import freeshearlayer_b200 as fsl
    rng = np.random.default_rng(n)
    X = rng.uniform(0.1, 1.0, (n, 8)).astype(np.float32)
    Y = rng.uniform(0.0, 0.1, n).astype(np.float32)
    t = fsl.Trainer(n + 3, seed=9)
    t.set_samples(X, Y)
    for _ in range(2):  # shuffled once
        t.train(1, 128, 1e-4)
        x, y = t.samples()
        order = _order(n, 9)
        assert np.array_equal(x, X[order]) and np.array_equal(y, Y[order])
