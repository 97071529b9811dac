"""The training kernel at the edges of its tiles (128 samples a tile, several
tiles a block): gradients against the CPU oracle, and repeatability."""
import numpy as np
import pytest

from tests.test_gpu_closure import GROUPS, _random_samples

pytestmark = pytest.mark.gpu


# one sample; one short of, and one over, a tile; one tile over a tile per block
@pytest.mark.parametrize("n", [1, 127, 129, 128 * 148 + 1])
def test_gradient_at_tile_edges(n):
    import freeshearlayer_b200 as fsl
    from oracle import mlp_oracle as mo
    X, Y = _random_samples(n, 23)
    tr = fsl.Trainer(max(n, 128), seed=3)
    tr.set_samples(X, Y)
    tr.set_loss(0)
    p = tr.weights()
    p[9472] = 0.05
    tr.set_weights(p)
    g, loss = tr.gradient(n)
    again, _ = tr.gradient(n)
    assert np.array_equal(g, again)  # every sum has one order
    loss_ref, g_ref = mo.loss_and_grad(p, X, Y)
    # the oracle rounds to BF16 where the kernel does; what is left is the
    # approximate tanh (2^-11 relative) through three layers and the BF16
    # steps (2^-8) of the few values that it moves across a rounding boundary
    assert abs(loss - loss_ref) <= 2e-2 * loss_ref
    for name, (a, b) in GROUPS.items():
        ref = g_ref[a:b]
        assert np.linalg.norm(g[a:b] - ref) <= 3e-2 * np.linalg.norm(ref), name
