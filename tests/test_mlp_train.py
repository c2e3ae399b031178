"""The training kernels against the FP64 reference network: batch sizes at the
edges of their tiles (32, 64 rows), of the switch between them, and of the
batch slices of the weight gradients."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 31, 33, 64, 65, 127, 128, 129, 1000, 1025, 2304, 2305, 2369, 5003])
def test_gradient(batch):
    """FP32 products and sums of up to 256 terms forward and `batch` terms in
    the weight gradients, each rounding 2^-24 of a partial sum: within 1e-5 of
    the largest gradient entry (the sums' roundings add up like a random walk,
    sqrt(5003 + 2 x 256) 2^-24 = 4e-6) and of the loss."""
    from rigidfibers_kth_b200.learned import Trainer

    rng = np.random.default_rng(batch)
    tr = Trainer(seed=3)
    w = tr.weights()
    x = rng.standard_normal((batch, 144)).astype(np.float32)
    y = (0.1 * rng.standard_normal((batch, 225))).astype(np.float32)
    loss, g = tr.loss_grad(x, y)
    loss2, g2 = tr.loss_grad(x, y)
    tr.close()
    assert loss == loss2 and np.array_equal(g, g2)
    loss_ref, g_ref = mlp_ref.loss_grad(w.astype(np.float64), x, y)
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref
    assert np.abs(g - g_ref).max() <= 1e-5 * np.abs(g_ref).max()


def test_training_is_reproducible_over_ragged_batches():
    """Two trainers with one seed end with the same weights; the last batch of an
    epoch is smaller than the others."""
    from rigidfibers_kth_b200.learned import Trainer

    rng = np.random.default_rng(9)
    x = rng.standard_normal((777, 144)).astype(np.float32)
    y = (0.1 * rng.standard_normal((777, 225))).astype(np.float32)
    out = []
    for _ in range(2):
        tr = Trainer(seed=5)
        tr.add_samples(x, y)
        losses = [tr.train(1, batch=100, lr=1e-3) for _ in range(3)]
        out.append((losses, tr.weights()))
        tr.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
    assert out[0][0][2] < out[0][0][0]
