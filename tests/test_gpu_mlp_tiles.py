"""The proposer's tile kernel at the edges of its 64-sample tiles, with more tiles than CTAs, and
through a shuffled index.  Tolerances as for the whole network: 2e-4 of the largest value (FP32
sums of at most 64 products of order one per layer against float64, 1e-4 for the mean loss)."""
import numpy as np
import pytest

import mlp_ref
from redgb.proposer import Proposer

pytestmark = pytest.mark.gpu


def _net(seed):
    rng = np.random.RandomState(seed)
    w = (rng.randn(mlp_ref.N) * 0.3).astype(np.float32)
    mean, std = rng.randn(8).astype(np.float32), rng.uniform(0.5, 2.0, 8).astype(np.float32)
    p = Proposer(seed)
    p.set_params(w)
    p.set_normalisation(mean, std)
    return p, w, mean, std, rng


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 128, 191, 19457, 39000])
def test_tiles_match_oracle(gpulib, n):
    p, w, mean, std, rng = _net(n)
    x = (rng.randn(n, 8) * std + mean).astype(np.float32)
    y = rng.randn(n).astype(np.float32)
    z = ((x - mean) / std).astype(np.float64)
    ref, _ = mlp_ref.forward(w, z)
    assert np.max(np.abs(p.forward(x) - ref)) <= 2e-4 * max(1.0, np.max(np.abs(ref)))
    g, loss = p.gradient(x, y)
    gr, lr = mlp_ref.gradient(w, z, y.astype(np.float64))
    assert abs(loss - lr) <= 1e-4 * lr
    assert np.max(np.abs(g - gr)) <= 2e-4 * np.max(np.abs(gr))
    # the buffers of a larger call serve a smaller one
    assert np.array_equal(p.forward(x[:1]), p.forward(x)[:1])


def test_shuffled_batch_has_the_batch_loss(gpulib):
    """One epoch of one batch reads the samples through a shuffled index: the loss before its
    update is the batch's."""
    p, w, mean, std, rng = _net(5)
    x = (rng.randn(130, 8) * std + mean).astype(np.float32)
    y = rng.randn(130).astype(np.float32)
    _, lr = mlp_ref.gradient(w, ((x - mean) / std).astype(np.float64), y.astype(np.float64))
    assert abs(p.train(x, y, epochs=1, batch=130, lr=1e-3) - lr) <= 1e-4 * lr
