"""The proposer's mean loss where a batch's samples begin to go to the sum one by one.  Tolerance as
for the smaller batches: 1e-4 of the loss (a serial FP32 sum of 70 000 positive terms is 2e-5 off)."""
import numpy as np
import pytest

import mlp_ref
from redgb.proposer import Proposer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65536, 65537, 65569, 70001])
def test_long_batch_loss(gpulib, n):
    rng = np.random.RandomState(n)
    w = (rng.randn(mlp_ref.N) * 0.3).astype(np.float32)
    x, y = rng.randn(n, 8).astype(np.float32), rng.randn(n).astype(np.float32)
    p = Proposer(1)
    p.set_params(w)
    p.set_normalisation(np.zeros(8, np.float32), np.ones(8, np.float32))
    _, loss = p.gradient(x, y)
    ref, _ = mlp_ref.forward(w, x.astype(np.float64))
    want = np.mean((ref - y.astype(np.float64)) ** 2)
    assert abs(loss - want) <= 1e-4 * want
    assert abs(p.train(x, y, epochs=1, batch=n, lr=1e-3) - want) <= 1e-4 * want
