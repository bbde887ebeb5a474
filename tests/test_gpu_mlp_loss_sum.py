"""The proposer's mean loss at batch sizes from one tile to a million: the same accuracy at all of them.
Tolerance 5e-6 of the loss: a thread's chain of at most 52 additions and a tree of 5 round by less than
1e-6 together, and the CTAs' 608 partial sums, added one by one in FP32, by sqrt(608 / 3) 2^-24 = 0.9e-6
as random roundings (five times that is allowed); the forward pass in FP32 is below 1e-6 in the mean."""
import numpy as np
import pytest

import mlp_ref
from redgb.proposer import Proposer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 65536, 65537, 100000, 1000000])
def test_loss_of_any_batch(gpulib, n):
    rng = np.random.RandomState(7)
    w = (rng.randn(mlp_ref.N) * 0.2).astype(np.float32)
    x, y = rng.randn(n, 8).astype(np.float32), rng.randn(n).astype(np.float32)
    p = Proposer(1)
    p.set_params(w)
    p.set_normalisation(np.zeros(8, np.float32), np.ones(8, np.float32))
    _, loss = p.gradient(x, y)
    want = np.mean(np.concatenate([(mlp_ref.forward(w, x[k:k + 50000].astype(np.float64))[0] - y[k:k + 50000]) ** 2
                                   for k in range(0, n, 50000)]))
    assert abs(loss - want) <= 5e-6 * want, (loss, want, loss / want - 1)
