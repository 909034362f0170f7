"""The one-launch loss and gradient of the presize network at its edges
(rows around a tile, more tiles than blocks, a stretch of the data, gathered
minibatches) against the float64 restatement.

Tolerance: an entry is a sum over the rows of products of at most three
chains of 128 FP32 products, each within 128 x 2^-24 = 8e-6 of its size; 2e-4
of the largest entry leaves room for a hidden unit whose sign flips."""
import numpy as np
import pytest

from gls.capi import Trainer
from oracle import mlp_ref
from test_gpu_presize import random_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 63, 64, 65, 200, 9_729, 30_000])
@pytest.mark.parametrize("first", [0, 37])
def test_gradient_rows(first, n, gpu):
    rng = np.random.default_rng(n + first)
    X = random_rows(rng, first + n + 5)
    t = rng.uniform(0, 8, len(X)).astype(np.float32)
    with Trainer(seed=n) as tr:
        tr.set_data(X, t)
        p = tr.params()
        for huber in (1.0, 0.25):
            g, loss = tr.grad(first, n, huber)
            lref, gref = mlp_ref.loss_grad(p, X[first:first + n], t[first:first + n], huber)
            assert abs(loss - lref) <= 1e-5 * max(1.0, abs(lref))
            assert np.abs(g - gref).max() <= 2e-4 * np.abs(gref).max()


def test_epoch_takes_every_row_once(gpu):
    """One epoch with a zero step size: its mean loss is the mean over all
    rows, whatever their order, with a last minibatch of 3 rows."""
    rng = np.random.default_rng(8)
    X = random_rows(rng, 1_003)
    t = rng.uniform(0, 8, 1_003).astype(np.float32)
    with Trainer(seed=2) as tr:
        tr.set_data(X, t)
        p = tr.params()
        loss = tr.fit(2, batch=100, lr=0.0, huber=1.0, seed=5)
    lref, _ = mlp_ref.loss_grad(p, X, t, 1.0)
    assert np.abs(loss - lref).max() <= 1e-5 * max(1.0, lref)
