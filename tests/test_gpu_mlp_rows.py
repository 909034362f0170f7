"""Every row enters the presize network's gradient once: one row at a time gets
a residual that outweighs all others together, so that the gradient is that
row's, and one lost or doubled changes it by half or more.

Tolerance: as for the gradient itself, 2e-4 of the largest entry (chains of 128
FP32 products, and room for a hidden unit whose sign flips); the other rows'
residuals add at most 30,000 x 10 to 1e7."""
import numpy as np
import pytest

from gls.capi import Trainer
from oracle import mlp_ref
from test_gpu_presize import random_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 9_728, 9_729, 30_000])
def test_each_row_counts_once(n, gpu):
    rng = np.random.default_rng(n)
    X = random_rows(rng, n)
    t = rng.uniform(0, 8, n).astype(np.float32)
    marks = sorted({k for k in (0, 63, 64, n // 2, 152 * 64 - 1, 152 * 64, 152 * 64 + 64, n - 65, n - 64, n - 1) if 0 <= k < n})
    with Trainer(seed=n) as tr:
        tr.set_data(X, t)
        p = tr.params()
        for row in marks:
            tt = t.copy()
            tt[row] = 1e7
            tr.set_data(X, tt)
            tr.set_params(p)   # new data set the output bias to their mean target
            g, loss = tr.grad(0, n, 1e9)
            lref, gref = mlp_ref.loss_grad(p, X, tt, 1e9)
            assert abs(loss - lref) <= 1e-5 * abs(lref), row
            assert np.abs(g - gref).max() <= 2e-4 * np.abs(gref).max(), row
            _, one = mlp_ref.loss_grad(p, X[row:row + 1], tt[row:row + 1], 1e9)
            assert np.abs(gref - one / n).max() <= 0.1 * np.abs(gref).max()   # the gradient is that row's
