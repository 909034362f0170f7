"""gls_levelize's polled sweeps and radix packing at their edges, against a
numpy longest-path: one to three sort passes (levels past 2^8 and 2^16), tile
remainders, instance counts past the resident threads."""
import numpy as np
import pytest

from gls.capi import levelize_gpu

pytestmark = pytest.mark.gpu


def check(level, ps, pr):
    order, start = levelize_gpu(ps, pr)
    want = np.argsort(level, kind="stable")
    assert np.array_equal(order, want)
    nl = int(level.max()) + 1
    assert np.array_equal(start, np.concatenate([np.searchsorted(level[want], np.arange(nl)), [len(level)]]))


@pytest.mark.parametrize("n", [1, 2, 255, 257, 2047, 2048, 2049, 66_000])
def test_chain(n, gpu):
    """One instance per level, listed from the last to the first."""
    level = np.arange(n)[::-1].copy()
    ps = np.minimum(np.arange(n + 1), n - 1).astype(np.uint64)
    check(level, ps, np.arange(1, n).astype(np.uint32))


@pytest.mark.parametrize("n,depth", [(5_000, 3), (30_001, 256), (30_001, 257), (700_003, 40)])
def test_shuffled_layers(n, depth, gpu):
    """Instances of random layers in random order, each with one predecessor in
    the layer before and up to two anywhere before that."""
    rng = np.random.default_rng(n + depth)
    level = rng.integers(0, depth, n)
    level[rng.permutation(n)[:depth]] = np.arange(depth)   # no empty layer
    by = np.argsort(level, kind="stable")
    first = np.searchsorted(level[by], np.arange(depth + 1))
    size = np.diff(first)
    has = level > 0
    below = np.maximum(level - 1, 0)
    one = by[first[below] + (rng.random(n) * size[below]).astype(np.int64)]
    far = by[(rng.random((n, 2)) * first[np.maximum(level, 1)][:, None]).astype(np.int64)]
    extra = rng.integers(0, 3, n) * has
    cnt = has + extra
    ps = np.zeros(n + 1, np.uint64)
    np.cumsum(cnt, out=ps[1:])
    rows = np.stack([one, far[:, 0], far[:, 1]], 1)
    keep = np.arange(3)[None, :] < cnt[:, None]
    check(level, ps, rows[keep].astype(np.uint32))
