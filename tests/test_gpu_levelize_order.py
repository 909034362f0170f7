"""GPU levelization of instance graphs in random file order, with one and with
several instances a thread, against levels computed on the host."""
import time

import numpy as np
import pytest

from gls.capi import GlsError, levelize_gpu

pytestmark = pytest.mark.gpu


def layered(n, depth, seed):
    """n instances of `depth` levels (each with an instance) in random file
    order: (pred_start, pred, level of every instance)."""
    rng = np.random.default_rng(seed)
    lev = np.sort(np.concatenate([np.arange(depth), rng.integers(0, depth, n - depth)]))
    start = np.searchsorted(lev, np.arange(depth + 1))
    place = rng.permutation(n)
    lo, hi = start[np.maximum(lev - 1, 0)], start[lev]
    a = (lo + rng.random(n) * (hi - lo)).astype(np.int64)   # from the level before
    b = (rng.random(n) * hi).astype(np.int64)               # from any before
    has = lev > 0
    pred = np.empty((n, 2), np.int64)
    pred[place] = np.stack([place[np.minimum(a, n - 1)], place[np.minimum(b, n - 1)]], 1)
    level = np.empty(n, np.int64)
    level[place] = lev
    has = level > 0
    ps = np.zeros(n + 1, np.uint64)
    ps[1:] = np.cumsum(2 * has)
    return ps, pred[has].ravel().astype(np.uint32), level


@pytest.mark.parametrize("n,depth", [(1_000, 30), (311_296, 5), (311_297, 40), (700_001, 90), (1_300_000, 3)])
def test_levels_in_random_file_order(n, depth, gpu):
    ps, pred, level = layered(n, depth, n)
    order, start = levelize_gpu(ps, pred)
    assert len(start) == depth + 1
    assert np.array_equal(order, np.argsort(level, kind="stable"))
    assert np.array_equal(start, np.searchsorted(np.sort(level), np.arange(depth + 1)))


def test_large_loop_is_refused(gpu):
    ps, pred, level = layered(700_001, 6, 1)
    one = int(np.flatnonzero(level == 1)[0])
    last = int(np.flatnonzero(level == 5)[0])
    # an instance of the first level behind one of the last, which reads it
    pred = pred.copy()
    pred[int(ps[one])] = last
    pred[int(ps[last])] = one
    with pytest.raises(GlsError):
        levelize_gpu(ps, pred)


def test_time_does_not_grow_with_the_polls(gpu):
    """2 M instances of 400 levels, several a thread: some 10 ms; looked at one
    by one until each has its level, 180 ms."""
    ps, pred, _ = layered(2_000_000, 400, 7)
    levelize_gpu(ps, pred)
    took = []
    for _ in range(3):
        t = time.perf_counter()
        levelize_gpu(ps, pred)
        took.append(time.perf_counter() - t)
    assert min(took) < 0.08
