"""The device prune at the list lengths where its sorts change: one block up to 4,096
candidates, a cluster of blocks up to 114,688, tiles in global memory above; against the host
restatement of StereoMatch::pruneMatch (src/srcSTB/StereoMatch.cpp:631-980).  Selections are
compared exactly."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi
from tests.test_prune import _prune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2, 33, 4095, 4096, 4097, 4608, 16 * 4096 + 1, 114_688, 114_689,
                               130_000])
def test_selection_at_the_sorts_limits(M):
    rng = np.random.default_rng(M)
    n_cam, n_pts = 3, max(2, M // 6)
    ids = np.unique(rng.integers(0, n_pts, size=(M + M // 8 + 8, n_cam)).astype(np.int32), axis=0)
    if len(ids) < M:  # a few points only: all triples
        ids = np.stack(np.meshgrid(*[np.arange(n_pts)] * n_cam, indexing="ij"), -1)
        ids = ids.reshape(-1, n_cam).astype(np.int32)
    ids = ids[np.sort(rng.permutation(len(ids))[:M])]
    assert len(ids) == M
    e = rng.random(M) * 0.05
    e[rng.random(M) < 0.3] = 0.011  # ties
    e[rng.random(M) < 0.02] = np.inf
    counts = [n_pts] * n_cam
    ctx = _ffi.Context(0)
    try:
        got = ctx.prune_matches(ids, e, counts)
        again = ctx.prune_matches(ids, e, counts)
    finally:
        ctx.close()
    assert np.array_equal(got, _prune(ids, e, counts, [1] * n_cam))
    assert np.array_equal(got, again)


@pytest.mark.parametrize("drop", [0.0, 0.1])
def test_selection_at_the_pools_limits(drop):
    """Pools of a point in registers (32), in shared memory (128) and in global memory, with
    checks that tie within the tolerance and some that are not finite."""
    rng = np.random.default_rng(int(10 * drop))
    sizes = [1, 2, 31, 32, 33, 34, 64, 127, 128, 129, 130, 513, 1500]
    first = np.repeat(np.arange(len(sizes)), sizes)
    M = len(first)
    ids = np.c_[first, rng.integers(0, M // 3, M), rng.permutation(M)].astype(np.int32)
    ids = ids[np.lexsort(ids.T[::-1])]
    e = rng.integers(1, 400, M) * 1e-4 * (1.0 + rng.integers(-1, 2, M) * 2e-10)
    e[rng.random(M) < drop] = np.nan
    counts = [len(sizes), M, M]
    ctx = _ffi.Context(0)
    try:
        got = ctx.prune_matches(ids, e, counts)
    finally:
        ctx.close()
    assert np.array_equal(got, _prune(ids, e, counts, [1] * 3))
