"""The device prune on long lists: the sort's tiles add up each other's digit counts up to 256
tiles of 4,096 candidates and have them scanned above.  Selections are compared exactly with the
host restatement; what the sorts cost grows with the candidates, not with their square."""
import re

import numpy as np
import pytest

from pyopenlpt_b200 import _ffi
from tests.test_prune import _prune

pytestmark = pytest.mark.gpu

LIMIT = 256 * 4096


def _list(M):
    rng = np.random.default_rng(M)
    n_pts = M // 3
    ids = rng.integers(0, n_pts, (M, 3)).astype(np.int32)
    ids[:, 0].sort()
    e = rng.random(M) * 0.05
    e[rng.random(M) < 0.2] = 0.011  # ties
    e[rng.random(M) < 0.01] = np.inf
    return ids, e, [n_pts] * 3


@pytest.mark.parametrize("M", [LIMIT, LIMIT + 1, LIMIT + 4096 * 3 + 77])
def test_selection_on_both_sides_of_the_scan(M):
    ids, e, counts = _list(M)
    ctx = _ffi.Context(0)
    try:
        got = ctx.prune_matches(ids, e, counts)
    finally:
        ctx.close()
    assert np.array_equal(got, _prune(ids, e, counts, [1] * 3))


def test_sort_cost_is_linear():
    """Device time of the sorts of 8 million candidates against 1 million: 8 times, and half as
    much again for the caches (it was 30 times with sums in every block)."""
    from torch.profiler import ProfilerActivity, profile

    us = []
    ctx = _ffi.Context(0)
    try:
        for M in (1_000_000, 8_000_000):
            ids, e, counts = _list(M)
            ctx.prune_matches(ids, e, counts)
            with profile(activities=[ProfilerActivity.CUDA]) as p:
                ctx.prune_matches(ids, e, counts)
            us.append(sum(k.device_time_total for k in p.key_averages()
                          if re.search("rs_hist|rs_scatter|scan_sums|scan_tiles", k.key)))
    finally:
        ctx.close()
    print(f"sorts and scans: {us[0]:.0f} us, {us[1]:.0f} us")
    assert 0.0 < us[1] <= 12.0 * us[0]
