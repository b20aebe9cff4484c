"""The pinned block of the read-backs: none before the first one, and results on both sides of the
sizes at which it grows (64 KB and its doubles up to 1 MB), also where a call's second result makes
it grow.  All comparisons are exact."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi
from tests.test_readback_gpu import _context

pytestmark = pytest.mark.gpu


def _pinned_kb():
    # pinned host memory counts as shared
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("RssShmem"))


def test_contexts_without_read_backs_pin_nothing():
    held = [_ffi.Context(0) for _ in range(2)]
    before = _pinned_kb()
    held += [_ffi.Context(0) for _ in range(32)]
    grown = _pinned_kb() - before
    for c in held:
        c.close()
    assert grown < 8 << 10  # 32 contexts of 1 MB were 32 MB


def test_block_grows_with_the_results():
    # 16 B a position and 8 B a pixel: the positions alone, then both, pass 64 KB, 128 KB, ..
    sizes = [1, 2730, 2731, 4096, 4097, 5461, 5462, 8193, 21845, 21846, 40_000, 43_690, 43_691, 5]
    ctx, cams = _context(2)
    try:
        rng = np.random.default_rng(7)
        for n in sizes:
            xy = [rng.random((n, 2)) * 255.0 for _ in cams]
            ctx.upload_detections(xy)
            for c, want in enumerate(xy):
                got, rc = ctx.get_peaks(c, n)
                assert np.array_equal(got, want)
                assert np.array_equal(rc, np.floor(want[:, ::-1] + 0.5).astype(np.int32))
    finally:
        ctx.close()
