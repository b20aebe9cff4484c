"""A sparse frame after a dense one on the same context: the buffers that the dense frame grew stay,
what the sparse frame costs does not depend on them.  The same candidates, and at most 1.3 times
the time on a fresh context (the smallest of 50 calls each; it was 1.7 times and more where the
grids followed the buffers)."""
import time

import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
N_CAM, SIDE = 4, 512


def _context(cams):
    ctx = _ffi.Context(0)
    ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
    return ctx


def _time(ctx, p):
    best = np.inf
    for _ in range(50):
        t = time.perf_counter()
        ctx.stereo_match(p)
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("n", [200, 3000])
def test_sparse_after_dense(n):
    cams = synth.ring_rig(N_CAM, SIDE, SIDE, min(synth.focal_for_volume(N_CAM, SIDE, VOLUME)))
    rng = np.random.default_rng(n)
    lo, hi = np.array(VOLUME[0::2]), np.array(VOLUME[1::2])
    fresh, used = _context(cams), _context(cams)
    try:
        xyz = lo + (hi - lo) * rng.random((n, 3))
        dets = [fresh.project(c, xyz) for c in range(N_CAM)]
        # 32 million pairs at the first level, of which the 3D gate lets next to none through
        dense = [rng.random((16000 + c, 2)) * (SIDE - 1.0) for c in range(N_CAM)]
        wide = synth.IPRSettings(match_cam_count=N_CAM, tol_2d_px=0.07 * SIDE, tol_3d_mm=1e-7)
        s = synth.IPRSettings(match_cam_count=N_CAM, tol_2d_px=1.0, tol_3d_mm=0.06)
        p = _ffi.sm_params(s, VOLUME)
        used.upload_detections(dense)
        used.stereo_match(_ffi.sm_params(wide, VOLUME))
        lists, times = [], []
        for ctx in (fresh, used):
            ctx.upload_detections(dets)
            n_cand, _ = ctx.stereo_match(p)
            lists.append(ctx.candidates(n_cand))
            times.append(_time(ctx, p))
        print(f"{n} detections: fresh {times[0] * 1e6:.0f} us, after a dense frame "
              f"{times[1] * 1e6:.0f} us")
        for a, b in zip(*lists):
            assert np.array_equal(a, b)
        assert len(lists[0][0]) > n // 2
        assert times[1] <= 1.3 * times[0]
    finally:
        fresh.close()
        used.close()
