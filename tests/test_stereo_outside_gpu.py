"""Detections far outside the image (only a caller's own lists hold such): they seed paths of the
stereo search like any other, and FP64 decides their 2D tests at the tolerance."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth
from tests.test_stereo_levels_gpu import _close, _fundamental

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [12.0, 3000.0])
@pytest.mark.parametrize("side,tol", [(64, 0.5), (301, 1.0)])
def test_seeds_outside_the_image(side, tol, sides):
    """Seeds at `sides` image sides on the line of a detection of the other camera, offset by the
    tolerance and up to 2e-3 px around it; a tuple is a match when both epipolar distances are
    within the tolerance (either way within 1e-7 px of it: coordinates of order 1e6 in FP64)."""
    volume = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
    cams = synth.ring_rig(2, side, side, min(synth.focal_for_volume(2, side, volume)))
    rng = np.random.default_rng(side)
    n = 400
    inside = rng.random((n + 1, 2)) * (side - 1.0)
    lines = np.c_[inside[:n], np.ones(n)] @ _fundamental(cams[1], cams[0]).T
    lines /= np.linalg.norm(lines[:, :2], axis=1, keepdims=True)
    along = np.c_[-lines[:, 1], lines[:, 0]] * rng.choice([-1.0, 1.0], (n, 1))
    off = rng.choice([-1.0, 1.0], n) * (tol + rng.uniform(-2e-3, 2e-3, n))
    seeds = (lines[:, :2] * (off - lines[:, 2])[:, None]
             + along * (sides * side * rng.uniform(1.0, 1.5, (n, 1))))
    dets = [seeds, inside]
    s = synth.IPRSettings(match_cam_count=2, tol_2d_px=tol, tol_3d_mm=1e9)
    limit = (-1e12, 1e12, -1e12, 1e12, -1e12, 1e12)
    ctx = _ffi.Context(0)
    try:
        ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
        ctx.upload_detections(dets)
        n_cand, _ = ctx.stereo_match(_ffi.sm_params(s, limit))
        got = set(map(tuple, ctx.candidates(n_cand)[0]))
    finally:
        ctx.close()
    pairs, sure = _close(cams, dets, 0, 1, tol)
    assert set(map(tuple, pairs[sure])) <= got <= set(map(tuple, pairs))
    assert 50 < len(got)
