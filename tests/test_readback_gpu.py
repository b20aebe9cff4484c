"""Results read back to the host: through the context's pinned block (up to 1 MB a call) and
directly above it, and the matches gathered on the device against those picked from the
downloaded candidates.  All comparisons are exact."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)


def _context(n_cam=4, side=256):
    f = min(synth.focal_for_volume(n_cam, side, VOLUME, fill=1.05))
    cams = synth.ring_rig(n_cam, side, side, f)
    ctx = _ffi.Context(0)
    ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
    return ctx, cams


@pytest.mark.parametrize("n", [1, 255, 257, 43_690, 43_691, 65_536, 65_537])
def test_detections_come_back_as_they_went(n):
    # 24 B a detection: 43,690 fill the block; 65,537 positions alone exceed it
    ctx, cams = _context()
    try:
        rng = np.random.default_rng(n)
        xy = [rng.random((max(1, n - 3 * c), 2)) * 255.0 for c in range(len(cams))]
        ctx.upload_detections(xy)
        for c, want in enumerate(xy):
            got, _ = ctx.get_peaks(c, len(want))
            assert np.array_equal(got, want)
            assert np.array_equal(ctx.get_peaks(c, 1)[0], want[:1])  # a shorter list
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [1, 40, 3000])
def test_matches_before_and_after_the_candidates(n):
    ctx, cams = _context(4, 512)
    try:
        rng = np.random.default_rng(n)
        lo, hi = np.array(VOLUME[0::2]), np.array(VOLUME[1::2])
        xyz = lo + (hi - lo) * rng.random((n, 3))
        ctx.upload_detections([np.stack([ctx.project(c, xyz)], 0).reshape(-1, 2)
                               for c in range(len(cams))])
        s = synth.IPRSettings(match_cam_count=4, tol_2d_px=1.0, tol_3d_mm=0.05)
        n_cand, n_match = ctx.stereo_match(_ffi.sm_params(s, VOLUME))
        ids, x = ctx.matches(n_match)  # gathered on the device
        cids, _, cx = ctx.candidates(n_cand)  # the whole list is on the host from here on
        ids2, x2 = ctx.matches(n_match)
        assert n_match > 0
        assert np.array_equal(ids, ids2) and np.array_equal(x, x2)
        rows = {tuple(r): i for i, r in enumerate(cids)}
        at = [rows[tuple(r)] for r in ids]
        assert at == sorted(at) and np.array_equal(cx[at], x)
    finally:
        ctx.close()
