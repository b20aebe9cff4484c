"""Lists and grids beyond 2^24 entries are refused (status 5, unsupported), the largest within are
not: the grid of one camera, the points and the candidates of the prune."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

MOST = 1 << 24


@pytest.mark.parametrize("cols,fits", [(4096, True), (4097, False)])
def test_grid_of_a_camera(cols, fits):
    cams = synth.ring_rig(3, 4096, cols, 4000.0)
    s = synth.IPRSettings(match_cam_count=3, idmap_cell_px=1, tol_2d_px=1.0, tol_3d_mm=0.1)
    p = _ffi.sm_params(s, (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0))
    xyz = np.random.default_rng(0).random((50, 3)) * 10.0 - 5.0
    ctx = _ffi.Context(0)
    try:
        ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
        ctx.upload_detections([ctx.project(c, xyz) for c in range(3)])
        if fits:  # three grids of 2^24 cells
            assert ctx.stereo_match(p)[1] == 50
        else:
            with pytest.raises(_ffi.OlptError, match="16M entries"):
                ctx.stereo_match(p)
    finally:
        ctx.close()


@pytest.mark.parametrize("candidates,points", [(MOST + 1, MOST), (1, MOST + 1)])
def test_prune(candidates, points):
    ids = (np.arange(candidates) % points).astype(np.int32)[:, None]  # pools of one or two
    ctx = _ffi.Context(0)
    try:
        with pytest.raises(_ffi.OlptError, match="16M entries"):
            ctx.prune_matches(ids, np.zeros(candidates), [points])
        assert ctx.prune_matches(ids[:1], np.zeros(1), [MOST]).tolist() == [True]
    finally:
        ctx.close()
