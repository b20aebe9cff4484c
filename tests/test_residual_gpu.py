"""The residual image (windows splatted by atomic maxima, then one streaming pass) against the
restated reference (Shake::calResidueImage) at ragged widths, for every image type, with windows
that overlap, cross the border and lie outside.  FP64 to 1e-9: exp() may round differently, by an
ulp of values up to 200.  FP32 to 5e-3, as for the existing residual test: single-precision
exponents (relative error 1e-7 of up to about 10) on amplitudes of 200."""
import numpy as np
import pytest

from oracle.restated import Restated
from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)


@pytest.mark.parametrize("n", [0, 1, 40, 30_000])  # 2 pairs a warp, and 32
@pytest.mark.parametrize("rows,cols,dtype", [
    (64, 64, np.uint8), (33, 61, np.uint8), (50, 63, np.uint16), (7, 66, np.float32),
    (61, 37, np.float64), (5, 3, np.uint16)])
def test_residual_against_the_restatement(rows, cols, dtype, n):
    n_cam = 3
    rng = np.random.default_rng(rows * cols + n)
    cams = synth.ring_rig(n_cam, rows, cols,
                          min(synth.focal_for_volume(n_cam, max(rows, cols), VOLUME)))
    imgs = [rng.integers(0, 250, (rows, cols)).astype(dtype) for _ in range(n_cam)]
    lo, hi = np.array(VOLUME[0::2]), np.array(VOLUME[1::2])
    xyz = lo + (hi - lo) * (1.3 * rng.random((n, 3)) - 0.15)
    table = synth.otf_grid(n_cam, (3, 2, 2), (150.0, 200.0), (0.3, 0.9), seed=3)
    oracle = Restated()
    s = synth.IPRSettings(radius_obj=2.0)
    ctx = _ffi.Context(0)
    try:
        ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
        ctx.upload_otf(3, 2, 2, VOLUME, table)
        ctx.upload_images(imgs)
        ctx.upload_objects(xyz)
        for precision, atol in ((1, 1e-9), (0, 5e-3), (0, 5e-3)):  # the planes are cleared
            ctx.residual(_ffi.shake_params(s, precision))
            for c in range(n_cam):
                uv = ctx.project(c, xyz) if n else np.zeros((0, 2))
                otf = oracle.otf_param((3, 2, 2), VOLUME, table, n_cam, c, xyz)
                want = oracle.residual(imgs[c], uv, otf, 2.0, 1)
                got = ctx.residual_image(c, (rows, cols))
                assert np.max(np.abs(got - want)) <= atol, (precision, c)
    finally:
        ctx.close()
