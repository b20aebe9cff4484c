"""The FP32 shake of ROIs above 64 pixels: 32 lanes an object up to two waves of 148 x 16 objects, 8
beyond where four blocks' ROIs fit an SM's shared memory, else 32.  One object more, out of every
camera's sight, does not change a bit of the others, scores included."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
LIMIT = 2 * 148 * 16


@pytest.mark.parametrize("n_cam,radius,ratio,kind", [
    (2, 4.0, 2, "pinhole"), (4, 3.0, 2, "pinhole"), (4, 2.25, 2, "pinhole"), (6, 2.25, 2, "poly"),
    (6, 2.5, 2, "poly"),  # three blocks
    (8, 4.0, 2, "pinhole"), (4, 1.5, 2, "pinhole")])
def test_widths_of_large_rois_give_the_same_bits(n_cam, radius, ratio, kind):
    rng = np.random.default_rng(n_cam)
    side = (256, 256) if kind == "poly" else (240, 301)
    if kind == "poly":
        cams = synth.poly_rig(n_cam, side[0], VOLUME, seed=n_cam)
    else:
        cams = synth.ring_rig(n_cam, *side, min(synth.focal_for_volume(n_cam, side[0], VOLUME,
                                                                       fill=1.3)))
    lo, hi = np.array(VOLUME[0::2]), np.array(VOLUME[1::2])
    xyz = lo + (hi - lo) * rng.random((LIMIT, 3))
    imgs = [rng.integers(0, 200, side).astype(np.uint8) for _ in cams]
    start = xyz + rng.normal(0, 0.03, xyz.shape)
    table = synth.otf_grid(n_cam, (2, 2, 2), (150.0, 220.0), (0.2, 0.6), seed=1)
    table[3] = rng.uniform(-1.0, 1.0, table[3].shape)
    s = synth.IPRSettings(radius_obj=radius, ratio_augimg=ratio, n_shake_loop=2)
    out = []
    for objects in (start, np.concatenate([start, [[1e4, 1e4, 1e4]]])):
        ctx = _ffi.Context(0)
        try:
            ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
            ctx.upload_otf(2, 2, 2, VOLUME, table)
            ctx.upload_images(imgs)
            ctx.upload_objects(objects)
            ctx.shake(_ffi.shake_params(s, 0))
            out.append(ctx.objects())
        finally:
            ctx.close()
    for name in ("xyz", "uv", "score"):
        assert np.array_equal(out[0][name], out[1][name][:LIMIT]), name
    assert np.max(np.abs(out[0]["xyz"] - start)) > 0.0
