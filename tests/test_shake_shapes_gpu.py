"""The FP32 shake runs 32 lanes an object for up to 148 x 16 objects and 8 beyond.  Both form the
same sums, so one object more, out of every camera's sight, must not change a bit of the others:
over cameras, window radii (windows that are not a power of two wide, clipped at the borders)
and camera models."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
LIMIT = 148 * 16


@pytest.mark.parametrize("n_cam,radius,ratio,kind", [
    (2, 2.0, 2, "pinhole"), (3, 1.0, 2, "pinhole"), (4, 2.5, 3, "pinhole"), (5, 2.0, 2, "poly"),
    (6, 2.0, 2, "pinhole"), (6, 1.5, 2, "poly"), (8, 2.0, 2, "pinhole")])
def test_both_widths_give_the_same_bits(n_cam, radius, ratio, kind):
    rng = np.random.default_rng(n_cam)
    side = (256, 256) if kind == "poly" else (240, 301)
    if kind == "poly":
        cams = synth.poly_rig(n_cam, side[0], VOLUME, seed=n_cam)
    else:
        cams = synth.ring_rig(n_cam, *side, min(synth.focal_for_volume(n_cam, side[0], VOLUME,
                                                                       fill=1.1)))
    lo, hi = np.array(VOLUME[0::2]), np.array(VOLUME[1::2])
    xyz = lo + (hi - lo) * rng.random((LIMIT, 3))
    imgs = [synth.render(c, xyz, 200.0, 0.5, 0.5, 2.0, 255, np.uint8, rng) for c in cams]
    start = xyz + rng.normal(0, 0.03, xyz.shape)
    far = np.array([[1e4, 1e4, 1e4]])
    s = synth.IPRSettings(radius_obj=radius, ratio_augimg=ratio, n_shake_loop=2)
    out = []
    for objects in (start, np.concatenate([start, far])):
        ctx = _ffi.Context(0)
        try:
            ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
            ctx.upload_otf(2, 2, 2, VOLUME, synth.otf_table_array(n_cam, (200.0, 0.5, 0.5)))
            ctx.upload_images(imgs)
            ctx.upload_objects(objects)
            ctx.shake(_ffi.shake_params(s, 0))
            out.append(ctx.objects())
        finally:
            ctx.close()
    for name in ("xyz", "uv"):
        assert np.array_equal(out[0][name], out[1][name][:LIMIT]), name
    assert np.max(np.abs(out[0]["xyz"] - start)) > 0.0
