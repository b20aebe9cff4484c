"""Contexts with different rigs at work at the same time: their kernels are the same device
functions, whose shared memory depends on the rig, so what one thread asks for must not take away
what another has been granted.  Every result equals that of the context on its own."""
import threading

import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
FRAMES = 64


def _at_once(jobs):
    """The jobs' results, each run by a thread of its own."""
    out, gate = [None] * len(jobs), threading.Barrier(len(jobs))

    def run(i):
        gate.wait()
        try:
            out[i] = jobs[i]()
        except Exception as e:  # noqa: BLE001 - handed to the test's thread
            out[i] = e

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in out:
        if isinstance(r, Exception):
            raise r
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [40, 148 * 16 + 1])  # 32 and 8 lanes an object in FP32
def test_shake_of_a_pinhole_and_a_polynomial_rig(n, precision):
    n_cam, side = 6, 128
    rng = np.random.default_rng(n)
    lo, hi = np.array(VOLUME[0::2]), np.array(VOLUME[1::2])
    xyz = lo + (hi - lo) * rng.random((n, 3))
    s = synth.IPRSettings(n_shake_loop=8)
    ctxs = []
    try:
        for cams in (synth.ring_rig(n_cam, side, side,
                                    min(synth.focal_for_volume(n_cam, side, VOLUME))),
                     synth.poly_rig(n_cam, side, VOLUME, seed=3)):
            ctx = _ffi.Context(0)
            ctxs.append(ctx)
            ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
            ctx.upload_otf(2, 2, 2, VOLUME, synth.otf_table_array(n_cam, (200.0, 0.5, 0.5)))
            ctx.upload_images([synth.render(c, xyz, 200.0, 0.5, 0.5, 2.0, 255, np.uint8, rng)
                               for c in cams])

        def job(ctx, times):
            for _ in range(times):
                ctx.upload_objects(xyz)
                ctx.shake(_ffi.shake_params(s, precision))
            return ctx.objects()

        want = [job(c, 1) for c in ctxs]
        got = _at_once([lambda c=c: job(c, 200) for c in ctxs])
        for g, w in zip(got, want):
            for name in ("xyz", "uv", "score", "flags"):
                assert np.array_equal(g[name], w[name]), name
    finally:
        for c in ctxs:
            c.close()


def test_predictive_fields_of_different_bins():
    """21 bins an axis take 107 KB of a block's shared memory, 11 bins 43 KB."""
    seq = synth.make_sequence(n_particles=40, n_frames=1, n_cam=2, n_row=64, n_col=64, focal=300.0,
                              volume=VOLUME, a=200.0, noise=0.0, bits=8, seed=1)
    ipr = synth.IPRSettings(n_loop_ipr=1, n_shake_loop=1, match_cam_count=2)
    stb = synth.STBSettings(pf_nx=2, pf_ny=2, pf_nz=2, n_initial_frames=FRAMES)
    bins = [21, 11, 21, 11, 11, 11]
    ctxs = []
    try:
        params = []
        for b in bins:
            ctx = _ffi.Context(0)
            ctxs.append(ctx)
            ctx.upload_cameras([_ffi.camera_desc(c) for c in seq.cams])
            ctx.upload_otf(2, 2, 2, VOLUME, synth.otf_table_array(2, seq.otf_abc))
            params.append(_ffi.stb_params(ipr, stb, VOLUME, 0, FRAMES - 1, 0))
            for k in range(3):
                params[-1].pf_nbin[k] = b

        def job(ctx, p, times):
            for _ in range(times):
                ctx.stb_configure(p)
                for t in range(FRAMES):  # the last one computes all fields
                    ctx.upload_images(seq.frames[0])
                    ctx.stb_process_frame(t)
            return [ctx.stb_tracks(k) for k in range(4)]

        want = [job(c, p, 1) for c, p in zip(ctxs, params)]
        got = _at_once([lambda c=c, p=p: job(c, p, 60) for c, p in zip(ctxs, params)])
        for g, w in zip(got, want):
            for a, b in zip(g, w):
                assert all(np.array_equal(x, y) for x, y in zip(a, b))
    finally:
        for c in ctxs:
            c.close()
