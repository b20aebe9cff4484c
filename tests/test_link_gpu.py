"""The linking of short tracks to new particles (STB::linkShortTrack, src/srcSTB/STB.cpp:743-872)
against a numpy restatement: displacement of the long tracks around, weighted by distance, within
a radius that grows in five steps; the nearest new particle around the estimate; first come, first
served.  With long tracks, with a few (short tracks out of their reach) and without, and a search
radius that needs the larger steps.  The lists are compared exactly: what is appended are the
particles themselves, and no decision of these scenes lies within rounding of its limit."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
SHORT = 1  # index of the active short tracks
NEAR = 1e-9


def _link(p, key, disp, obj, base_r):
    """Object linked to a short track that ends at p, or -1."""
    fac = 1.0
    d2 = np.sum((key - p) ** 2, axis=1)
    for step in range(5):
        if step:
            fac *= 1.1
        R = base_r * fac
        near = d2 < (3.0 * base_r * fac) ** 2
        vel = np.zeros(3)
        if near.any():
            L2 = np.clip(0.64 * d2[near].mean(), (0.1 * R) ** 2, (0.8 * R) ** 2)
            w = 1.0 / (1.0 + d2[near] / (L2 + 1e-12))
            vel = (w[:, None] * disp[near]).sum(axis=0) / w.sum()
        for q in ([p + vel] if near.any() else [p + vel, p]):
            e2 = np.sum((obj - q) ** 2, axis=1)
            j = int(np.argmin(e2))
            assert abs(np.sqrt(e2[j]) - R) > NEAR  # not a matter of rounding
            if e2[j] < R * R:
                return j
    return -1


def _rows(tid, frame, xyz):
    """A track list as the tracks' (frames, points)."""
    cut = np.flatnonzero(np.diff(tid)) + 1
    return list(zip(np.split(frame, cut), np.split(xyz, cut))) if len(tid) else []


@pytest.mark.parametrize("n,n_long,base_r", [(700, 350, 0.35), (700, 350, 0.2), (700, 350, 0.08), (700, 6, 0.3),
                                             (400, 0, 0.5), (5, 3, 0.5)])
def test_short_tracks_link_as_restated(n, n_long, base_r):
    seq = synth.make_sequence(n_particles=n, n_frames=5, n_cam=4, n_row=384, n_col=384,
                              focal=1900.0, volume=VOLUME, a=200.0, noise=2.0, bits=8, gamma=4e3,
                              r_core=6.0, drift=(5.0, 0.0, 0.0), seed=n)
    rng = np.random.default_rng(n_long)
    # particles that are there in all frames
    stay = [i for i in range(n) if all(ids[i] == i for ids in seq.ids)]
    stay = list(rng.permutation(stay))
    long_p, rest = stay[:n_long], stay[n_long:]
    short_p = rest[: max(2, (4 * len(rest)) // 5)]
    ipr = synth.IPRSettings(n_loop_ipr=2, n_shake_loop=2)
    stb = synth.STBSettings(radius_search_track=base_r)
    ctx = _ffi.Context(0)
    try:
        ctx.upload_cameras([_ffi.camera_desc(c) for c in seq.cams])
        ctx.upload_otf(2, 2, 2, seq.volume, synth.otf_table_array(4, seq.otf_abc))
        ctx.stb_configure(_ffi.stb_params(ipr, stb, VOLUME, 0, 4, 1))

        def put(which, particles, first):
            tid = np.repeat(np.arange(len(particles)), [4 - f for f in first])
            fr = np.concatenate([np.arange(f, 4) for f in first]) if particles else []
            xyz = (np.concatenate([[seq.truth[t][p] for t in range(f, 4)]
                                   for p, f in zip(particles, first)]) if particles
                   else np.zeros((0, 3)))
            ctx.stb_set_tracks(which, tid, fr, xyz)

        put(0, long_p, [0] * len(long_p))
        put(SHORT, short_p, list(2 + np.arange(len(short_p)) % 2))  # two points or one
        before = _rows(*ctx.stb_tracks(SHORT))
        ctx.upload_images(seq.frames[4])
        ctx.stb_process_frame(4)
        _, n_ext, n_new = ctx.stb_counts()
        objects = ctx.stb_frame_objects()
        after = _rows(*ctx.stb_tracks(SHORT))
    finally:
        ctx.close()
    assert len(objects) == n_ext + n_new and n_new > 0
    extended, new = objects[:n_ext], objects[n_ext:]
    assert n_ext == len(long_p)  # none was flagged, so the extended are in the list's order
    last = np.array([seq.truth[3][p] for p in long_p]).reshape(-1, 3)
    key, disp = last.astype(np.float32).astype(np.float64), extended - last
    owner, want = {}, []
    for fr, xyz in before:
        j = _link(xyz[-1], key, disp, new, base_r)
        if j >= 0 and j not in owner:
            owner[j] = True
            want.append((np.append(fr, 4), np.vstack([xyz, new[j]])))
    print(f"{len(before)} short tracks, {len(want)} linked, {n_ext} long, {n_new} new")
    assert len(want) > 0 or base_r < 0.1  # nothing is that near
    want += [(np.array([4]), new[j:j + 1]) for j in range(len(new)) if j not in owner]
    assert len(after) == len(want)
    for (fa, xa), (fw, xw) in zip(after, want):
        assert np.array_equal(fa, fw) and np.array_equal(xa, xw)
