"""The stereo expansion over every way its levels are run: without a look at the counts (up to
16,384 seeds), with one after each level, and with levels repeated because their pairs or paths
did not fit; against all tuples of detections whose epipolar distances are within the tolerance
both ways.  The 3D gates are opened, so that the 2D tests alone decide.  Both sides compute the
distances in FP64 from coordinates of order 1e3; tuples within 1e-7 px of the tolerance may
fall on either side."""
import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu


def _fundamental(a, b):
    """F with F x_a = the line of x_a on camera b (normal of unit length after scaling)."""
    R = b.R @ a.R.T
    t = b.T - R @ a.T
    tx = np.array([[0, -t[2], t[1]], [t[2], 0, -t[0]], [-t[1], t[0], 0]])
    K = [np.array([[c.fx, 0, c.cx], [0, c.fy, c.cy], [0, 0, 1.0]]) for c in (a, b)]
    return np.linalg.inv(K[1]).T @ tx @ R @ np.linalg.inv(K[0])


def _close(cams, dets, i, j, tol):
    """Pairs (of cameras i < j) whose larger distance is below tol + 1e-7, and which of them are
    below tol - 1e-7."""
    xi, xj = (np.c_[d, np.ones(len(d))] for d in (dets[i], dets[j]))
    li, lj = xi @ _fundamental(cams[i], cams[j]).T, xj @ _fundamental(cams[j], cams[i]).T
    li /= np.linalg.norm(li[:, :2], axis=1, keepdims=True)
    lj /= np.linalg.norm(lj[:, :2], axis=1, keepdims=True)
    out, sure = [], []
    for k in range(0, len(xi), 1024):
        d = np.maximum(np.abs(li[k:k + 1024] @ xj.T), np.abs(xi[k:k + 1024] @ lj.T))
        p = np.argwhere(d < tol + 1e-7)
        out.append(p + [k, 0])
        sure.append(d[p[:, 0], p[:, 1]] < tol - 1e-7)
    return np.concatenate(out), np.concatenate(sure)


@pytest.mark.parametrize("n_cam,n,side,tol", [
    (2, 1, 64, 1.0),
    (2, 300, 64, 6.0),       # more pairs than 8 a seed
    (3, 150, 64, 8.0),       # more paths than 16 a seed, at the last level
    (4, 60, 64, 12.0),       # and at an inner one
    (2, 16_384, 1024, 0.5),
    (2, 16_385, 1024, 0.5),  # a look at every level
    (2, 16_385, 512, 4.0),   # and its pairs do not fit
])
def test_candidates_are_the_tuples_within_the_tolerance(n_cam, n, side, tol):
    volume = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)
    cams = synth.ring_rig(n_cam, side, side, min(synth.focal_for_volume(n_cam, side, volume)))
    rng = np.random.default_rng(n * n_cam)
    dets = [rng.random((n + c, 2)) * (side - 1.0) for c in range(n_cam)]
    s = synth.IPRSettings(match_cam_count=n_cam, tol_2d_px=tol, tol_3d_mm=1e4)
    limit = (-1e6, 1e6, -1e6, 1e6, -1e6, 1e6)
    ctx = _ffi.Context(0)
    try:
        ctx.upload_cameras([_ffi.camera_desc(c) for c in cams])
        ctx.upload_detections(dets)
        runs = []
        for _ in range(2):  # the second over the buffers that the first one grew
            n_cand, _ = ctx.stereo_match(_ffi.sm_params(s, limit))
            runs.append(ctx.candidates(n_cand))
    finally:
        ctx.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    got = set(map(tuple, runs[0][0]))
    assert len(got) == len(runs[0][0])

    tuples, sure = _close(cams, dets, 0, 1, tol)
    for c in range(2, n_cam):
        # 2 = surely close, 1 = within 1e-7 of the tolerance
        ok = [np.zeros((len(dets[i]), len(dets[c])), np.int8) for i in range(c)]
        for i in range(c):
            p, q = _close(cams, dets, i, c, tol)
            ok[i][p[:, 0], p[:, 1]] = 1 + q
        worst = np.min([ok[i][tuples[:, i]] for i in range(c)], axis=0)
        at, new = np.nonzero(worst)
        sure = sure[at] & (worst[at, new] == 2)
        tuples = np.c_[tuples[at], new]
    assert set(map(tuple, tuples[sure])) <= got <= set(map(tuple, tuples))
    assert len(got) > 0 or n == 1
