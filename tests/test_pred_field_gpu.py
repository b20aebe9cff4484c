"""The predictive field's nodes against a numpy restatement of PredField::calPredField
(PredField.cpp:20-90) on the same objects.  The field's file holds nine digits of values up to
about 10 mm, and its sums of at most 1e5 exponentials are equal up to 1e-11: 1e-7 mm."""
import os

import numpy as np
import pytest

from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu

VOLUME = (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)


def _context(seq):
    ctx = _ffi.Context(0)
    ctx.upload_cameras([_ffi.camera_desc(c) for c in seq.cams])
    ctx.upload_otf(2, 2, 2, seq.volume, synth.otf_table_array(len(seq.cams), seq.otf_abc))
    return ctx


def _sequence(n, frames, seed):
    return synth.make_sequence(n_particles=n, n_frames=frames, n_cam=4, n_row=384, n_col=384,
                               focal=1900.0, volume=VOLUME, a=200.0, noise=2.0, bits=8, gamma=4e3,
                               r_core=6.0, drift=(5.0, 0.0, 0.0), seed=seed)


def _node(prev, curr, node, r, n_bin):
    """Displacement of one grid node."""
    a = curr[np.all(np.abs(curr - node) < r, axis=1)]
    b = prev[np.all(np.abs(prev - node) < r, axis=1)]
    if not len(a) or not len(b):
        return np.zeros(3)
    m, c = (n_bin - 1) / (4 * r), float((n_bin - 1) // 2)
    x = (m * (a[:, None] - b[None]) + c).reshape(-1, 3)
    pdf = np.zeros((n_bin,) * 3)
    for step in np.ndindex(3, 3, 3):
        # round() of the reference: halves away from zero (the bins are not negative)
        at = np.floor(x + 0.5).astype(int) - 1 + step
        ok = np.all((at >= 0) & (at < n_bin), axis=1)
        w = np.exp(-np.sum((at - x) ** 2, axis=1))
        np.add.at(pdf, tuple(at[ok].T), w[ok])
    if not pdf.max() > 1e-1:
        return np.zeros(3)
    pk = np.array(np.unravel_index(np.argmax(pdf), pdf.shape))
    out = np.zeros(3)
    for ax in range(3):
        if pk[ax] in (0, n_bin - 1):
            out[ax] = -2 * r if pk[ax] == 0 else 2 * r
            continue
        y = pk[ax] + np.array([-1.0, 0.0, 1.0])
        lo, hi = pk.copy(), pk.copy()
        lo[ax] -= 1
        hi[ax] += 1
        v = np.log(np.maximum([pdf[tuple(lo)], pdf[tuple(pk)], pdf[tuple(hi)]], 1e-4))
        num = (v[0] * (y[1] ** 2 - y[2] ** 2) - v[1] * (y[0] ** 2 - y[2] ** 2)
               + v[2] * (y[0] ** 2 - y[1] ** 2))
        yc = -0.5 * num / (v[0] * (y[2] - y[1]) - v[2] * (y[0] - y[1]) + v[1] * (y[0] - y[2]))
        out[ax] = ((yc if np.isfinite(yc) else y[1]) - c) / m
    return out


@pytest.mark.parametrize("n,n_bin,r", [(300, 11, 3.0), (300, 5, 3.0), (1200, 21, 2.5)])
def test_field_nodes_against_numpy(tmp_path, n, n_bin, r):
    seq = _sequence(n, 4, n)
    ipr = synth.IPRSettings(n_loop_ipr=2, n_shake_loop=2)
    stb = synth.STBSettings(pf_nx=5, pf_ny=4, pf_nz=3, pf_r=r)
    p = _ffi.stb_params(ipr, stb, VOLUME, 0, 3, 1, str(tmp_path) + "/")
    p.pf_smooth = 0
    for k in range(3):
        p.pf_nbin[k] = n_bin
    ctx = _context(seq)
    objects = []
    try:
        ctx.stb_configure(p)
        for t in range(4):
            ctx.upload_images(seq.frames[t])
            ctx.stb_process_frame(t)
        ctx.flush_track_files()
        for t in range(2):
            ctx.upload_images(seq.frames[t])
            objects.append(ctx.ipr_result(ctx.ipr_run(p.ipr))[0])
    finally:
        ctx.close()
    field = np.loadtxt(os.path.join(tmp_path, "PredField_1_2.csv"), delimiter=",")
    nodes = [np.linspace(VOLUME[2 * k], VOLUME[2 * k + 1], m) for k, m in enumerate((5, 4, 3))]
    want = np.array([_node(objects[0], objects[1], np.array([x, y, z]), r, n_bin)
                     for x in nodes[0] for y in nodes[1] for z in nodes[2]])
    assert np.any(want != 0.0)
    assert np.max(np.abs(field - want)) <= 1e-7
