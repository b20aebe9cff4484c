"""The fused inference of the learned proposal at its tiles' edges (128 rows a tile, one tile a
block at a time): rows do not depend on one another, so a shorter batch gives the same bits,
and the longest is held to the oracle within the bound of the existing forward test."""
import numpy as np
import pytest

from oracle import mlp_ref as R
from pyopenlpt_b200 import _ffi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cam", [2, 4, 5, 8])
def test_rows_at_the_tiles_edges(n_cam):
    rng = np.random.default_rng(n_cam)
    ctx = _ffi.Context(0)
    try:
        ctx.upload_cameras([_ffi.camera_desc(c) for c in synth.ring_rig(n_cam, 64, 64, 300.0)])
        n_in = R.n_in(n_cam)
        flat = R.init(n_cam, n_in)
        ctx.mlp_set_params(flat)
        full = 148 * 128 + 1  # one row beyond a tile for every SM
        x = np.clip(rng.normal(0.2, 0.3, (full, n_in)), -1, 2).astype(np.float32)
        got = ctx.mlp_forward(x)
        for n in (1, 127, 128, 129, 255, 257, 148 * 128):
            assert np.array_equal(ctx.mlp_forward(x[:n]), got[:n]), n
    finally:
        ctx.close()
    pick = np.r_[0:200, full - 200:full]
    want, _ = R.forward(flat, x[pick])
    assert np.max(np.abs(got[pick] - want)) < 3e-2
