"""The two-pass detector at its bands' edges (512 chunks of 16 bytes a band, one row at least)
against the restated Imgio detection: integer images exactly; float images the same spots in the
same order, positions to 1e-9 px (log() may round differently)."""
import ctypes as C

import numpy as np
import pytest

from oracle.restated import Restated
from pyopenlpt_b200 import _ffi

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _detect(img, threshold):
    H, W = img.shape
    row = W * img.dtype.itemsize
    pitch = (row + 15) // 16 * 16
    padded = np.zeros((H, pitch), np.uint8)
    padded[:, :row] = np.ascontiguousarray(img).view(np.uint8).reshape(H, row)
    dev = torch.from_numpy(padded).cuda()
    cap = (H * W + 1) // 2  # what the entry asks for
    x, y = (torch.zeros(cap, dtype=torch.float64, device="cuda") for _ in range(2))
    rc = torch.zeros((cap, 2), dtype=torch.int32, device="cuda")
    n = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    st = _ffi.lib().olpt_find_peaks_noalloc(p(dev), _ffi._DTYPES[img.dtype], H, W,
                                            C.c_int64(pitch), C.c_double(threshold), p(x), p(y),
                                            p(rc), C.c_int64(cap), p(n), None)
    assert st == 0
    torch.cuda.synchronize()
    k = int(n.item())
    return np.stack([x.cpu().numpy()[:k], y.cpu().numpy()[:k]], 1)


@pytest.mark.parametrize("dtype,shape", [
    (np.uint8, (127, 64)), (np.uint8, (128, 64)), (np.uint8, (129, 64)), (np.uint8, (130, 50)),
    (np.uint8, (5, 8192)), (np.uint8, (5, 8193)), (np.uint8, (3, 16)), (np.uint8, (3, 17)),
    (np.uint16, (257, 32)), (np.uint16, (66, 129)), (np.uint16, (4, 4097)),
    (np.float32, (65, 63)), (np.float64, (65, 31)), (np.float64, (3, 3))])
@pytest.mark.parametrize("threshold", [0.0, 30.5, 190.0])
def test_bands_against_the_restatement(dtype, shape, threshold):
    rng = np.random.default_rng(shape[0] * 31 + shape[1])
    img = rng.integers(0, 200, shape).astype(dtype)
    if np.dtype(dtype).kind == "f":
        img += rng.random(shape).astype(dtype)
    got = _detect(img, threshold)
    want = Restated().find_peaks(img, threshold)
    assert got.shape == want.shape
    if np.dtype(dtype).kind == "f":
        assert np.all(np.abs(got - want) <= 1e-9)
    else:
        assert np.array_equal(got, want)
