"""The two-pass detector on rows wider than a band's 512 chunks of 16 bytes (each row is a band of
several rounds, of which some hold no spot) and on floating-point levels, whose fits it keeps
there: the restated detection's spots in its order, positions of floating-point levels to 1e-9 px
(log() may round differently), of integers exactly.  Levels that are not finite or below the
clamp take part."""
import numpy as np
import pytest

from oracle.restated import Restated
from tests.test_peaks_bands_gpu import _detect

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.0, 0.0002, 0.01, 1.0])
@pytest.mark.parametrize("dtype,shape", [
    (np.float32, (5, 2048)), (np.float32, (5, 2049)), (np.float32, (4, 9001)),
    (np.float64, (4, 1024)), (np.float64, (4, 1025)), (np.float64, (5, 5003)),
    (np.float64, (40, 130)), (np.uint16, (4, 9001)), (np.uint8, (3, 16_384))])
def test_wide_rows(dtype, shape, share):
    rng = np.random.default_rng(shape[1] + int(share * 1e4))
    img = rng.integers(0, 20, shape).astype(np.float64)
    spot = rng.random(shape) < share
    img[spot] += rng.integers(30, 200, int(spot.sum()))
    if np.dtype(dtype).kind == "f":
        img += rng.random(shape)
        odd = rng.random(shape) < 0.02
        img[odd] = rng.choice([np.nan, np.inf, -np.inf, -3.0], int(odd.sum()))
    img = img.astype(dtype)
    got, want = _detect(img, 30.0), Restated().find_peaks(img, 30.0)
    assert got.shape == want.shape
    if np.dtype(dtype).kind == "f":
        assert np.all(np.abs(got - want) <= 1e-9)
    else:
        assert np.array_equal(got, want)
