"""Thresholding, closing and hole filling away from the ordinary."""
import numpy as np
import pytest
from scipy import ndimage

pytestmark = pytest.mark.gpu


def field_of(sal):
    """A field whose saliency is `sal`, exactly: diagonal (sal, 0)."""
    f = np.zeros(sal.shape + (2, 2), np.float32)
    f[..., 0, 0] = sal
    return f


def test_otsu_of_an_infinite_range_is_zero():
    """No bin has a between-class variance that is a number: the threshold
    stays at its start, 0, and every positive saliency is above it."""
    from tiralib_gb300 import reconstruct as R
    v = np.random.default_rng(0).uniform(0.1, 1.0, (40, 50)).astype(np.float32)
    v[3, 4] = np.inf
    assert R._otsu_threshold(v.ravel()) == 0.0
    assert R.saliency_threshold(field_of(v)).all()


@pytest.mark.parametrize("H,W", [(65535 * 8, 3), (65535 * 8 + 1, 3), (600000, 5)])
def test_fill_of_an_image_taller_than_a_grid(H, W):
    """65535 blocks of 8 rows, one row more, and several rows more."""
    from tiralib_gb300 import reconstruct as R
    m = np.random.default_rng(H).random((H, W)) < 0.6
    got = R.saliency_threshold(field_of(m), fill=True, threshold=0.5)
    np.testing.assert_array_equal(got, ndimage.binary_fill_holes(m))
