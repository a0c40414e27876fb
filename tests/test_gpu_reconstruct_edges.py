"""Thresholding, closing and hole filling away from the ordinary."""
import numpy as np
import pytest

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
