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


def spiral(n):
    """A background path one pixel wide from the border to the middle of an
    n x n image, in foreground walls, with closed cells beside it."""
    fg = np.ones((n, n), bool)
    y, x, dy, dx = 0, 0, 0, 1
    fg[0, 0] = False
    for length in [n - 1] + [v for k in range(n - 1, 0, -2) for v in (k, k)]:
        for _ in range(length):
            y, x = y + dy, x + dx
            if not (0 <= y < n and 0 <= x < n):
                break
            fg[y, x] = False
        dy, dx = dx, -dy
    return fg


@pytest.mark.parametrize("mask", [
    spiral(401), spiral(401)[:, ::-1], ~spiral(400), spiral(97).T,
    np.indices((1, 1000)).sum(0) % 3 == 0, np.indices((1000, 1)).sum(0) % 3 == 0,
    np.pad(np.zeros((300, 700), bool), 1, constant_values=True),           # one hole whose rows span many warps
    np.pad(np.tile(np.pad(np.zeros((1, 1), bool), 1, constant_values=True), (90, 90)), 1),
], ids=["spiral", "mirrored", "walls", "transposed", "1xN", "Nx1", "wide hole", "cells"])
def test_fill_of_long_and_thin_background(mask):
    from tiralib_gb300 import reconstruct as R
    mask = np.ascontiguousarray(mask)
    np.testing.assert_array_equal(R.saliency_threshold(field_of(mask), fill=True, threshold=0.5),
                                  ndimage.binary_fill_holes(mask))


@pytest.mark.parametrize("radius", [7, 8, 9, 12])
@pytest.mark.parametrize("H,W", [(33, 31), (129, 200), (1, 90)])
def test_closing_on_both_sides_of_the_one_pass_radius(radius, H, W):
    from tiralib_gb300 import reconstruct as R
    m = np.random.default_rng(radius).random((H, W)) < 0.02
    want = ndimage.binary_fill_holes(ndimage.binary_closing(m, np.ones((2 * radius + 1,) * 2, bool)))
    np.testing.assert_array_equal(R.saliency_threshold(field_of(m), fill=True, threshold=0.5, close_radius=radius), want)
