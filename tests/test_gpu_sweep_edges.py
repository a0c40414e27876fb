"""The parameter sweep where its launches divide: windows on both sides of the
widest that is staged, powers of 1 and above on fields that fill the GPU with
one set and fields that do not, entry tables past one launch's share."""
import numpy as np
import pytest

from test_gpu_sweep_batch import field

pytestmark = pytest.mark.gpu


def check(H, W, params, samples=20, plate=True):
    """A set's field and score do not depend on the sets it is voted with: the
    same entries and the same order of sums, whichever launch, bands and kernel
    the others bring.  (One set against a single vote: test_gpu_sweep_batch.)"""
    from tiralib_gb300 import metrics, optimize
    I, G = field(H, W, 1), field(H, W, 2)
    scores, fields = optimize.tk_sweep(G, I, params, samples=samples, plate=plate, return_fields=True)
    np.testing.assert_allclose(optimize.tk_sweep(G, I, params, samples=samples, plate=plate), scores, rtol=1e-10)
    for k, p in enumerate(params):
        _, alone = optimize.tk_sweep(G, I, [p], samples=samples, plate=plate, return_fields=True)
        np.testing.assert_array_equal(fields[k], alone[0])
        assert np.isfinite(fields[k]).all() and np.abs(fields[k]).max() > 0
        assert abs(scores[k] - metrics.simf(G, fields[k])) <= 1e-10 * abs(scores[k])


@pytest.mark.parametrize("params", [
    [(57.7, 0.0, 1), (58.0, 0.0, 1), (1.0, 0.0, 2), (58.4, 2.0, 3)],       # windows of 347 and 349 pixels
    [(29.5, 0.0, 1), (29.8, 0.0, 1), (2.0, 1.0, 1)],                       # 177 and 179: two CTAs per SM and one
])
def test_windows_at_the_staging_limits(params):
    check(33, 45, params)


@pytest.mark.parametrize("H,W", [(16 * 32, 19 * 32), (16 * 32, 19 * 32 - 32)])
def test_powers_apart_on_fields_that_fill_the_gpu(H, W):
    check(H, W, [(2.0, 0.0, 1), (1.5, 2.0, 3), (4.0, 0.0, 2), (3.0, 1.0, 1)], samples=7)


def test_entry_tables_past_one_launch():
    """73 windows of 341 pixels are 8.5 M entries, a launch's share is 8.4 M."""
    from tiralib_gb300 import optimize
    I, G = field(20, 24, 3), field(20, 24, 4)
    params = [(56.7 + 0.002 * k, 0.0, 1 + k % 3) for k in range(73)]
    scores = optimize.tk_sweep(G, I, params)
    some = [0, 71, 72]
    np.testing.assert_allclose(optimize.tk_sweep(G, I, [params[k] for k in some]), scores[some], rtol=1e-10)
