"""The separable 3D vote of planes whose sums over all exponentials pass the
scratch's 2 GiB: exponentials in several passes."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_vote3_sep import THREADS, kernels_of, receivers_of, rel, spd_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma2", [0.0, 2.0])
def test_wide_planes(sigma2):
    """1001 x 1003: 34 sums of 17 exponentials are 2.32 GB a plane.  The
    separable vote's tolerance (test_gpu_vote3_sep): 1e-5 per receiver."""
    import torch
    import tiralib_gb300 as tv
    shape, sigma, hw = (8, 1001, 1003), 4.0, 12
    T = np.tile(spd_field((8, 143, 59), 5), (1, 7, 17, 1, 1))
    dev = torch.from_numpy(np.ascontiguousarray(T[..., [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]])).cuda()
    tv.memory_stats(reset_peak=True)
    (out, _, _), names = kernels_of(lambda: tv.vote3(dev, sigma, sigma2, w=25, parity=False, layout="sym6",
                                                     out_layout="sym6"))
    assert "k_sep_xy" in names
    # padded moments (rows of 1024 + 24, 1008 of them), voted planes, the sums
    assert tv.memory_stats()[1] <= 15 * 4 * 8 * 1008 * 1048 + 6 * 4 * 8 * 1001 * 1003 + (2 << 30)
    rec = receivers_of(shape, 1, 100)
    ref = O.tensorvote3_f64(T, sigma, sigma2, 2 * hw + 1, 1, receivers=rec, threads=THREADS).reshape(-1, 6)[rec]
    assert rel(out.cpu().numpy().reshape(-1, 6)[rec].astype(np.float64), ref).max() < 1e-5
