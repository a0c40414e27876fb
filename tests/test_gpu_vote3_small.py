"""The pair-by-pair 3D vote on either side of the volume at which a CTA takes
four receiver planes instead of one, and in slabs whose last one is short."""

import numpy as np
import pytest
from oracle import oracle as O
from test_gpu_vote3_sep import THREADS, kernels_of, spd_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 152, 32), (24, 153, 32), (25, 145, 32), (3, 48, 608), (3, 48, 609)])
def test_both_plane_counts_match_fp64_oracle(shape):
    """114 groups of 32 x 8 x 4 receivers and one row or column more.  A
    receiver has 5^3 pairs of some 50 FP32 operations, folded plane by plane
    into compensated sums: sqrt(25 * 50) 2^-24 = 2.1e-6 of the largest entry."""
    import torch
    import tiralib_gb300 as tv
    T = spd_field(shape, sum(shape))
    (out, _, _), names = kernels_of(lambda: tv.vote3(torch.from_numpy(T).cuda(), 0.9, w=5, parity=False,
                                                     out_layout="sym6"))
    assert "k_vote3_fast" in names
    ref = O.tensorvote3_f64(T, 0.9, 0.0, 5, 1, threads=THREADS)
    assert np.abs(out.cpu().numpy() - ref).max() <= 2.1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("sigma,w,kw", [(1.2, 7, {}), (0.8, 5, {"ball": True})])
def test_a_short_last_slab_votes_like_the_whole(sigma, w, kw):
    """172 planes in slabs of 24: the last slab's 4 planes alone would be a
    small volume."""
    import torch
    import tiralib_gb300 as tv
    rng = np.random.default_rng(9)
    A = rng.normal(size=(4096, 3, 3)).astype(np.float32)
    shape = (172, 160, 160)
    T = np.ascontiguousarray((A @ np.swapaxes(A, -1, -2))[rng.integers(0, 4096, size=int(np.prod(shape)))]
                             .reshape(shape + (3, 3)), np.float32)
    (host, _, _), names = kernels_of(lambda: tv.vote3(T, sigma, w=w, **kw))
    assert "k_vote3_fast" in names
    dev, _, _ = tv.vote3(torch.from_numpy(T).cuda(), sigma, w=w, **kw)
    np.testing.assert_array_equal(host, dev.cpu().numpy())
