"""Ways through the separable 3D vote: host outputs in slabs, a volume cut into
z-slabs, and Gaussians of any width against the window."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_vote3_sep import THREADS, kernels_of, receivers_of, rel, spd_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(164, 160, 168), (173, 160, 160)])
def test_host_outputs_in_slabs_equal_device_outputs(shape):
    """Receiver planes leave in slabs as their windows complete: the same sums,
    the same bits."""
    import torch
    import tiralib_gb300 as tv
    vol = np.random.default_rng(8).normal(size=shape).astype(np.float32)
    kw = dict(sigma_st=1.5, sigma1=3.0, w=0, samples=20, out_layout="planes", evecs="cartesian")
    host, names = kernels_of(lambda: tv.pipeline3(vol, **kw))
    assert "k_sep_xy" in names
    dev = tv.pipeline3(torch.from_numpy(vol).cuda(), **kw)
    for h, d in zip(host, dev):
        np.testing.assert_array_equal(h, d.cpu().numpy())


def test_host_field_in_several_passes_and_slabs():
    """10 planes a pass at 1001 x 1003 and 17 exponentials would be 23 GB of
    sums: planes one by one, receivers handed out eight at a time."""
    import torch
    import tiralib_gb300 as tv
    T = np.tile(spd_field((10, 143, 59), 6), (1, 7, 17, 1, 1))
    T = np.ascontiguousarray(T[..., [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]])
    kw = dict(w=25, sigma1=4.0, layout="sym6", out_layout="sym6", evals=True)
    (h, eh, _), names = kernels_of(lambda: tv.vote3(T, **kw))
    assert "k_sep_xy" in names
    d, ed, _ = tv.vote3(torch.from_numpy(T).cuda(), **kw)
    np.testing.assert_array_equal(h, d.cpu().numpy())
    np.testing.assert_array_equal(eh, ed.cpu().numpy())


@pytest.mark.parametrize("parts", [2, 7])
def test_z_slabs_of_a_volume(parts):
    """A slab's passes begin at its own first plane, and a thin slab may be
    voted pair by pair: either is within 7e-6 of the exact vote of the same
    voters, per receiver (test_gpu_vote3_sep), and the tolerance is twice that."""
    import tiralib_gb300 as tv
    from tiralib_gb300 import slabs
    vol = np.random.default_rng(parts).normal(size=(90, 64, 72)).astype(np.float32)
    (out, _, _), names = kernels_of(lambda: tv.pipeline3(vol, 1.0, 3.0, w=0, samples=20, out_layout="planes",
                                                         evecs="cartesian"))
    assert "k_sep_xy" in names
    got = np.concatenate([slabs.pipeline3_slab(vol, z0, z1, 1.0, 3.0)[0] for z0, z1 in slabs.partition(90, parts)],
                         axis=1)
    flat = lambda o: np.moveaxis(o, 0, -1).reshape(-1, 6).astype(np.float64)
    assert rel(flat(got), flat(out)).max() < 1.4e-5


@pytest.mark.parametrize("sigma,sigma2,w", [(2.0, 5.0, 31), (4.0, 0.6, 25), (1.0, 4.0, 0), (3.0, 3.0, 0),
                                            (3.0, 2.999, 0),
                                            (10.0, 0.0, 41), (1.0, 0.0, 25), (0.6, 0.0, 21)])
def test_gaussians_of_any_width(sigma, sigma2, w):
    """The second Gaussian wider, narrower, equal and nearly so; one Gaussian
    wider than its window, and windows of 12 and 17 sigma, past which FP32 has
    no weight left."""
    import torch
    import tiralib_gb300 as tv
    shape = (40, 70, 90)
    T = spd_field(shape, 11)
    (out, _, _), names = kernels_of(lambda: tv.vote3(torch.from_numpy(T).cuda(), sigma, sigma2, w=w, parity=False,
                                                     out_layout="sym6"))
    assert "k_sep_xy" in names
    rec = receivers_of(shape, 3, 200)
    ww = w or 2 * int(np.float32(3.0) * np.float32(max(sigma, sigma2))) + 1
    ref = O.tensorvote3_f64(T, sigma, sigma2, ww, 1, receivers=rec, threads=THREADS).reshape(-1, 6)[rec]
    assert rel(out.cpu().numpy().reshape(-1, 6)[rec].astype(np.float64), ref).max() < 1e-5
