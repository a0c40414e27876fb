"""A vote of no term (stick, plate and ball off): zero tensors and their
eigenpairs in every output, at every power and from host arrays of the size
that is voted in slabs."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

OFF = dict(stick=False, plate=False, ball=False)


@pytest.mark.parametrize("power", [2, 32])
@pytest.mark.parametrize("parity", [True, False])
def test_no_terms_at_a_power_writes_every_output(power, parity):
    import torch
    import tiralib_gb300 as tv
    T = torch.ones((5, 6, 7, 3, 3), device="cuda")
    junk = [torch.full((5 * 6 * 7 * 9,), 7.0, device="cuda") for _ in range(20)]
    del junk                                               # what the outputs' memory holds before
    out, ev, vec = tv.vote3(T, 1.5, w=5, power=power, parity=parity, out_layout="sym6", evals=True, evecs="cartesian",
                            **OFF)
    assert float(out.abs().max()) == 0.0
    assert float(ev.abs().max()) == 0.0
    frame = O.evecs3cart(np.zeros((1, 9), np.float32), np.zeros((1, 3), np.float32))[0]
    np.testing.assert_array_equal(vec.cpu().numpy().reshape(-1, 3, 3), np.broadcast_to(frame, (5 * 6 * 7, 3, 3)))


@pytest.mark.parametrize("power", [1, 2])
def test_no_terms_on_a_large_host_field(power):
    import tiralib_gb300 as tv
    T = np.ones((164, 160, 168, 6), np.float32)
    for _ in range(2):                                     # the second output may land on the first one's memory
        out, _, _ = tv.vote3(T, 1.5, w=5, power=power, layout="sym6", out_layout="sym6", **OFF)
        assert out.min() == 0.0 and out.max() == 0.0
        out.fill(7.0)
        del out
