"""Calls from several host threads at once, each with a window of its own:
the kernels' shared-memory limits are one value per kernel in the process, so
no call may lower another's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spd(shape, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn(shape + (3, 3), device="cuda", generator=g)
    return (A @ A.mT).contiguous()


def together(calls, repeats):
    """Runs every call `repeats` times in a thread of its own; the results of
    the last ones."""
    import torch
    out, errors, start = [None] * len(calls), [], threading.Barrier(len(calls))

    def run(k):
        start.wait()
        try:
            for _ in range(repeats):
                out[k] = calls[k]()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]
    return out


@pytest.mark.parametrize("what", ["structure2", "power", "separable", "pairs", "vote2"])
def test_windows_of_different_threads_do_not_meet(what):
    import torch
    import tiralib_gb300 as tv
    if what == "structure2":
        img = [torch.rand((64, 64), device="cuda") for _ in range(4)]
        calls = [lambda s=s, x=x: tv.structure_tensor2(x, s) for s, x in zip((0.7, 6.5, 0.7, 6.5), img)]
        repeats = 1500
    elif what == "vote2":
        f = [spd((32, 32), k)[..., :2, :2].reshape(32, 32, 4).contiguous() for k in range(4)]

        def vote2(x, w):
            out = torch.empty_like(x)
            tv.tensorvote(out, x, 2.0, 0.0, 1, w, 32, 32, True, True, 20)
            return out
        calls = [lambda w=w, x=x: vote2(x, w) for w, x in zip((5, 61, 5, 61), f)]
        repeats = 400
    else:
        shape, windows, kw, repeats = {"power": ((6, 6, 6), (3, 43), dict(power=2), 400),
                                       "separable": ((48, 64, 64), (21, 37), dict(), 60),
                                       "pairs": ((6, 6, 6), (3, 43), dict(), 400)}[what]
        T = [spd(shape, k) for k in range(4)]
        calls = [lambda w=w, x=x: tv.vote3(x, w / 6, w=w, **kw)[0] for w, x in zip(windows * 2, T)]
    want = [c().cpu().numpy() for c in calls]
    for got, ref in zip(together(calls, repeats), want):
        np.testing.assert_array_equal(got.cpu().numpy(), ref)
