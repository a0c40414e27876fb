"""Calls that need less scratch than they like: with the device nearly full
the sweep votes fewer sets at a time.  In a process of its own, whose memory is its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import sys
sys.path[:0] = [{here!r}, {repo!r}]
import numpy as np
import torch
import tiralib_gb300 as tv
from tiralib_gb300 import optimize
from test_gpu_vote3_sep import kernels_of

def leave(free):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert tv.lib().tvgb_release_cached_memory() == 0
    return torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")

{body}
print("passed")
"""

SWEEP = """
n = 2048
I = torch.rand((n, n, 2, 2), device="cuda")
I = (I @ I.mT).contiguous()
G = I.flip(0).contiguous()
params = [(0.5 + 0.01 * k, 0.0, 1 + k % 2) for k in range(20)]       # 64 MB a field: 16 sets at a time
want = np.asarray(optimize.tk_sweep(G, I, params))
hog = leave(400 << 20)
np.testing.assert_allclose(np.asarray(optimize.tk_sweep(G, I, params)), want, rtol=1e-10)
"""

@pytest.mark.parametrize("body", [SWEEP], ids=["sweep"])
def test_a_nearly_full_device(body):
    code = CHILD.format(here=HERE, repo=os.path.dirname(HERE), body=body)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("passed\n"), r.stdout[-2000:] + r.stderr[-4000:]
