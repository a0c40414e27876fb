"""The separable 3D vote's tables (tiralib_gb300/csrc/vote3_sep_tables.inc):
|o|^-2k as sums of exponentials, to 1.5e-7 of each value."""
import os
import re

import numpy as np
import pytest

INC = os.path.join(os.path.dirname(__file__), "..", "tiralib_gb300", "csrc", "vote3_sep_tables.inc")
NUM = r"\{([^{}]*)\}"


def rows():
    for m in re.finditer(r"\{(\d+),\s*(\d+),\s*" + r",\s*".join([NUM] * 4), open(INC).read()):
        yield int(m[1]), int(m[2]), [np.array([float(v) for v in m[i].split(",") if v.strip()]) for i in (3, 4, 5, 6)]


def test_rows_reach_the_widest_window_in_order():
    ext = [(smax, T) for smax, T, _ in rows()]
    assert ext == sorted(ext) and ext[-1][0] >= 3 * 20 ** 2


@pytest.mark.parametrize("row", list(rows()), ids=lambda r: str(r[0]))
def test_relative_error_everywhere(row):
    smax, T, (b, *w) = row
    assert all(len(v) == T for v in (b, *w)) and b[0] == 0.0 and (np.diff(b) > 0).all()
    s = np.arange(1, smax + 1, dtype=float)
    E = np.exp(-np.outer(s, b))
    for k in range(3):
        assert np.abs(E @ w[k] * s ** (k + 1) - 1).max() < 1.5e-7
