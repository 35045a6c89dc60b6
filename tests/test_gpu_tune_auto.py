"""Tuning never leaves AUTO slower than it was: rows that are not strictly dominant, where the refinement is ruled
out and AUTO's own kernels (the sweeps, the window kernel) are not in the tuner's table."""
import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu


def _kernels(s, b):
    s.profile(True)
    x = s.solve(b)
    kinds = [k for k, _ in s.profile_read()]
    s.profile(False)
    return x, kinds


@pytest.mark.parametrize("scale", [1.6, 8.0])  # sweeps that settle and sweeps that do not
def test_auto_stays_with_its_own_kernel(scale):
    m = gen.random_upper(60_000, 2.0 if scale > 2 else 8.0, 0.9, 64, 5)
    val = m.val * scale
    val[m.row_ptr[:-1]] = m.val[m.row_ptr[:-1]]
    b = gen.uniform(7, m.n)
    with sp.Solver(0) as s:
        s.analyse(m.row_ptr, m.col, val)
        s.solve(b)
        x, before = _kernels(s, b)
        best, ms = s.autotune(rhs=1, reps=1)
        assert ms[best] == np.min(ms)
        y, after = _kernels(s, b)
    assert after == before
    if scale < 2:  # (the other's solution grows past the largest double)
        assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(x))
