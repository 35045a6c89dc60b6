"""Levels walked in chunks (window.cu) against the oracle, bit for bit, around the sizes where the
chunks start (8,192 rows) and change shape, on matrices whose chunks merge within their run-up, ones
whose rows need the sweeps (few or only far columns), and ones that end in the one-CTA walk."""
import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mean,band,p_near", [
    (8191, 8.0, 64, 0.9), (8192, 8.0, 64, 0.9), (8193, 8.0, 64, 0.9), (40_000, 8.0, 1, 1.0), (100_003, 2.0, 64, 0.9),
    (350_001, 8.0, 64, 0.9), (700_000, 5.0, 64, 0.5), (60_000, 8.0, 512, 0.9), (90_001, 30.0, 64, 0.9), (50_000, 8.0, 64, 0.0),
    (70_000, 0.2, 64, 0.9), (30_000, 16.0, 4000, 1.0)])
def test_levels_match_oracle(orc, n, mean, band, p_near):
    m = gen.random_upper(n, mean, p_near, band, n % 89 + 1)
    with sp.Solver(0) as s:
        s.analyse(m.row_ptr, m.col, m.val)
        lv, ml = orc.levels(m.row_ptr.astype(np.uint64), m.col)
        assert s.info()["max_level"] == ml
        assert np.array_equal(s.levels(), lv)
        ptr, rows = s.level_buckets()
        ptr_o, rows_o = orc.level_buckets(lv, ml)
        assert np.array_equal(ptr, ptr_o) and np.array_equal(rows, rows_o)
