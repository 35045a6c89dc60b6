"""Level buckets against the oracle, bit for bit, on both sides of the width where ranks within the levels
give way to the radix sort, with levels around the rank kernel's four lanes and the warp."""
import numpy as np
import pytest

import sptrsv_gb300 as sp

pytestmark = pytest.mark.gpu


def _strided(n, widths):
    """Row i depends on the first row of the level above (levels of the given widths from the end, the
    last width repeated)."""
    level_of, first, end, k = np.empty(n, np.int64), [], n, 0
    while end > 0:
        w = min(end, widths[min(k, len(widths) - 1)])
        level_of[end - w:end] = k
        first.append(end - w)
        end -= w
        k += 1
    i = np.arange(n)
    dep = level_of > 0
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(1 + dep)
    col, val = np.empty(rp[-1], np.int32), np.full(rp[-1], 0.5)
    col[rp[:-1]], val[rp[:-1]] = i, 2.0
    col[rp[:-1][dep] + 1] = np.array(first)[level_of[dep] - 1]
    return rp, col, val


@pytest.mark.parametrize("n,widths", [
    (1, [1]), (2, [2]), (31, [1]), (33, [3]), (1000, [4]), (1001, [5]), (5120, [256]), (5140, [257]), (5121, [256]),
    (9000, [31]), (9001, [33]), (20_000, [20_000]), (20_000, [2200, 1]), (20_000, [2300, 1]), (150_000, [1, 7, 64, 2])])
def test_buckets_match_oracle(orc, n, widths):
    rp, col, val = _strided(n, widths)
    with sp.Solver(0) as s:
        s.analyse(rp, col, val)
        lv, ml = orc.levels(rp.astype(np.uint64), col)
        assert np.array_equal(s.levels(), lv)
        ptr, rows = s.level_buckets()
        ptr_o, rows_o = orc.level_buckets(lv, ml)
        assert np.array_equal(ptr, ptr_o) and np.array_equal(rows, rows_o)
