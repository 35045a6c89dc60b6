"""The panels' diagonal-block inverses (supernodal.cu: 32-row blocks, eight columns a CTA) at the widths
where blocks, columns and chunks end, against the oracle's serial solve: elementwise error <= 1e-10,
relative residual <= 1e-12, as the other FP64 paths."""
import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wmin,wmax", [(1, 1), (7, 9), (31, 33), (64, 64), (63, 65), (255, 257), (300, 520), (1, 256)])
def test_widths(orc, wmin, wmax):
    m = gen.supernodal_random(4000, wmin, wmax, 40.0, 0.8, 400, wmax)
    rhs = 3
    b = gen.uniform(wmin, m.n * rhs)
    rpu = m.row_ptr.astype(np.uint64)
    ref = orc.base_gauss_upper(rpu, m.col, m.val, b, rhs)
    with sp.Solver(0) as s:
        s.analyse(m.row_ptr, m.col, m.val)
        s.set_supernodes(m.snodes)
        x = s.solve(b, rhs=rhs, schedule="supernodal")
    assert np.max(np.abs(x - ref) / np.maximum(np.abs(ref), 1e-6 * np.abs(ref).max())) <= 1e-10
    assert orc.rel_residual(rpu, m.col, m.val, x, b, rhs) <= 1e-12


@pytest.mark.parametrize("row", [0, 17, 40, 99])
def test_one_row_out_of_its_supernode_is_rejected(row):
    """A partition of 50-row supernodes over a matrix whose row `row` has an extra column."""
    m = gen.supernodal_random(200, 50, 50, 10.0, 1.0, 30, 4)
    rp, col, val = m.row_ptr.copy(), m.col, m.val
    used = set(col[rp[row]:rp[row + 1]])
    new = next(c for c in range(199, row, -1) if c not in used)
    at = int(rp[row] + np.searchsorted(col[rp[row]:rp[row + 1]], new))
    col, val = np.insert(col, at, new), np.insert(val, at, 0.5)
    rp[row + 1:] += 1
    with sp.Solver(0) as s:
        s.analyse(rp, col, val)
        with pytest.raises(sp.SptrsvError) as e:
            s.set_supernodes(m.snodes)
        assert e.value.status == -14
