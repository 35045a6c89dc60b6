"""What FP64 AUTO's sweeps (settle.cu) take on and leave to the exact kernels: calls that the exact kernels
answer are answered, and as well."""
import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver():
    s = sp.Solver(0)
    yield s
    s.close()


def test_small_spin_budget(solver):
    """A budget for waits on rows, shorter than a sweep: 2M rows, where the exact kernel has no such wait either."""
    m = gen.random_upper(2_000_000, 8.0, 0.9, 64, 5)
    solver.analyse(m.row_ptr, m.col, m.val)
    b = gen.uniform(6, m.n)
    y = solver.solve(b)
    x = solver.solve(b, spin_budget_ns=20_000)
    assert np.max(np.abs(x - y)) <= 1e-12 * np.max(np.abs(y))
