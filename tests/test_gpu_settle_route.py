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


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("rhs", [1, 3])
def test_without_cooperative_launches(monkeypatch, graphs, rhs):
    """Cooperative launches refused: FP64 AUTO and the mixed solve answer all the same, on a handle and on host arrays."""
    m = gen.random_upper(20_000, 8.0, 0.9, 64, 5)
    b = gen.uniform(6, m.n * rhs)
    with sp.Solver(0) as s:
        y = s.analyse(m.row_ptr, m.col, m.val).solve(b, rhs=rhs, schedule="syncfree_window" if rhs == 1 else "syncfree_warp")
    monkeypatch.setenv("SPTRSV_NO_COOPERATIVE", "1")
    if not graphs:
        monkeypatch.setenv("SPTRSV_NO_GRAPH", "1")
    with sp.Solver(0) as s:
        s.analyse(m.row_ptr, m.col, m.val)
        for _ in range(2):
            x = s.solve(b, rhs=rhs)  # (the window kernel's last bits follow its timing, the warp kernel's do not)
            assert np.max(np.abs(x - y)) <= (1e-12 * np.max(np.abs(y)) if rhs == 1 else 0.0)
        x = s.solve(b, rhs=rhs, precision="mixed")
        assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(y))
    z = np.zeros_like(b)
    assert sp.base_gauss_upper(m.n, m.val, m.row_ptr.astype(np.uint64), m.col, z, b, rhs) >= 0
    assert np.max(np.abs(z - y)) <= 1e-9 * np.max(np.abs(y))


@pytest.mark.parametrize("n,rhs,layout", [
    (20_000, 2, sp.ROW_MAJOR), (20_001, 3, sp.COL_MAJOR), (60_002, 4, sp.ROW_MAJOR), (200_003, 8, sp.COL_MAJOR),
    (20_005, 17, sp.ROW_MAJOR), (20_006, 33, sp.COL_MAJOR)])
def test_several_right_hand_sides_repeat(n, rhs, layout):
    """With several right-hand sides FP64 AUTO repeats bit for bit, on one handle and on another."""
    m = gen.random_upper(n, 8.0, 0.9, 64, 5)
    b = gen.uniform(6, n * rhs)
    first = None
    for _ in range(2):
        with sp.Solver(0) as s:
            s.analyse(m.row_ptr, m.col, m.val)
            for _ in range(4):
                x = s.solve(b, rhs=rhs, layout=layout)
                first = x if first is None else first
                assert np.array_equal(x, first)


def test_one_right_hand_side_repeats_to_rounding(solver):
    """With one, solves differ by roundings (2^-53 of a term, a few terms to a row): the window kernel's do too."""
    m = gen.random_upper(200_000, 8.0, 0.9, 64, 5)
    solver.analyse(m.row_ptr, m.col, m.val)
    b = gen.uniform(6, m.n)
    for schedule in ("auto", "syncfree_window"):
        x = [solver.solve(b, schedule=schedule) for _ in range(4)]
        for y in x[1:]:
            assert np.max(np.abs(y - x[0])) <= 16 * 2.0**-53 * np.max(np.abs(x[0]))
