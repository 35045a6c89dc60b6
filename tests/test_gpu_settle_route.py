"""What FP64 AUTO's sweeps (settle.cu) take on and leave to the exact kernels: calls that the exact kernels
answer are answered, and as well."""
import ctypes

import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import _lib, gen

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


def _chain(n, w):
    """x_i = b_i - w x_i+1."""
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.where(np.arange(n) < n - 1, 2, 1))
    col, val = np.empty(rp[-1], np.int32), np.empty(rp[-1])
    col[rp[:-1]], val[rp[:-1]] = np.arange(n), 1.0
    col[rp[:-2] + 1], val[rp[:-2] + 1] = np.arange(1, n), w
    return rp, col, val


def _kernels(s, n, rhs):
    s.profile(True)
    x = s.solve(gen.uniform(1, n * rhs), rhs=rhs)
    kinds = [k for k, _ in s.profile_read()]
    s.profile(False)
    return x, kinds


SETTLE = 16


@pytest.mark.parametrize("rhs", [1, 3])
@pytest.mark.parametrize("w,tries", [(0.9, 1), (1.0, 1), (1.001, 1), (0.5, 9)])
def test_sweeps_that_do_not_settle_are_tried_once(w, tries, rhs):
    """30,000 rows deep, so that an attempt is cheap beside the exact kernel: one attempt, and the exact
    kernel's result from the first solve on (several right-hand sides: its bits)."""
    n = 30_000
    with sp.Solver(0) as s:
        s.analyse(*_chain(n, w))
        runs = [_kernels(s, n, rhs) for _ in range(3)]
        assert [SETTLE in k for _, k in runs] == [q < tries for q in range(3)]
        if rhs > 1:
            assert all(np.array_equal(x, runs[0][0]) for x, _ in runs)
        s.analyse(*_chain(n, 0.3))  # another matrix on the handle
        assert SETTLE in _kernels(s, n, rhs)[1]


@pytest.mark.parametrize("w,swept", [(0.5, True), (1.0, False)])
def test_rows_that_are_not_dominant(w, swept):
    """3,000 rows deep, where an attempt in vain would be a good part of the exact kernel's time."""
    with sp.Solver(0) as s:
        s.analyse(*_chain(3_000, w))
        assert (SETTLE in _kernels(s, 3_000, 1)[1]) == swept


@pytest.mark.parametrize("rhs", [1, 3])
@pytest.mark.parametrize("entries,swept", [(30, True), (3_000, False), (19_000, False)])
def test_one_long_row(orc, entries, swept, rhs):
    """A row that one lane would walk through global memory in every sweep goes to the exact kernel."""
    n, at = 40_000, 20_000
    m = gen.random_upper(n, 7.0, 0.9, 64, 5)
    rng = np.random.default_rng(3)
    c = np.concatenate([[at], np.sort(rng.choice(np.arange(at + 1, n), entries, replace=False))]).astype(np.int32)
    v = np.concatenate([[entries + 1.0], rng.uniform(-1, 1, entries)])
    a, e = m.row_ptr[at], m.row_ptr[at + 1]
    rp = m.row_ptr.copy()
    rp[at + 1:] += len(c) - (e - a)
    col, val = np.concatenate([m.col[:a], c, m.col[e:]]), np.concatenate([m.val[:a], v, m.val[e:]])
    with sp.Solver(0) as s:
        s.analyse(rp, col, val)
        x, kinds = _kernels(s, n, rhs)
    assert (SETTLE in kinds) == swept
    ref = orc.base_gauss_upper(rp.astype(np.uint64), col, val, gen.uniform(1, n * rhs), rhs)
    assert np.max(np.abs(x - ref)) <= 1e-10 * np.max(np.abs(ref))


def test_tuned_options_that_name_the_sweeps_are_refused(solver):
    m = gen.random_upper(100, 4.0, 0.9, 8, 2)
    solver.analyse(m.row_ptr, m.col, m.val)
    assert _lib.lib().sptrsv_set_tuned(solver.handle, 1, ctypes.byref(sp.make_opts(schedule=100))) == 0
    with pytest.raises(sp.SptrsvError) as e:
        solver.solve(np.ones(m.n))
    assert e.value.status == -15
    x = solver.solve(np.ones(m.n * 2), rhs=2)  # another class of right-hand sides
    assert np.isfinite(x).all()


def test_refused_sweeps_are_tried_again_with_the_next_matrix(monkeypatch):
    n = 30_000
    m = gen.random_upper(n, 8.0, 0.9, 64, 5)
    with sp.Solver(0) as s:
        monkeypatch.setenv("SPTRSV_NO_COOPERATIVE", "1")
        s.analyse(m.row_ptr, m.col, m.val)
        assert SETTLE not in _kernels(s, n, 1)[1]
        monkeypatch.delenv("SPTRSV_NO_COOPERATIVE")
        assert SETTLE not in _kernels(s, n, 1)[1]
        s.analyse(m.row_ptr, m.col, m.val)
        assert SETTLE in _kernels(s, n, 1)[1]


def test_attempts_are_spaced_out_and_come_back():
    """After a failure 8 solves without an attempt, after the next 16; right-hand sides that settle end that."""
    n = 30_000
    with sp.Solver(0) as s:
        s.analyse(*_chain(n, 0.9))
        assert [k for k in range(30) if SETTLE in _kernels(s, n, 1)[1]] == [0, 9, 26]
        # a band that contracts, and one entry at its end
        s.analyse(*_chain(n, 0.7))
        e = np.zeros(n)
        e[-1] = 1.0
        assert np.max(np.abs(s.solve(e) - (-0.7) ** np.arange(n - 1, -1, -1))) <= 1e-12
        assert SETTLE in [k for _ in range(9) for k in _kernels(s, n, 1)[1]]
        assert SETTLE in _kernels(s, n, 1)[1]
