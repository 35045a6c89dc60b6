"""FP64 AUTO's sweeps (settle.cu) against the oracle's serial solve and against the exact kernels, over
what the dispatch accepts: tiles that end mid-way, one to many right-hand sides in both layouts,
unsorted rows, rows without off-diagonals, rows longer than the staging buffers, values of very
different size, and matrices whose sweeps do not contract (the exact kernel behind them answers).

Tolerances: relative residual 1e-12, as the other FP64 paths (or ten times the serial solve's own,
where x is so much larger than b that substitution itself does not reach 1e-12); the term-relative error within 1e-13
(rounding in any order is ~1e-14 there), 1e-11 on chains of 30,000 rows that do not contract (n u);
elementwise 1e-9 against max(|x_i|, 1e-6 of the column's largest): u times that ratio, with room for
ten rounding errors.
"""
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


def _check(orc, solver, rp, col, val, b, rhs=1, layout=sp.COL_MAJOR, term=1e-13):
    solver.analyse(rp, col, val)
    n = len(rp) - 1
    rpu = np.asarray(rp, dtype=np.uint64)
    ref = orc.base_gauss_upper(rpu, col, val, b, rhs)
    bb = b if layout == sp.COL_MAJOR else b.reshape(rhs, n).T.copy().reshape(-1)
    x = solver.solve(bb, rhs=rhs, layout=layout)
    if layout != sp.COL_MAJOR:
        x = x.reshape(n, rhs).T.copy().reshape(-1)
    d, a = np.abs(x - ref).reshape(rhs, n), np.abs(ref).reshape(rhs, n)
    assert (d / np.maximum(a, 1e-6 * a.max(axis=1, keepdims=True))).max() <= max(1e-9, term)
    own = orc.rel_residual(rpu, col, val, ref, b, rhs)
    assert orc.rel_residual(rpu, col, val, x, b, rhs) <= max(1e-12, 10 * own)
    assert orc.term_rel_error(rpu, col, val, ref, x, b, rhs) <= term
    return x


@pytest.mark.parametrize("n,rhs,layout", [
    (20_000, 1, sp.COL_MAJOR), (20_011, 1, sp.COL_MAJOR), (31_999, 1, sp.ROW_MAJOR), (200_003, 1, sp.COL_MAJOR),
    (20_001, 2, sp.ROW_MAJOR), (20_002, 3, sp.COL_MAJOR), (20_003, 5, sp.ROW_MAJOR), (20_007, 8, sp.COL_MAJOR),
    (20_005, 9, sp.ROW_MAJOR), (20_006, 17, sp.COL_MAJOR), (20_009, 33, sp.ROW_MAJOR)])
def test_sizes_and_layouts(orc, solver, n, rhs, layout):
    m = gen.random_upper(n, 8.0, 0.9, 64, n % 97 + rhs)
    _check(orc, solver, m.row_ptr, m.col, m.val, gen.uniform(n, n * rhs), rhs, layout)


@pytest.mark.parametrize("mean,band,p_near", [(0.5, 64, 0.9), (16.0, 64, 0.9), (8.0, 4000, 0.5), (3.0, 2, 1.0)])
def test_shapes_match_exact_kernel(orc, solver, mean, band, p_near):
    m = gen.random_upper(60_001, mean, p_near, band, int(mean * 4))
    b = gen.uniform(band, m.n)
    x = _check(orc, solver, m.row_ptr, m.col, m.val, b)
    y = solver.solve(b, schedule="syncfree_window")
    assert np.max(np.abs(x - y) / np.maximum(np.abs(y), 1e-6 * np.abs(y).max())) <= 1e-9


@pytest.mark.parametrize("rhs", [1, 4])
def test_unsorted_rows_long_rows_and_scales(orc, solver, rhs):
    """Shuffled rows, a few rows of 3,000 entries, row scales over 200 binades, columns of b over 60."""
    n = 40_000
    m = gen.random_upper(n, 7.0, 0.9, 64, 5)
    rng = np.random.default_rng(3)
    rp0, rows, cols, vals = m.row_ptr, [], [], []
    for i in range(n):
        c, v = m.col[rp0[i]:rp0[i + 1]].copy(), m.val[rp0[i]:rp0[i + 1]].copy()
        if i in (100, 101, 20_000):
            c = np.concatenate([[i], rng.choice(np.arange(i + 1, n), 3000, replace=False)]).astype(np.int32)
            v = np.concatenate([[4000.0], rng.uniform(-1, 1, 3000)])
        q = 1 + rng.permutation(len(c) - 1)
        s = 2.0 ** rng.integers(-100, 100)
        rows.append(len(c))
        cols.append(np.concatenate([c[:1], c[q]]))
        vals.append(np.concatenate([v[:1], v[q]]) * s)
    rp = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    col, val = np.concatenate(cols).astype(np.int32), np.concatenate(vals)
    scale = np.array([val[rp[i]] for i in range(n)])
    b = (gen.uniform(9, n * rhs).reshape(rhs, n) * scale * (2.0 ** np.arange(0, 60, 60 // rhs)[:rhs, None])).reshape(-1)
    _check(orc, solver, rp, col, val, b, rhs)


@pytest.mark.parametrize("rhs", [1, 3])
@pytest.mark.parametrize("kind", ["chain", "growing"])
def test_not_contracting(orc, solver, kind, rhs):
    """A bidiagonal chain x_i = b_i + w x_{i+1}: |w| = 1 (no contraction), and |w| = 1.001."""
    n = 30_000
    w = 1.0 if kind == "chain" else 1.001
    rp = np.zeros(n + 1, dtype=np.int64)
    rp[1:] = np.cumsum(np.where(np.arange(n) < n - 1, 2, 1))
    col, val = np.empty(rp[-1], dtype=np.int32), np.empty(rp[-1])
    col[rp[:-1]], val[rp[:-1]] = np.arange(n), 1.0
    col[rp[:-2] + 1], val[rp[:-2] + 1] = np.arange(1, n), w
    _check(orc, solver, rp, col, val, gen.uniform(1, n * rhs), rhs, term=1e-11)


def test_special_values(solver):
    """Zero right-hand side; an infinity and a NaN in b end where substitution puts them."""
    m = gen.random_upper(30_000, 8.0, 0.9, 64, 2)
    solver.analyse(m.row_ptr, m.col, m.val)
    assert not solver.solve(np.zeros(m.n)).any()
    for v in (np.inf, np.nan):
        b = gen.uniform(4, m.n)
        b[15_000] = v
        x, y = solver.solve(b), solver.solve(b, schedule="syncfree_window")
        assert np.array_equal(np.isfinite(x), np.isfinite(y))
        ok = np.isfinite(y)
        assert np.array_equal(x[~ok], y[~ok], equal_nan=True)
        assert np.max(np.abs(x[ok] - y[ok])) <= 1e-12


def test_named_schedule_of_the_sweeps_is_refused(solver):
    m = gen.random_upper(100, 4.0, 0.9, 8, 2)
    solver.analyse(m.row_ptr, m.col, m.val)
    with pytest.raises(sp.SptrsvError) as e:
        solver.solve(np.ones(m.n), schedule=100)
    assert e.value.status == -15
