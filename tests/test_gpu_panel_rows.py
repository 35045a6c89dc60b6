"""FP64 panel products by warps of four rows (panel_rows.cu) where their items end: right-hand sides that
leave a group of two half full, chunks whose rows are not a multiple of four, rectangles shorter and
longer than a step of 32 columns, trees and bands; batches whose chunks are 64, 128 and 256 rows, and the
panel modes switched between a batch's creation and its lists.

Tolerances: elementwise 1e-10 against max(|x_i|, 1e-6 of the largest) and residual 1e-12 against the
oracle, as the other FP64 paths; the batch's chosen mode at its tolerance of 1e-12."""
import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu


def _close(x, ref):
    return np.max(np.abs(x - ref) / np.maximum(np.abs(ref), 1e-6 * np.abs(ref).max()))


@pytest.mark.parametrize("rhs", [1, 2, 3, 7, 33])
@pytest.mark.parametrize("kind", ["band5", "band33", "tree", "wide"])
def test_solves(orc, kind, rhs):
    if kind == "tree":
        m = gen.laplace3d_nd_cholesky_gpu(9, leaf=3)
    elif kind == "wide":
        m = gen.supernodal_random(3000, 1, 70, 50.0, 0.5, 900, 3)
    else:
        m = gen.laplace2d_cholesky(int(kind[4:]))
        m.snodes = np.append(np.arange(0, m.n, 23 if kind == "band5" else 250), m.n).astype(np.int32)
    b = gen.uniform(rhs, m.n * rhs)
    rpu = m.row_ptr.astype(np.uint64)
    ref = orc.base_gauss_upper(rpu, m.col, m.val, b, rhs)
    with sp.Solver(0) as s:
        s.analyse(m.row_ptr, m.col, m.val)
        s.set_supernodes(m.snodes)
        x = s.solve(b, rhs=rhs, schedule="supernodal")
    assert _close(x, ref) <= 1e-10
    assert orc.rel_residual(rpu, m.col, m.val, x, b, rhs) <= 1e-12


@pytest.mark.parametrize("before,after", [("fp64", "tc"), ("fp64", "df"), ("df", "fp64"), ("tc", "fp64")])
def test_batch_keeps_its_panels_when_the_mode_changes(orc, before, after):
    """Panels built in one mode, lists built in another: 70 x 70 and 24 x 24 bands, 5 and 1 columns."""
    ms = [gen.laplace2d_cholesky(70), gen.laplace2d_cholesky(24), gen.random_upper(5000, 8.0, 0.9, 64, 1)]
    rhs = [5, 1, 2]
    prev = sp.set_panels_mode(before)
    try:
        B = sp.Batch([m.n for m in ms], rhs, np.concatenate([m.row_ptr for m in ms]), np.concatenate([m.col for m in ms]),
                     np.concatenate([m.val for m in ms]))
        B.schedule = ["panel64", "panel64", "jacobi"]
        b = gen.uniform(3, int(B.xb_off[-1]))
        first = B.solve(b)
        sp.set_panels_mode(after)
        B.schedule = ["panel64", "panel64", "jacobi"]
        second = B.solve(b)
    finally:
        sp.set_panels_mode(prev)
    for x in (first, second):
        for m, r, xs, bs in zip(ms, rhs, B.split(x), B.split(b)):
            ref = orc.base_gauss_upper(m.row_ptr.astype(np.uint64), m.col, m.val, bs.T.copy().reshape(-1), r)
            assert _close(xs.T.reshape(-1), ref) <= 1e-8
    B.close()


@pytest.mark.parametrize("rhs", [1, 2])
@pytest.mark.parametrize("band", [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 160, 255])
@pytest.mark.parametrize("chunk", [4, 37, 129, 250])
def test_bands_around_the_groups_of_steps(orc, chunk, band, rhs):
    """Own and solved columns around one to eight steps of 32, read two and four at a time."""
    n = 700
    k = np.minimum(band, n - 1 - np.arange(n))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(1 + k)
    off = np.arange(rp[-1]) - np.repeat(rp[:-1], 1 + k)
    col = (np.repeat(np.arange(n), 1 + k) + off).astype(np.int32)
    val = np.where(off == 0, 2.0, np.random.default_rng(band).uniform(-1.0, 1.0, len(off)) / band)
    b = gen.uniform(rhs, n * rhs)
    rpu = rp.astype(np.uint64)
    ref = orc.base_gauss_upper(rpu, col, val, b, rhs)
    with sp.Solver(0) as s:
        s.analyse(rp, col, val)
        s.set_supernodes(np.append(np.arange(0, n, chunk), n).astype(np.int32))
        x = s.solve(b, rhs=rhs, schedule="supernodal")
    assert _close(x, ref) <= 1e-10
    assert orc.rel_residual(rpu, col, val, x, b, rhs) <= 1e-12
