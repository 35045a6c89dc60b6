"""The mixed solve's inner solves as one launch each (tiles of 256 rows copied ahead) against the same
sweeps launched one by one over another layout: every row's sum is made in the same order, so the solutions
are equal bit for bit.  Sizes at the edges of a tile, of the tiles that stay in shared memory (two a block)
and of the grid, and matrices with tiles that no stage holds, with empty rows and with none but the
diagonal."""
import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu


def _clustered(n, at, length):
    """Mostly empty rows, with 300 rows of `length` entries from row `at` on."""
    k = np.zeros(n, np.int64)
    k[at:at + 300] = np.minimum(length, n - 1 - np.arange(at, at + 300))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(1 + k)
    off = np.arange(rp[-1]) - np.repeat(rp[:-1], 1 + k)
    col = (np.repeat(np.arange(n), 1 + k) + off).astype(np.int32)
    val = np.where(off == 0, 1.0 + 0.3 * np.repeat(k, 1 + k), np.where(off % 3 == 1, -0.25, 0.2))
    return rp, col, val


def _random(n, mean, p_near, band):
    m = gen.random_upper(n, mean, p_near, band, n % 97 + 2)
    return m.row_ptr, m.col, m.val


MATRICES = (
    [("random", (n, 8.0, 0.9, 64)) for n in (1, 2, 255, 256, 257, 511, 513, 5000, 155_648, 155_649, 311_296, 311_297,
                                             400_003, 700_001)]
    + [("random", (30_000, 12.9, 0.5, 300)), ("random", (30_000, 0.3, 0.9, 64)), ("random", (1_200_000, 5.0, 0.9, 64))]
    + [("clustered", (20_000, 0, 400)), ("clustered", (20_000, 19_600, 400)), ("clustered", (300_000, 1000, 100))])


def _equal(orc, monkeypatch, rp, col, val, rhs, layout):
    n = len(rp) - 1
    b = gen.uniform(n + 3, n * rhs)
    out = {}
    for kernel in ("", "batch8"):
        monkeypatch.setenv("SPTRSV_SWEEP_KERNEL", kernel)
        with sp.Solver(0) as s:
            s.analyse(rp, col, val)
            x = [s.solve(b, rhs=rhs, precision="mixed", schedule="jacobi", max_refine=20, layout=layout) for _ in range(2)]
            assert np.array_equal(x[0], x[1])
            assert s.last_refine()[1] <= 1e-13
            out[kernel] = x[0], s.last_sweeps()
    assert out[""][1] == out["batch8"][1]
    assert np.array_equal(out[""][0], out["batch8"][0])
    if layout == sp.COL_MAJOR:
        assert orc.rel_residual(rp.astype(np.uint64), col, val, out[""][0], b, rhs) <= 2e-13


@pytest.mark.parametrize("kind,args", MATRICES, ids=lambda v: v if isinstance(v, str) else "-".join(map(str, v)))
def test_loop_equals_single_sweeps(orc, monkeypatch, kind, args):
    _equal(orc, monkeypatch, *(_random(*args) if kind == "random" else _clustered(*args)), 1, sp.COL_MAJOR)


@pytest.mark.parametrize("rhs", [2, 3, 4, 5, 8, 12, 13])
@pytest.mark.parametrize("n", [1, 257, 20_001, 320_000])
def test_several_right_hand_sides(orc, monkeypatch, n, rhs):
    """Four columns a lane, up to the count where the kernels with lanes along the columns take over."""
    _equal(orc, monkeypatch, *_random(n, 8.0, 0.9, 64), rhs, sp.ROW_MAJOR if rhs % 2 else sp.COL_MAJOR)


def test_several_right_hand_sides_over_large_tiles(orc, monkeypatch):
    _equal(orc, monkeypatch, *_clustered(20_000, 700, 400), 6, sp.COL_MAJOR)
