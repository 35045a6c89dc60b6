"""FP64 AUTO's error where its sweeps contract slowly, in norm against a solution in extended precision.

The sweeps end when what is left is below 2^-54 of a row's largest term, half the rounding (2^-53) that
substitution makes in forming it: at most (2^-53 + 2^-54) / 2^-53 = 1.5 times substitution's own error."""
import numpy as np
import pytest

import sptrsv_gb300 as sp

pytestmark = pytest.mark.gpu

N = 19_968


def _rows(n, k, w):
    """k entries of value w beside a unit diagonal."""
    c = np.minimum(k, n - 1 - np.arange(n))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(1 + c)
    off = np.arange(rp[-1]) - np.repeat(rp[:-1], 1 + c)
    col = (np.repeat(np.arange(n), 1 + c) + off).astype(np.int32)
    return rp, col, np.where(off == 0, 1.0, w)


def _extended(k, w, b):
    x = np.zeros((len(b) + k, b.shape[1]), np.longdouble)
    v = np.full(k, w, np.longdouble)
    for i in range(len(b) - 1, -1, -1):
        x[i] = b[i] - v @ x[i + 1:i + 1 + k]
    return x[:len(b)]


@pytest.mark.parametrize("rhs", [1, 3])
@pytest.mark.parametrize("k,w,rhs_kind", [
    (1, -0.7, "positive"), (1, -0.7, "constant"), (2, -0.35, "positive"), (8, -0.075, "positive"), (1, -0.6, "positive"),
    (1, 0.6, "signed"), (1, -0.3, "positive"), (4, -0.15, "positive"), (1, -0.9, "positive")])
def test_slow_contraction(orc, k, w, rhs_kind, rhs):
    rp, col, val = _rows(N, k, w)
    b = np.random.default_rng(k).uniform(-1.0 if rhs_kind == "signed" else 0.0, 1.0, (N, rhs))
    if rhs_kind == "constant":
        b[:] = 1.0
    ref = _extended(k, w, b)
    own = orc.base_gauss_upper(rp.astype(np.uint64), col, val, b.T.copy().reshape(-1), rhs).reshape(rhs, N).T
    with sp.Solver(0) as s:
        x = s.analyse(rp, col, val).solve(b.reshape(-1), rhs=rhs, layout=sp.ROW_MAJOR).reshape(N, rhs)
    err = lambda y: float(np.sqrt(np.sum((y - ref) ** 2) / np.sum(ref ** 2)))
    assert err(x) <= 1.5 * err(own), (err(x), err(own))
