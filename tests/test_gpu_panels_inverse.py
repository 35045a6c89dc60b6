"""The error of the panels' inverted triangles on ill-conditioned ones, in norm against extended precision: one
supernode solved for the identity's columns gives T^-1 entry by entry.  Substitution, column by column with a
row's products in 32 partial sums, is what it is compared with; the ratio of two such errors scatters by
a few percent from matrix to matrix, so their means over four matrices may differ by 15 %."""
import numpy as np
import pytest

import sptrsv_gb300 as sp

pytestmark = pytest.mark.gpu

X = np.longdouble


def _triangle(w, cond, seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((w, w)))
    a = (q * np.logspace(0, -np.log10(cond), w)) @ q.T
    return np.linalg.cholesky((a + a.T) / 2).T.copy()


def _extended(t):
    w, tx = len(t), t.astype(X)
    x = np.zeros((w, w), X)
    for r in range(w - 1, -1, -1):
        v = -(tx[r, r + 1:] @ x[r + 1:])
        v[r] += 1
        x[r] = v / tx[r, r]
    return x


def _substitution(t):
    w = len(t)
    x = np.zeros((w, w))
    for r in range(w - 1, -1, -1):
        s = np.zeros((32, w))
        for k in range(r + 1, w, 32):
            h = min(32, w - k)
            s[:h] = (t[r, k:k + h].astype(X)[:, None] * x[k:k + h].astype(X) + s[:h].astype(X)).astype(np.float64)
        while len(s) > 1:
            s = s[:len(s) // 2] + s[len(s) // 2:]
        x[r] = -s[0] / t[r, r]
        x[r, :r] = 0.0
        x[r, r] = 1.0 / t[r, r]
    return x


@pytest.mark.parametrize("w,cond", [(256, 1e2), (256, 1e4), (256, 1e8), (128, 1e4), (33, 1e4)])
def test_error_beside_substitution(w, cond):
    rp = np.zeros(w + 1, np.int64)
    rp[1:] = np.cumsum(np.arange(w, 0, -1))
    col = np.concatenate([np.arange(i, w) for i in range(w)]).astype(np.int32)
    ours, theirs = [], []
    for seed in range(4):
        t = _triangle(w, cond, seed)
        ref = _extended(t)
        norm = np.sqrt(np.sum(ref ** 2))
        with sp.Solver(0) as s:
            s.analyse(rp, col, t[np.triu_indices(w)])
            s.set_supernodes(np.array([0, w], np.int32))
            x = s.solve(np.eye(w).reshape(-1), rhs=w, layout=sp.ROW_MAJOR, schedule="supernodal").reshape(w, w)
        ours.append(float(np.sqrt(np.sum((x - ref) ** 2)) / norm))
        theirs.append(float(np.sqrt(np.sum((_substitution(t) - ref) ** 2)) / norm))
    print(w, cond, np.mean(ours) / np.mean(theirs))
    assert np.mean(ours) <= 1.15 * np.mean(theirs)
