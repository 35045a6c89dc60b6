"""The solver's measured work: what a program that links this framework has it do.

A case is one call (or the one fixed sequence of calls) of a user's inner loop, through the public
entry points of ``sptrsv_gb300``: solves on a kept ``Solver`` handle, the analysis of a new matrix,
the multifrontal factorisation, a batch of uneven systems, and the reference's own host-array
interface.  The matrices are the ones the repository is tested and benchmarked on: random
diagonally dominant rows (``gen.random_upper``'s recipe, built here with torch on the GPU), band
Cholesky factors of the 2D Laplacian, nested-dissection Cholesky factors of the 3D Laplacian, and
the uneven mix of the first two.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import sptrsv_gb300 as sp
from sptrsv_gb300 import _lib, gen

#: Near dependencies of the random rows lie within this many columns of the diagonal, the share of
#: them that does, and the entries per row (the recipe of the large irregular system).
BAND, P_NEAR, MEAN = 64, 0.9, 8.0


def listed():
    return [
        # The smallest call: one right-hand side of a small system on a kept handle, as in an inner
        # loop of a preconditioner; launches and host latency are what it costs.
        {"name": "solve-1k", "kind": "solve", "matrix": "random", "n": 1000, "rhs": 1, "precision": "fp64", "row_major": False},
        # The plain FP64 case of the repository: the 64 x 64 grid's band factor.
        {"name": "solve-band-4k", "kind": "solve", "matrix": "band", "n": 64 * 64, "rhs": 1, "precision": "fp64", "row_major": False},
        # The large irregular system, exact FP64: a preconditioner's triangular solve.
        {"name": "solve-irregular-2m", "kind": "solve", "matrix": "random", "n": 2_000_000, "rhs": 1, "precision": "fp64", "row_major": False},
        # The same system through the FP32 + FP64 refinement, the benchmark's chosen form.
        {"name": "refine-irregular-2m", "kind": "solve", "matrix": "random", "n": 2_000_000, "rhs": 1, "precision": "mixed", "row_major": False},
        # A block of right-hand sides of a medium irregular system.
        {"name": "solve-block-200k", "kind": "solve", "matrix": "random", "n": 200_003, "rhs": 8, "precision": "fp64", "row_major": False},
        # A direct solver's solve phase on the 40^3 factor: one vector, and a block of them.
        {"name": "supernodal-40-1", "kind": "solve", "matrix": "nd", "n": 40**3, "rhs": 1, "precision": "fp64", "row_major": False},
        {"name": "supernodal-40-32", "kind": "solve", "matrix": "nd", "n": 40**3, "rhs": 32, "precision": "fp64", "row_major": False},
        # A direct solver's factor phase: A on the host, U left on the device.
        {"name": "factor-40", "kind": "factor", "n": 40**3},
        # The analysis of a new sparsity pattern: validation, levels, buckets, in-degrees.
        {"name": "analyse-500k", "kind": "analyse", "n": 499_999},
        # The reference's interface on host arrays: serial substitution's replacement, and the
        # supernodal one (a new matrix each call: upload, analysis, panels, solve).
        {"name": "dropin-gauss-100k", "kind": "dropin_gauss", "n": 99_991, "rhs": 1},
        {"name": "dropin-supernodal-20", "kind": "dropin_supernodal", "n": 20**3, "rhs": 4},
        # Many uneven systems at once, each by the schedule chosen for it.
        {"name": "batch-48", "kind": "batch", "mix": 2, "count": 48, "nmax": 30_000, "rhs_max": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "block", "refine", "band", "nd", "nd", "factor", "analyse",
                       "dropin_gauss", "dropin_supernodal", "batch"])
    rows = rng.random() < 0.3
    if kind == "solve":
        return {"kind": "solve", "matrix": "random", "n": _log_int(rng, 500, 2_000_000), "rhs": 1, "precision": "fp64",
                "row_major": False}
    if kind == "block":
        return {"kind": "solve", "matrix": "random", "n": _log_int(rng, 2_000, 200_000), "rhs": rng.randint(2, 8),
                "precision": "fp64", "row_major": rows}
    if kind == "refine":
        rhs = rng.choice([1, 1, rng.randint(2, 8)])
        return {"kind": "solve", "matrix": "random", "n": _log_int(rng, 2_000, 2_000_000 // rhs), "rhs": rhs,
                "precision": "mixed", "row_major": rows}
    if kind == "band":
        return {"kind": "solve", "matrix": "band", "n": rng.randint(24, 96) ** 2, "rhs": rng.choice([1, 1, 3]),
                "precision": "fp64", "row_major": rows}
    if kind == "nd":
        return {"kind": "solve", "matrix": "nd", "n": rng.randint(9, 40) ** 3, "rhs": _log_int(rng, 1, 32),
                "precision": "fp64", "row_major": rows}
    if kind == "factor":
        return {"kind": "factor", "n": rng.randint(9, 40) ** 3}
    if kind == "analyse":
        return {"kind": "analyse", "n": _log_int(rng, 1_000, 500_000)}
    if kind == "dropin_gauss":
        return {"kind": "dropin_gauss", "n": _log_int(rng, 1_000, 100_000), "rhs": rng.randint(1, 3)}
    if kind == "dropin_supernodal":
        return {"kind": "dropin_supernodal", "n": rng.randint(8, 20) ** 3, "rhs": rng.randint(1, 6)}
    return {"kind": "batch", "mix": rng.randint(1, 100_000), "count": rng.randint(4, 48),
            "nmax": _log_int(rng, 4_000, 30_000), "rhs_max": rng.randint(1, 16)}


# ------------------------------------------------------------------------------------------------
# Matrices, on the GPU

def _random_csr(n, seed):
    """gen.random_upper's distribution: Poisson(MEAN) off-diagonals a row, near ones within BAND of
    the diagonal, values U[-1, 1], diagonal 1 + sum |off|.  int32 row pointer, columns, values."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.poisson(torch.full((n,), MEAN, device="cuda"), generator=g).long()
    i = torch.repeat_interleave(torch.arange(n, device="cuda"), k)
    near = i + 1 + (torch.rand(len(i), generator=g, device="cuda", dtype=torch.float64) * BAND).long()
    far = i + 1 + (torch.rand(len(i), generator=g, device="cuda", dtype=torch.float64) * (n - 1 - i)).long()
    j = torch.where(torch.rand(len(i), generator=g, device="cuda") < P_NEAR, near, far)
    keep = j < n
    d = torch.arange(n, device="cuda")
    key = torch.unique(torch.cat([i[keep] * n + j[keep], d * n + d]))
    row, col = key // n, key % n
    val = torch.rand(len(key), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    diag = row == col
    val[diag] = 0.0
    val[diag] = 1.0 + torch.zeros(n, device="cuda", dtype=torch.float64).index_add_(0, row, val.abs())
    rp = torch.zeros(n + 1, device="cuda", dtype=torch.int64)
    rp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return rp.int(), col.int(), val


@functools.lru_cache(maxsize=4)
def _band_host(g):
    return gen.laplace2d_cholesky(g)


@functools.lru_cache(maxsize=6)
def _nd_host(g):
    """The 3D Laplacian's pattern in elimination order, and its fronts."""
    return gen.laplace3d_nd_matrix(g)[:5]


@functools.lru_cache(maxsize=2)
def _mix_host(mix, count, nmax, rhs_max):
    m = gen.mix(count, seed=mix, nmin=1000, nmax=nmax, rhs_max=rhs_max)
    return m, np.concatenate([np.diff(m.system(s)[0].row_ptr) for s in range(count)])


def _mix(case, seed):
    """The mix's structure with its rows scaled by the seed (an equilibrated batch), and right-hand sides."""
    m, lens = _mix_host(case["mix"], case["count"], case["nmax"], case["rhs_max"])
    val = m.val * np.repeat(0.5 + np.random.default_rng(seed).random(len(lens)), lens)
    return m, val, _rhs_values(len(m.b), seed)


def _side(n, power):
    return int(round(n ** (1.0 / power)))


class _View:
    """Device memory of a factor as torch sees it; the tensors made from it keep the factor."""

    def __init__(self, factor, ptr, count, typestr):
        self.factor = factor
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


class Factor:
    """A multifrontal factor kept on the device, as a direct solver keeps it."""

    def __init__(self, row_ptr, col, val, front_start, front_parent, max_width=400):
        L = _lib.lib()
        self.h = ctypes.c_void_p()
        rc = L.sptrsv_factor_multifrontal(0, len(row_ptr) - 1, row_ptr, col, val, len(front_start) - 1, front_start,
                                          front_parent, max_width, ctypes.byref(self.h))
        if rc:
            raise RuntimeError("sptrsv_factor_multifrontal: status %d" % rc)
        n, nnz, nsn = ctypes.c_int(), ctypes.c_int64(), ctypes.c_int()
        L.sptrsv_factor_info(self.h, ctypes.byref(n), ctypes.byref(nnz), ctypes.byref(nsn))
        self.n, self.nnz, self.nsn = n.value, nnz.value, nsn.value
        p = [ctypes.c_void_p() for _ in range(3)]
        rc = L.sptrsv_factor_device(self.h, *[ctypes.byref(q) for q in p])
        if rc:
            raise RuntimeError("sptrsv_factor_device: status %d" % rc)
        self.ptr = [q.value for q in p]

    def tensors(self):
        return (torch.as_tensor(_View(self, self.ptr[0], self.n + 1, "<i4"), device="cuda"),
                torch.as_tensor(_View(self, self.ptr[1], self.nnz, "<i4"), device="cuda"),
                torch.as_tensor(_View(self, self.ptr[2], self.nnz, "<f8"), device="cuda"))

    def host(self):
        rp, col = np.empty(self.n + 1, dtype=np.int64), np.empty(self.nnz, dtype=np.int32)
        val, sn = np.empty(self.nnz), np.empty(self.nsn + 1, dtype=np.int32)
        _lib.lib().sptrsv_factor_copy(self.h, rp, col, val, sn)
        return rp, col, val, sn

    def __del__(self):
        if self.h:
            _lib.lib().sptrsv_factor_free(self.h)


def _partition(front_start, max_width=400):
    """The supernodes of the factor: every front's pivots in equal pieces of at most max_width."""
    sn = [0]
    for f0, f1 in zip(front_start[:-1].tolist(), front_start[1:].tolist()):
        step = -(-(f1 - f0) // -(-(f1 - f0) // max_width))
        sn += [min(f1, a + step) for a in range(f0, f1, step)]
    return np.array(sn, dtype=np.int32)


def _fronts(g):
    """(first pivot, end of the pivots, rows below) of every front, in order."""
    rp, col, _, fs, fp = _nd_host(g)
    kids = [[] for _ in fp]
    for k, p in enumerate(fp):
        if p >= 0:
            kids[p].append(k)
    below = [None] * len(fp)
    for t in range(len(fp)):
        a, b = int(fs[t]), int(fs[t + 1])
        s = np.unique(np.concatenate([col[rp[a]:rp[b]]] + [below[k] for k in kids[t]]))
        below[t] = s[s >= b]
        yield a, b, below[t]


def _nd_input(n, seed):
    """An SPD matrix on the 3D Laplacian's pattern: a diffusion problem with varying coefficients."""
    rp, col, val, fs, fp = _nd_host(_side(n, 3))
    rng = np.random.default_rng(seed)
    v = np.where(val > 0, 6.0 + 0.5 * rng.random(len(val)), -1.0 + 0.25 * rng.random(len(val)))
    return rp, col, v, fs, fp


def _rhs_values(count, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    return torch.rand(count, generator=g, device="cuda", dtype=torch.float64) * 2 - 1


def _matrix(case, seed):
    """(row_ptr, col, val on the device, supernodes or None, what keeps them alive)."""
    if case["matrix"] == "random":
        return (*_random_csr(case["n"], seed), None, None)
    if case["matrix"] == "band":
        m = _band_host(_side(case["n"], 2))
        g = torch.Generator(device="cuda").manual_seed(seed)
        val = torch.from_numpy(m.val).cuda()
        # every row scaled: the factor of D A D for a diagonal D, as an equilibrated system has it
        s = 0.5 + torch.rand(m.n, generator=g, device="cuda", dtype=torch.float64)
        rp, col = torch.from_numpy(m.row_ptr).cuda(), torch.from_numpy(m.col).cuda()
        return rp.int(), col, val * s[col.long()], None, None
    f = Factor(*_nd_input(case["n"], seed))
    return (*f.tensors(), _partition(_nd_host(_side(case["n"], 3))[3]), f)


# ------------------------------------------------------------------------------------------------

def prepare(case, seed):
    st = {"kind": case["kind"]}
    if case["kind"] == "solve":
        n, rhs = case["n"], case["rhs"]
        rp, col, val, sn, keep = _matrix(case, seed)
        torch.cuda.synchronize()
        s = sp.Solver().analyse_device(n, col.numel(), rp.data_ptr(), col.data_ptr(), val.data_ptr())
        if sn is not None:
            s.set_supernodes(sn)
        st.update(solver=s, keep=(rp, col, val, keep), rhs=rhs, layout=sp.ROW_MAJOR if case["row_major"] else sp.COL_MAJOR,
                  opts=sp.make_opts(precision=case["precision"]))
        st["b"] = _rhs_values(n * rhs, seed)
        st["x"] = torch.empty(n * rhs, device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
    elif case["kind"] == "factor":
        st["input"] = _nd_input(case["n"], seed)
        st["factor"] = None
    elif case["kind"] == "analyse":
        st["csr"] = _random_csr(case["n"], seed)
        torch.cuda.synchronize()
        st["solver"] = sp.Solver()
    elif case["kind"] == "dropin_gauss":
        rp, col, val = (t.cpu().numpy() for t in _random_csr(case["n"], seed))
        st.update(n=case["n"], rhs=case["rhs"], row_index=rp.astype(np.uint64), col=col, val=val,
                  b=_rhs_values(case["n"] * case["rhs"], seed).cpu().numpy(), x=np.zeros(case["n"] * case["rhs"]))
    elif case["kind"] == "dropin_supernodal":
        rp, col, val, sn = Factor(*_nd_input(case["n"], seed)).host()
        st.update(n=case["n"], rhs=case["rhs"], row_index=rp.astype(np.uint64), col=col, val=val, snodes=sn,
                  b=_rhs_values(case["n"] * case["rhs"], seed).cpu().numpy(), x=np.zeros(case["n"] * case["rhs"]))
    elif case["kind"] == "batch":
        m, val, st["b"] = _mix(case, seed)
        st["batch"] = sp.Batch(m.n, m.rhs, m.row_ptr, m.col, val)
        st["x"] = torch.empty_like(st["b"])
        torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind == "solve":
        # the handle has a stream of its own: its sync() orders the result and reports the solve's status
        st["solver"].solve_device(st["b"].data_ptr(), st["x"].data_ptr(), st["rhs"], st["layout"], st["opts"])
        rc = st["solver"].sync()
        if rc:
            raise RuntimeError("solve: status %d" % rc)
        return st["x"]
    if kind == "factor":
        st["factor"] = None  # a refactorisation gives its memory back first
        st["factor"] = Factor(*st["input"])
        return list(st["factor"].tensors())
    if kind == "analyse":
        rp, col, val = st["csr"]
        s = st["solver"].analyse_device(rp.numel() - 1, col.numel(), rp.data_ptr(), col.data_ptr(), val.data_ptr())
        return {"levels": s.levels(), "level_rows": s.level_buckets()[1], "in_degree": s.in_degree()}
    if kind == "dropin_gauss":
        t = sp.base_gauss_upper(st["n"], st["val"], st["row_index"], st["col"], st["x"], st["b"], st["rhs"])
        if t < 0:
            raise RuntimeError("base_gauss_upper: status %d" % t)
        return st["x"]
    if kind == "dropin_supernodal":
        st["x"][:] = st["b"]  # solved in place, as the reference's callers do
        t = sp.supernodal_upper(len(st["snodes"]) - 1, st["snodes"], st["x"], st["val"], st["col"], st["row_index"], st["n"],
                                st["rhs"])
        if t < 0:
            raise RuntimeError("supernodal_upper: status %d" % t)
        return st["x"]
    st["batch"].solve_device(st["b"].data_ptr(), st["x"].data_ptr(), "chosen")
    st["batch"].sync()
    return st["x"]


# ------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _nd_size(g):
    """(entries of A, entries of U, flops of the factorisation)."""
    nnz = flops = 0
    for a, b, below in _fronts(g):
        w, m = b - a, len(below)
        nnz += w * (w + 1) // 2 + w * m
        flops += w**3 // 3 + w * w * m + w * m * (m + 1)
    return int(_nd_host(g)[0][-1]), nnz, flops


def _entries(case):
    if case.get("matrix") == "band":
        g = _side(case["n"], 2)
        return case["n"] * (g + 1) - g * (g + 1) // 2
    if case.get("matrix") == "nd" or case["kind"] == "dropin_supernodal":
        return _nd_size(_side(case["n"], 3))[1]
    return int(case["n"] * (MEAN * (1 - 0.03) + 1))  # merged and clipped off-diagonals, and the diagonal


def work(case):
    if case["kind"] == "batch":
        # half band factors (sqrt(n) + 1 entries a row), half random rows (10 a row on average)
        lo, hi = 1000.0, float(case["nmax"])
        ln = math.log(hi / lo)
        rows, cube = (hi - lo) / ln, (hi**1.5 - lo**1.5) / (1.5 * ln)
        m = (1 + case["rhs_max"]) / 2
        nnz, n = case["count"] / 2 * (cube + 11 * rows), case["count"] * rows
        return {"bytes": 12 * nnz + 4 * n + 16 * n * m, "flops": 2 * nnz * m}
    n = case["n"]
    if case["kind"] == "factor":
        a, u, flops = _nd_size(_side(n, 3))
        return {"bytes": 12 * a + 12 * u, "flops": flops}
    nnz = _entries(case)
    if case["kind"] == "analyse":
        return {"bytes": 12 * nnz + 4 * n + 16 * n, "flops": 2 * nnz}
    m = case["rhs"]
    return {"bytes": 12 * nnz + 4 * (n + 1) + 16 * n * m, "flops": 2 * nnz * m}


def _dense_solve(rp, col, val, b):
    """U x = b with U as a dense triangle."""
    n = rp.numel() - 1
    U = torch.zeros(n, n, device="cuda", dtype=torch.float64)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    U[row, col.long()] = val
    return torch.linalg.solve_triangular(U, b, upper=True)


def _sweep_solve(rp, col, val, b):
    """U x = b by sweeps x <- D^-1 (b - N x) until they stand still (dominant rows)."""
    n = rp.numel() - 1
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    off = row != col
    d = val[~off].unsqueeze(1)
    crow = torch.zeros(n + 1, device="cuda", dtype=torch.int64)
    crow[1:] = torch.cumsum(torch.bincount(row[off], minlength=n), 0)
    N = torch.sparse_csr_tensor(crow, col[off].long(), val[off], size=(n, n))
    x = b / d
    for k in range(600):
        y = (b - N @ x) / d
        if k % 10 == 9 and bool((y == x).all()):
            break
        x = y
    return x


def exact(case, seed):
    if case["kind"] == "analyse":
        return None  # whole numbers
    if case["kind"] == "batch":
        m, val, b = _mix(case, seed)
        out = []
        for s in range(m.count):
            c = m.system(s)[0]
            rp, col, v = (torch.from_numpy(a.copy()).cuda() for a in (c.row_ptr, c.col, val[m.nz_off[s]:m.nz_off[s + 1]]))
            bs = b[m.xb_off[s]:m.xb_off[s + 1]].reshape(c.n, -1)
            out.append((_dense_solve if m.kind[s] == 0 else _sweep_solve)(rp, col, v, bs).reshape(-1))
        return torch.cat(out)
    n = case["n"]
    if case["kind"] == "factor":
        if n > 20_000:
            return None
        rp, col, val, _, _ = _nd_input(n, seed)
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.from_numpy(np.diff(rp)).cuda())
        A = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        c = torch.from_numpy(col).cuda().long()
        A[row, c] = torch.from_numpy(val).cuda()
        A = torch.triu(A) + torch.triu(A, 1).T
        U = torch.linalg.cholesky(A, upper=True)
        rows, cols = [], []
        for a, b, below in _fronts(_side(n, 3)):
            for i in range(a, b):
                cols.append(np.concatenate([np.arange(i, b), below]))
                rows.append(np.full(len(cols[-1]), i))
        rows, cols = (torch.from_numpy(np.concatenate(v)).cuda() for v in (rows, cols))
        return [None, None, U[rows, cols]]
    rhs = case["rhs"]
    b = _rhs_values(n * rhs, seed)
    if case["kind"] == "solve":
        rp, col, val, _, keep = _matrix(case, seed)
        rows = case["row_major"]
        B = b.reshape(n, rhs) if rows else b.reshape(rhs, n).T.contiguous()
        x = (_sweep_solve if case["matrix"] == "random" else _dense_solve)(rp, col, val, B)
        del keep
        return (x if rows else x.T).contiguous().reshape(-1)
    B = b.reshape(rhs, n).T.contiguous()
    if case["kind"] == "dropin_gauss":
        x = _sweep_solve(*_random_csr(n, seed), B)
    else:
        f = Factor(*_nd_input(n, seed))
        x = _dense_solve(*f.tensors(), B)
    return x.T.contiguous().reshape(-1).cpu().numpy()
