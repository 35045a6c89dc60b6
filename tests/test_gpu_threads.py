"""Handles on several host threads at once, each with rows of another mean length (the sweeps' shared memory
follows it): every solve returns OK and, the mixed ones, the bits of a solve alone.  With graphs and
without (kernels launched on every solve)."""
import threading

import numpy as np
import pytest

import sptrsv_gb300 as sp
from sptrsv_gb300 import gen

pytestmark = pytest.mark.gpu

N = 12_000
RTOL = 1e-12  # FP64: rounding of the random recipe's solutions, as between the exact kernels


def _handle(mean):
    m = gen.random_upper(N, mean, 0.9, 64, 3)
    return sp.Solver(0).analyse(m.row_ptr, m.col, m.val), gen.uniform(1, N)


def _solve(s, b, precision):
    return s.solve(b, precision=precision, schedule="jacobi" if precision == "mixed" else "auto")


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("precision,means,handles,solves", [
    ("fp64", (4.0, 16.0, 8.0), 40, 100), ("mixed", (8.0, 12.5, 11.0), 40, 10)])
def test_handles_of_different_row_lengths(monkeypatch, precision, means, handles, solves, graphs):
    if not graphs:
        monkeypatch.setenv("SPTRSV_NO_GRAPH", "1")
    alone = []
    for mean in means:
        s, b = _handle(mean)
        alone.append(_solve(s, b, precision))
        s.close()
    wrong = []

    def work(mean, ref):
        for _ in range(handles):
            s, b = _handle(mean)
            for _ in range(solves):
                try:
                    x = _solve(s, b, precision)
                except sp.SptrsvError as e:
                    wrong.append((mean, e.status))
                    continue
                if precision == "mixed" and not np.array_equal(x, ref):
                    wrong.append((mean, "bits"))
                elif np.max(np.abs(x - ref)) > RTOL * np.max(np.abs(ref)):
                    wrong.append((mean, "x"))
            s.close()

    threads = [threading.Thread(target=work, args=a) for a in zip(means, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[:5])
