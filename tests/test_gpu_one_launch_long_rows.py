"""One-launch solver: long rows in the form of one cluster that gathers remotely
(two rows a thread) and in the grid form (one, two and four rows a thread), and
two contexts that solve at once, each on every SM."""
import threading

import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context
from tests.test_gpu_one_launch_paths import assemble, one_launch

pytestmark = pytest.mark.gpu


def banded_with_long_rows(n, widths, seed=2):
    """Five diagonals and one long row of each width; the slices without one have one offset a position."""
    rng = np.random.default_rng(seed)
    r = np.arange(n)
    R, C = [], []
    for off in (-2, -1, 1, 2):
        ok = (r + off >= 0) & (r + off < n)
        R.append(r[ok])
        C.append(r[ok] + off)
    # rows in different blocks, the last of all among them; two in one slice
    rows = [n // 3, n // 3 + 1, n // 2 + 7, n - 1, 0]
    for row, w in zip(rows, widths):
        R.append(np.full(w, row))
        C.append(rng.choice(n, w, replace=False))
    R, C = np.concatenate(R), np.concatenate(C)
    return assemble(n, R, C, -rng.uniform(0.2, 1.0, len(R)))


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_M_FP32])
@pytest.mark.parametrize("widths", [(12, 13, 12, 11), (129, 400, 1000, 33, 130), (40,)])
@pytest.mark.parametrize("n", [12000, 16384, 20000, 100000, 250000])
def test_long_rows(ctx, n, widths, prec):
    one_launch(ctx, banded_with_long_rows(n, widths), prec)


def test_two_contexts_at_once():
    # 44 blocks, and one on every SM
    work = [W.convdiff2d(150, 10.0), W.convdiff3d(48, 20.0)]
    data = [(A, W.rhs_from_solution(A, seed=3)[0]) for A in work]
    with Context(0) as c:
        alone = [c.solve_h(A, b, tol=1e-10) for A, b in data]
    out, errors = [[], []], []

    def go(i):
        try:
            with Context(0) as c:
                for k in range(6):
                    A, b = data[(i + k) % 2]
                    out[i].append(((i + k) % 2, c.solve_h(A, b, tol=1e-10)))
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=go, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for runs in out:
        for k, (x, _, _, si) in runs:
            assert si.status == N.SOLVE_CONVERGED and si.iters == alone[k][3].iters
            assert np.array_equal(x, alone[k][0])
