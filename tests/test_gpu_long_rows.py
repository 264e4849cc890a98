"""One long row among short ones whose column offsets are a subset of the long
row's: the slice could be laid out offset-aligned, but the wide pre-pass sums a
row over its first entries only, so it must be laid out compactly."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W

pytestmark = pytest.mark.gpu


def long_row_matrix(n, row, width, seed=1):
    """Tridiagonal, diagonally dominant, with one row of `width` consecutive entries around its diagonal."""
    rng = np.random.default_rng(seed)
    near = np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= 1
    M = np.where(near, -rng.uniform(0.2, 1.0, (n, n)), 0.0)
    M[row, row - width // 2: row - width // 2 + width] = -rng.uniform(0.01, 0.05, width)
    np.fill_diagonal(M, 0.0)
    np.fill_diagonal(M, 0.5 + 1.2 * np.abs(M).sum(1))
    C, R = np.nonzero(M.T)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(C, minlength=n))])
    return W.CSC(n, ptr.astype(np.int32), R.astype(np.int32), M[R, C])


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_M_BF16, N.PREC_MIXED_FP32])
@pytest.mark.parametrize("width", [16, 17, 20, 40])
def test_solution(ctx, width, prec):
    A = long_row_matrix(1000, 500, width)
    x_true = np.random.default_rng(3).standard_normal(A.n)
    b = A.matvec(x_true)
    x, _, _, si = ctx.solve_h(A, b, precision=prec, tol=1e-9)
    assert si.status == N.SOLVE_CONVERGED
    # ||x - x_true|| <= ||A^-1|| ||r||, and ||A^-1||_inf <= 1 / (dominance >= 0.5)
    assert np.max(np.abs(x - x_true)) <= 2.0 * 1e-9 * np.linalg.norm(b) * 2.0


def hub_slice_matrix(n, row, width, nlong, step):
    """A row of `width` entries with `nlong` - 1 rows of 17 entries in its slice of 32, short rows elsewhere."""
    A = long_row_matrix(n, row, width)
    M = np.zeros((n, n))
    M[A.idx, np.repeat(np.arange(n), np.diff(A.ptr))] = A.val
    rng = np.random.default_rng(5)
    first = row - row % 32
    others = [r for r in range(first, first + 32) if r != row][: nlong - 1]
    for r in others:
        cols = (r + step * np.arange(-8, 9)) % n
        M[r, cols] = -rng.uniform(0.01, 0.05, 17)
        M[r, r] = 0.5 + 1.2 * np.abs(M[r]).sum()
    C, R = np.nonzero(M.T)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(C, minlength=n))])
    return W.CSC(n, ptr.astype(np.int32), R.astype(np.int32), M[R, C])


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_M_FP32])
@pytest.mark.parametrize("width,nlong,step", [(400, 4, 7), (400, 5, 7), (400, 5, 1), (400, 31, 7), (400, 32, 1), (40, 6, 7), (64, 20, 1)])
def test_hub_row_beside_other_long_rows(ctx, width, nlong, step, prec):
    """Slices mostly of padding: compact, their long rows summed apart in the one-launch solver; others keep their slots."""
    A = hub_slice_matrix(1500, 505, width, nlong, step)
    x_true = np.random.default_rng(3).standard_normal(A.n)
    b = A.matvec(x_true)
    x, _, _, si = ctx.solve_h(A, b, precision=prec, tol=1e-9)
    assert si.status == N.SOLVE_CONVERGED
    assert np.max(np.abs(x - x_true)) <= 2.0 * 1e-9 * np.linalg.norm(b) * 2.0
