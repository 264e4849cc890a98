"""Solves that run as one launch: sizes at the edges of its slices, blocks,
clusters and grids, every precision form, long rows, and the sizes just past
its range; each against the known solution and the oracle's count."""
import numpy as np
import pytest

import oracle
from dcu_b200 import native as N
from dcu_b200 import workloads as W
from tests.test_gpu_long_rows import long_row_matrix

pytestmark = pytest.mark.gpu


def _band(n, seed=0):
    """Unsymmetric tridiagonal matrix plus one far entry a row, diagonally dominant."""
    rng = np.random.default_rng(seed)
    r = np.arange(n)
    R = np.concatenate([r[1:], r[:-1], r])
    C = np.concatenate([r[:-1], r[1:], (r * 7 + 3) % n])
    key = np.unique(C * n + R)
    C, R = key // n, key % n
    off = C != R
    C, R = C[off], R[off]
    V = -rng.uniform(0.2, 1.0, len(R))
    d = 0.5 + 1.2 * np.bincount(R, weights=-V, minlength=n)
    C, R, V = np.concatenate([C, r]), np.concatenate([R, r]), np.concatenate([V, d])
    o = np.lexsort((R, C))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(C, minlength=n))])
    return W.CSC(n, ptr.astype(np.int32), R[o].astype(np.int32), V[o])


def _check(ctx, A, prec, tol=1e-10, count=None):
    x_true = np.random.default_rng(A.n).standard_normal(A.n)
    b = A.matvec(x_true)
    x, _, _, si = ctx.solve_h(A, b, precision=prec, tol=tol, maxiter=2000)
    assert si.status == N.SOLVE_CONVERGED
    bn = np.linalg.norm(b)
    # the solver's own verified residual, and the same from outside: b - A x is
    # summed in another order there (a few rounding errors of |A| |x|)
    assert si.true_res < tol * bn
    assert abs(si.bnorm - bn) <= 1e-12 * bn
    slack = 1e-14 * np.linalg.norm(np.abs(A.val)) * np.linalg.norm(x)
    assert np.linalg.norm(b - A.matvec(x)) < tol * bn + slack
    if count is not None:
        assert abs(si.iters - count) <= 1, (si.iters, count)
    return x, si


# 1 .. one slice .. CTA of 256 rows .. 16 CTAs of 256 and of 1024 rows (16384)
# .. the grid form with 1, 2 and 4 rows a thread .. past it
SIZES = [1, 2, 31, 32, 33, 255, 256, 257, 4095, 4097, 16383, 16384, 16385, 75777, 151553, 303105]


@pytest.mark.parametrize("n", SIZES)
def test_sizes(ctx, n):
    A = _band(n) if n > 2 else W.CSC(n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32),
                                     np.arange(2.0, 2.0 + n))
    m, _, _, _ = oracle.spai(A, "householder")
    b = A.matvec(np.random.default_rng(A.n).standard_normal(A.n))
    ref = oracle.bicgstab(A, m, b, None, tol=1e-10, tol_mode="rel", maxiter=2000)
    # (a diagonal A is solved by the half step: omega = 0 / 0 in the oracle, as in the reference)
    _check(ctx, A, N.PREC_FP64, count=ref["iters"] if n > 2 else None)


@pytest.mark.parametrize("prec", [N.PREC_MIXED_FP32, N.PREC_MIXED_BF16, N.PREC_M_FP32, N.PREC_M_BF16])
@pytest.mark.parametrize("n", [33, 5000, 40000])
def test_forms(ctx, n, prec):
    # (tolerance above what FP32 search vectors reach without replacements)
    _check(ctx, _band(n, 3), prec, tol=1e-9)


@pytest.mark.parametrize("width", [16, 17, 33, 130])
@pytest.mark.parametrize("n", [300, 1000])
def test_long_row(ctx, n, width):
    for prec in (N.PREC_FP64, N.PREC_M_BF16):
        _check(ctx, long_row_matrix(n, n // 2, width), prec)


def test_repeats_are_bit_identical(ctx):
    for A in (W.circuit_like(n=2000, target_nnz=9400), W.convdiff2d(150, 10.0)):
        b, _ = W.rhs_from_solution(A, seed=3)
        out = [ctx.solve_h(A, b, tol=1e-10) for _ in range(3)]
        assert all(np.array_equal(o[0], out[0][0]) and o[3].iters == out[0][3].iters for o in out)


def test_counter_and_limits(ctx):
    A = W.convdiff2d(40, 10.0)
    b, _ = W.rhs_from_solution(A, seed=3)
    x, _, _, si = ctx.solve_h(A, b, maxiter=5, tol=1e-30, verify=0)
    assert si.status == N.SOLVE_MAXITER and si.iters == 5 and si.true_res > 0
    x, _, _, si = ctx.solve_h(A, b, maxiter=1)
    assert si.status == N.SOLVE_MAXITER and si.iters == 1 and not x.any()
