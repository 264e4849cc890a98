"""Which solves run as one launch, told by the launches of the call (the launch
sequence takes two chunks of 8 iterations of five and more at least), and its
forms with scattered columns beyond one cluster's shared vectors."""
import numpy as np
import pytest

import oracle
from dcu_b200 import native as N
from dcu_b200 import workloads as W
from tests.test_gpu_one_launch import _band

pytestmark = pytest.mark.gpu


def assemble(n, R, C, V):
    """CSC of the off-diagonal entries (R, C, V), repeats dropped, with a row-dominant diagonal."""
    key, first = np.unique(C.astype(np.int64) * n + R, return_index=True)
    C, R, V = key // n, key % n, V[first]
    off = R != C
    C, R, V = C[off], R[off], V[off]
    r = np.arange(n)
    d = 0.5 + 1.2 * np.bincount(R, weights=np.abs(V), minlength=n)
    C, R, V = np.concatenate([C, r]), np.concatenate([R, r]), np.concatenate([V, d])
    o = np.lexsort((R, C))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(C, minlength=n))])
    return W.CSC(n, ptr.astype(np.int32), R[o].astype(np.int32), V[o])


def scattered(n, deg=4, seed=0):
    rng = np.random.default_rng(seed)
    return assemble(n, rng.integers(0, n, n * deg), rng.integers(0, n, n * deg), -rng.uniform(0.2, 1.0, n * deg))


def one_launch(ctx, A, prec, expect=True, tol=1e-10, count=None):
    """A solve whose analysis, build and iterations take under 60 launches if and only if one launch is expected."""
    x_true = np.random.default_rng(A.n).standard_normal(A.n)
    b = A.matvec(x_true)
    before = ctx.launches
    x, _, _, si = ctx.solve_h(A, b, precision=prec, tol=tol, maxiter=2000)
    launches = ctx.launches - before
    assert si.status == N.SOLVE_CONVERGED and si.true_res < tol * np.linalg.norm(b)
    assert launches < 60 if expect else launches > 80, launches
    # row-dominant by 0.5 and more: ||A^-1||_inf <= 2
    assert np.max(np.abs(x - x_true)) <= 2.0 * tol * np.linalg.norm(b) + 1e-12 * np.max(np.abs(x_true))
    if count is not None:
        assert abs(si.iters - count) <= 1
    return x


# the whole vectors in each CTA up to about 6500 rows; the grid form above; edges of its blocks of 512 rows
@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_M_BF16])
@pytest.mark.parametrize("n", [600, 5000, 8191, 8192, 8193, 12000, 16384, 16385])
def test_scattered_columns(ctx, n, prec):
    A = scattered(n)
    count = None
    if prec == N.PREC_FP64:
        m, _, _, _ = oracle.spai(A, "householder")
        b = A.matvec(np.random.default_rng(A.n).standard_normal(A.n))
        count = oracle.bicgstab(A, m, b, None, tol=1e-10, tol_mode="rel", maxiter=2000)["iters"]
    x = one_launch(ctx, A, prec, count=count)
    b = A.matvec(np.random.default_rng(A.n).standard_normal(A.n))
    again, _, _, _ = ctx.solve_h(A, b, precision=prec, tol=1e-10, maxiter=2000)
    assert np.array_equal(x, again)


def test_scattered_columns_with_long_rows(ctx):
    # (entries of the long rows beside 512 short ones: too much for a cluster's CTA of 1024 rows)
    A = W.circuit_like(n=12000, target_nnz=56400)
    b, x_true = W.rhs_from_solution(A, seed=3)
    x, _, _, si = ctx.solve_h(A, b, tol=1e-10, maxiter=2000)
    assert si.status == N.SOLVE_CONVERGED
    assert np.linalg.norm(b - A.matvec(x)) < 1.1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [31, 257, 4096, 16384, 16385, 75777, 303105 - 1])
def test_taken(ctx, n):
    one_launch(ctx, _band(n), N.PREC_FP64)


@pytest.mark.parametrize("n,prec", [(303105, N.PREC_FP64), (4096, N.PREC_MIXED_FP32), (20000, N.PREC_MIXED_BF16)])
def test_not_taken(ctx, n, prec):
    one_launch(ctx, _band(n), prec, expect=False, tol=1e-9)
