"""Systems of a batch do not see each other: the padding of the offset-aligned
layout reaches over a system's ends (stencils), where the neighbour's vectors
may be unwritten scratch or hold its NaN."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


def _batch(P, count):
    k = np.arange(count)[:, None]
    ptr = np.concatenate([[0], (P.ptr[None, 1:] + P.nnz * k).ravel()]).astype(np.int32)
    return W.CSC(P.n * count, ptr, (P.idx[None, :] + P.n * k).ravel().astype(np.int32), np.tile(P.val, count))


def _solve(ctx, A, offs, B, **opt):
    import torch

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = d(np.asarray(offs, np.int32)), A.n, A.nnz, d(A.ptr), d(A.idx), d(A.val), d(B)
    X = torch.zeros(B.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    it, st, _, _ = ctx.batch_solve_d(*args, X, **opt)
    return X.cpu().numpy(), it, st


# clusters of 1, 4 and 16 CTAs, more systems than run at once; the tiles
SHAPES = [(2, 7, 400, 1), (2, 40, 60, 4), (3, 13, 60, 1), (3, 16, 16, 8), (2, 6, 4096, 2)]


@pytest.mark.parametrize("dim,m,count,nrhs", SHAPES)
def test_scratch_of_an_earlier_call(dim, m, count, nrhs):
    A = _batch(W.convdiff(dim, m, 10.0), count)
    offs = np.arange(count + 1) * (A.n // count)
    B = np.random.default_rng(1).standard_normal((A.n, nrhs))
    with Context(0) as c:
        _solve(c, A, offs, np.full(B.shape, np.nan))    # every vector of the scratch NaN
        X, it, st = _solve(c, A, offs, B, tol=1e-10)
    assert (st == N.SOLVE_CONVERGED).all()
    with Context(0) as c:
        X0, it0, _ = _solve(c, A, offs, B, tol=1e-10)
    assert np.array_equal(X, X0) and np.array_equal(it, it0)


@pytest.mark.parametrize("dim,m,count,nrhs", SHAPES)
def test_a_bad_right_hand_side_stays_in_its_system(ctx, dim, m, count, nrhs):
    A = _batch(W.convdiff(dim, m, 10.0), count)
    n = A.n // count
    offs = np.arange(count + 1) * n
    B = np.random.default_rng(2).standard_normal((A.n, nrhs))
    X0, it0, st0 = _solve(ctx, A, offs, B, tol=1e-10)
    bad = [0, count // 2, count - 1]
    for s in bad:
        B[s * n + n // 3, 0] = np.nan
    X, it, st = _solve(ctx, A, offs, B, tol=1e-10)
    assert (st0 == N.SOLVE_CONVERGED).all()
    assert (st[bad, 0] == N.SOLVE_BREAKDOWN).all()
    keep = np.ones((count, nrhs), bool)
    keep[bad, 0] = False
    assert (st[keep] == N.SOLVE_CONVERGED).all() and np.array_equal(it[keep], it0[keep])
    rows = np.repeat(keep, n, axis=0)
    assert np.array_equal(X[rows], X0[rows])
