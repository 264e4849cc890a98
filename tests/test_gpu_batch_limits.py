"""Batches at the limits of what the entry point takes: no rows at all, and the
batch's iteration counter when a pair breaks down inside an iteration."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import DcuError

pytestmark = pytest.mark.gpu


def _solve(ctx, A, offs, B, **opt):
    import torch

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X = torch.zeros(B.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    out = ctx.batch_solve_d(d(np.asarray(offs, np.int32)), A.n, A.nnz, d(A.ptr), d(A.idx), d(A.val), d(B), X, **opt)
    return X.cpu().numpy(), *out


@pytest.mark.parametrize("nsys", [1, 3])
@pytest.mark.parametrize("nrhs", [1, 8])
def test_a_batch_without_rows_is_refused(ctx, nsys, nrhs):
    A = W.convdiff2d(4, 10.0)
    with pytest.raises(DcuError, match="empty batch"):
        _solve(ctx, A, [0] * (nsys + 1), np.ones((A.n, nrhs)))


def test_counter_of_a_breakdown_inside_an_iteration(ctx):
    """A cyclic shift (M = 0 there) beside a diagonal: exact arithmetic, r = (b1, 0) after the first
    iteration, y = M p = 0 in the second, (r*, A y) = 0.  The pair stopped with one finished iteration, the
    batch in its second."""
    n = 6
    cols = [[1], [2], [0], [3], [4], [5]]
    A = W.CSC(n, np.arange(n + 1, dtype=np.int32), np.concatenate(cols).astype(np.int32), np.ones(n))
    # |b1|^2 = |b2|^2: alpha = 2
    X, it, st, _, si = _solve(ctx, A, [0, n], np.ones((n, 1)), tol=1e-10)
    assert st[0, 0] == N.SOLVE_BREAKDOWN and it[0, 0] == 1 and si.iters == 2
    assert np.array_equal(X[:, 0], [0.0, 0.0, 0.0, 1.0, 1.0, 1.0])


@pytest.mark.parametrize("count,rows,nrhs,tiles", [(4096, 16, 1, True), (100, 16, 1, False), (3000, 64, 2, True), (140, 64, 8, False)])
def test_many_small_systems_go_to_the_tiles(ctx, count, rows, nrhs, tiles):
    """Clusters pay a fixed time a system and iteration: hundreds at once, not thousands one after another."""
    P = W.convdiff2d(int(rows ** 0.5), 10.0)
    k = np.arange(count)[:, None]
    ptr = np.concatenate([[0], (P.ptr[None, 1:] + P.nnz * k).ravel()]).astype(np.int32)
    A = W.CSC(P.n * count, ptr, (P.idx[None, :] + P.n * k).ravel().astype(np.int32), np.tile(P.val, count))
    Xt = np.random.default_rng(1).standard_normal((A.n, nrhs))
    B = np.stack([A.matvec(Xt[:, q]) for q in range(nrhs)], 1)
    before = ctx.launches
    X, it, st, _, si = _solve(ctx, A, np.arange(count + 1) * P.n, B, tol=1e-10)
    launches = ctx.launches - before
    assert (st == N.SOLVE_CONVERGED).all()
    assert np.linalg.norm(X - Xt) <= 1e-8 * np.linalg.norm(Xt)
    # the tiles take five launches an iteration and more, the clusters one a size
    assert (launches > 5 * it.max()) == tiles
