"""Batches solved a cluster per system: every cluster size (systems of 4 to
5000 rows, at the edges of a CTA's rows), 1 to 8 right-hand sides, rows longer
than the prefetched entries, frozen and zero right-hand sides, x0 and maxiter;
against the known solutions and the oracle's counts."""
import numpy as np
import pytest

import oracle
from dcu_b200 import native as N
from dcu_b200 import workloads as W
from tests.test_gpu_spai_groups import matrix

pytestmark = pytest.mark.gpu


def _assemble(parts):
    offs = np.cumsum([0] + [A.n for A in parts])
    ptr = np.concatenate([[0]] + [A.ptr[1:].astype(np.int64) + z for A, z in
                                  zip(parts, np.cumsum([0] + [A.nnz for A in parts]))])
    return offs, W.CSC(int(offs[-1]), ptr.astype(np.int32),
                       np.concatenate([A.idx + o for A, o in zip(parts, offs)]).astype(np.int32),
                       np.concatenate([A.val for A in parts]))


def _run(ctx, parts, nrhs, X0=None, B=None, **opt):
    import torch

    offs, A = _assemble(parts)
    rng = np.random.default_rng(5)
    Xt = rng.standard_normal((A.n, nrhs))
    if B is None:
        B = np.stack([A.matvec(Xt[:, q]) for q in range(nrhs)], 1)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X = d(np.zeros_like(Xt) if X0 is None else X0)
    before = ctx.launches
    it, st, _, si = ctx.batch_solve_d(d(offs.astype(np.int32)), A.n, A.nnz, d(A.ptr), d(A.idx), d(A.val), d(B), X, **opt)
    # a launch per cluster size, none per iteration
    assert ctx.launches - before < 40
    return offs, A, Xt, B, X.cpu().numpy(), it, st, si


def _systems(nrhs):
    # rows a pass takes: 128 at 8 right-hand sides, 256 at 4, 512 below
    unit = {8: 128, 4: 256}.get(nrhs, 512)
    sizes = [4, 31, 32, 33, 2 * unit - 1, 2 * unit, 2 * unit + 1, 4 * unit + 5, 8 * unit + 3]
    if nrhs == 8:
        sizes += [16 * unit, 16 * unit + 1, 16 * unit + 240]   # 16 CTAs from 2049 rows
    return [matrix(n, min(n, 3 + n % 4), min(n, 6), n) for n in sizes]


@pytest.mark.parametrize("nrhs", [1, 2, 4, 8])
def test_cluster_sizes(ctx, nrhs):
    parts = _systems(nrhs)
    offs, A, Xt, B, X, it, st, si = _run(ctx, parts, nrhs, tol=1e-10)
    assert (st == N.SOLVE_CONVERGED).all() and si.iters == it.max()
    for s, P in enumerate(parts):
        r = slice(offs[s], offs[s + 1])
        m, _, _, _ = oracle.spai(P, "householder")
        for q in range(nrhs):
            ref = oracle.bicgstab(P, m, B[r, q], None, tol=1e-10, tol_mode="rel", maxiter=1000)
            assert abs(int(it[s, q]) - ref["iters"]) <= 1
            res = np.linalg.norm(B[r, q] - P.matvec(X[r, q]))
            # the recurrence residual met 1e-10; the true one differs by rounding
            assert res < 1.01e-10 * np.linalg.norm(B[r, q])


def test_long_rows_and_x0(ctx):
    parts = [matrix(700, 12, 9, 1), matrix(300, 15, 20, 2), matrix(1500, 7, 5, 3)]
    X0 = np.random.default_rng(1).standard_normal((2500, 2))
    offs, A, Xt, B, X, it, st, _ = _run(ctx, parts, 2, X0=X0, tol=1e-11)
    assert (st == N.SOLVE_CONVERGED).all()
    assert np.linalg.norm(X - Xt) < 1e-9 * np.linalg.norm(Xt)


def test_frozen_pairs_and_limits(ctx):
    parts = [matrix(400, 5, 5, 4), matrix(900, 6, 9, 5)]
    offs, A = _assemble(parts)
    rng = np.random.default_rng(2)
    B = rng.standard_normal((A.n, 4))
    B[:, 1] = 0.0                                  # x = 0 solves it before the first iteration
    _, _, _, _, X, it, st, _ = _run(ctx, parts, 4, B=B, tol=1e-10)
    assert (st == N.SOLVE_CONVERGED).all() and (it[:, 1] == 1).all() and not X[:, 1].any()
    _, _, _, _, X, it, st, si = _run(ctx, parts, 4, B=B, tol=1e-30, maxiter=4)
    assert (st[:, [0, 2, 3]] == N.SOLVE_MAXITER).all() and (it[:, [0, 2, 3]] == 4).all() and si.iters == 4
    assert np.isfinite(X).all()
    B[10, 2] = np.nan                              # one bad right-hand side leaves the others alone
    _, _, _, _, X2, it, st, _ = _run(ctx, parts, 4, B=B, tol=1e-10)
    assert st[0, 2] == N.SOLVE_BREAKDOWN and (np.delete(st, 2, 1) == N.SOLVE_CONVERGED).all()


def test_repeats_are_bit_identical(ctx):
    parts = [matrix(n, 5, 5, n) for n in (150, 600, 2300, 5000, 350)]
    out = [_run(ctx, parts, 4, tol=1e-10)[4] for _ in range(3)]
    assert all(np.array_equal(o, out[0]) for o in out)
