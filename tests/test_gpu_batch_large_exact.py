"""A batch of 2^22 stored slots and more whose values are all exact in FP32: the
batched kernels read A's FP64 values, whatever the plain form of a single
solve of that size reads."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 8])
@pytest.mark.parametrize("pe", [20.0, 20.1])   # every value exact in FP32, some not
def test_known_solutions(nrhs, pe):
    import torch

    P, count = W.convdiff3d(54, pe), 4
    k = np.arange(count)[:, None]
    ptr = np.concatenate([[0], (P.ptr[None, 1:] + P.nnz * k).ravel()]).astype(np.int32)
    idx = (P.idx[None, :] + P.n * k).ravel().astype(np.int32)
    val, n = np.tile(P.val, count), P.n * count
    assert len(idx) > 1 << 22
    Xt = np.random.default_rng(3).standard_normal((n, nrhs))
    B = np.empty_like(Xt)
    for s in range(count):
        for q in range(nrhs):
            B[s * P.n:(s + 1) * P.n, q] = P.matvec(Xt[s * P.n:(s + 1) * P.n, q])
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X = torch.zeros(n, nrhs, dtype=torch.float64, device="cuda")
    with Context(0) as c:
        it, st, _, si = c.batch_solve_d(d(np.arange(count + 1, dtype=np.int32) * P.n), n, len(idx), d(ptr), d(idx), d(val),
                                        d(B), X, tol=1e-10)
    assert (st == N.SOLVE_CONVERGED).all() and si.a_fp32 == 0
    # A is an M-matrix whose rows and columns are dominant on the boundary only; at Pe 20 the error of
    # these solves stays within 1e3 residuals (1e-8 residuals give 2.5e-8 at 128^3)
    assert np.linalg.norm(X.cpu().numpy() - Xt) <= 1e-7 * np.linalg.norm(Xt)
