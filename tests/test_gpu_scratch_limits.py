"""Calls that find no device memory for the scratch they can do without: they
take the path without it and give the same answer."""
import contextlib

import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def room(left_bytes):
    """The free device memory taken, but for left_bytes and a few MB."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:
        want = torch.cuda.mem_get_info()[0] - left_bytes
        # (torch serves requests under 10 MB from pieces of 20 MB)
        while want >= 10 << 20:
            try:
                held.append(torch.empty(want, dtype=torch.uint8, device="cuda"))
                want = torch.cuda.mem_get_info()[0] - left_bytes
            except torch.OutOfMemoryError:
                want -= 2 << 20
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def warm(*calls):
    """Loads the kernels of the calls on a context of their own (and frees it)."""
    with Context(0) as c:
        for A, b, opt in calls:
            c.solve_h(A, b, **opt)


def test_plain_form_without_the_fp32_copy():
    A = W.convdiff3d(86, 20.0)                    # 4.4 M slots: a copy of 17.6 MB
    b, _ = W.rhs_from_solution(A, seed=6)
    opt = dict(precision=N.PREC_FP64, tol=1e-6)
    warm((A, b, opt))
    with Context(0) as c:
        c.set_exact_a32(False)
        x, _, _, s = c.solve_h(A, b, **opt)
        c.set_exact_a32(True)
        with room(8 << 20):
            x1, _, _, s1 = c.solve_h(A, b, **opt)
        x2, _, _, s2 = c.solve_h(A, b, **opt)
    assert (s.a_fp32, s1.a_fp32, s2.a_fp32) == (0, 0, 1)
    assert s1.status == N.SOLVE_CONVERGED and np.array_equal(x1, x) and np.array_equal(x2, x)


def test_one_launch_solver_without_its_vectors():
    big, A = W.convdiff2d(552, 10.0), W.convdiff2d(548, 10.0)   # 304704 rows: the launches; 300304: one launch, 9.6 MB
    opt = dict(precision=N.PREC_FP64, tol=1e-4)
    bb, _ = W.rhs_from_solution(big, seed=6)
    b, _ = W.rhs_from_solution(A, seed=6)
    warm((big, bb, opt), (A, b, opt))
    with Context(0) as c:
        c.solve_h(big, bb, **opt)
        with room(4 << 20):
            before = c.launches
            x, _, _, s = c.solve_h(A, b, **opt)
            assert c.launches - before > 80
        assert s.status == N.SOLVE_CONVERGED
        assert np.linalg.norm(b - A.matvec(x)) < 1.01e-4 * np.linalg.norm(b)
        before = c.launches
        c.solve_h(A, b, **opt)
        assert c.launches - before < 60


def test_build_without_the_lists_of_the_larger_groups():
    import torch

    A = W.convdiff3d(128, 20.0)                   # 2 M columns: lists of 16.8 MB
    d = [torch.from_numpy(a).cuda() for a in (A.ptr, A.idx, A.val)]
    m = [torch.zeros(A.nnz, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    with Context(0) as c:
        c.build_d(A.n, A.nnz, *d, m[0], precision=N.PREC_FP64)
    with Context(0) as c:
        c.build_d(A.n, A.nnz, *d, m[1], precision=N.PREC_MIXED_FP32, ls_method=N.LS_HOUSEHOLDER)
        torch.cuda.synchronize()
        with room(8 << 20):
            info = c.build_d(A.n, A.nnz, *d, m[1], precision=N.PREC_FP64)
    assert info.cols_small == A.n and torch.equal(m[0], m[1])
