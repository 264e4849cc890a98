"""The autotuner on an operator that solves in one launch: what it keeps must not
decide for larger operators of the same form, which it did not measure."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


def test_a_small_operator_leaves_the_first_step_to_the_size():
    import torch

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    small, large = W.convdiff2d(40, 10.0), W.convdiff3d(86, 20.0)
    assert large.nnz > 1 << 22
    with Context(0) as c:
        b, _ = W.rhs_from_solution(small, seed=3)
        t = c.autotune_d(small.n, small.nnz, d(small.ptr), d(small.idx), d(small.val), d(b), reps=3, precision=N.PREC_FP64)
        assert t.k1_split == -1 and c.get_tuning(N.PREC_FP64).k1_split == -1
        b, _ = W.rhs_from_solution(large, seed=3)
        _, _, _, si = c.solve_h(large, b, precision=N.PREC_FP64, tol=1e-6)
        assert si.status == N.SOLVE_CONVERGED
        # split first step from 2^22 entries on: six kernels an iteration (five with the fused one)
        assert len(c.profile_iteration(2)) == 6
