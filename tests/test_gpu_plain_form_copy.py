"""The plain FP64 form on a large operator (2^22 stored slots on): A read from
its exact FP32 copy, and the split first step, leave the iterates bit-identical."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pe,copy", [(20.0, 1), (20.1, 0)])
def test_copy_and_split_keep_the_iterates(pe, copy):
    A = W.convdiff3d(86, pe)
    assert A.nnz > 1 << 22
    b, _ = W.rhs_from_solution(A, seed=6)
    with Context(0) as c:
        x, _, _, s = c.solve_h(A, b, precision=N.PREC_FP64)
        assert s.status == N.SOLVE_CONVERGED and s.a_fp32 == copy
        c.set_exact_a32(False)
        x1, _, _, s1 = c.solve_h(A, b, precision=N.PREC_FP64)
        assert s1.a_fp32 == 0 and s1.iters == s.iters and s1.res == s.res and np.array_equal(x1, x)
        c.set_tuning(N.PREC_FP64, k1_split=0)
        x2, _, _, s2 = c.solve_h(A, b, precision=N.PREC_FP64)
        assert s2.iters == s.iters and np.array_equal(x2, x)
