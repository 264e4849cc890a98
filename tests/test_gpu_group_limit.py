"""A tuned |I| limit (group_max_ni) between the group kernel's first size (28
rows) and its 32: columns up to the limit stay on a group, the rest go to the
CTA kernel."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


def matrix(n=600, seed=4):
    """Columns of 6 and 7 random entries near the diagonal: |I| of 20 to 40, candidates up to 49."""
    rng = np.random.default_rng(seed)
    ptr, idx, val = [0], [], []
    for c in range(n):
        near = np.arange(max(0, c - 40), min(n, c + 41))
        rows = np.union1d(rng.choice(near, 5 + c % 2, replace=False), [c])
        idx.append(rows)
        val.append(np.where(rows == c, 10.0, rng.uniform(-1, 1, len(rows))))
        ptr.append(ptr[-1] + len(rows))
    return W.CSC(n, np.array(ptr, np.int32), np.concatenate(idx).astype(np.int32), np.concatenate(val))


def heights(A):
    cols = [A.idx[A.ptr[c]:A.ptr[c + 1]] for c in range(A.n)]
    return np.array([len(np.unique(np.concatenate([cols[j] for j in cols[c]]))) for c in range(A.n)])


@pytest.mark.parametrize("limit", [24, 28, 29, 30, 31, 32])
def test_columns_above_the_limit_go_to_the_cta_kernel(limit):
    A = matrix()
    h = heights(A)
    assert ((h > 28) & (h <= 32)).sum() > 50 and (h > 32).sum() > 10 and np.diff(A.ptr).max() <= 7
    with Context(0) as c:
        m0, _, b0 = c.build_h(A)
        c.set_tuning(N.PREC_FP64, group_max_ni=limit)
        m, _, b = c.build_h(A)
    # (32 is the default: taller columns stay on the larger groups)
    assert b.cols_large == (0 if limit == 32 else (h > limit).sum()) and b.cols_small + b.cols_large == A.n
    assert b0.cols_large == 0
    assert np.max(np.abs(m - m0)) <= 1e-12 * np.max(np.abs(m0))
