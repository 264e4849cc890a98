"""Hub columns by panels where a block has fewer rows than columns, or a zero
column: counted as singular as on the one-CTA path, the other columns unharmed."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


def from_columns(n, cols):
    ptr = np.concatenate([[0], np.cumsum([len(r) for r, _ in cols])]).astype(np.int32)
    return W.CSC(n, ptr, np.concatenate([r for r, _ in cols]).astype(np.int32), np.concatenate([v for _, v in cols]))


def matrix(wide, rows, zero, n=900, seed=5):
    """Column 0 has `wide` entries; the columns it names lie within `rows` rows (0: each has its own
    diagonal, |I| >= |J|); `zero` of them hold zeros only.  The rest is a diagonal with two entries beside it."""
    rng = np.random.default_rng(seed)
    J = np.sort(rng.choice(np.arange(1, n), wide, replace=False))
    inside = np.sort(rng.choice(n, rows, replace=False)) if rows else None
    cols = []
    for c in range(n):
        if c == 0:
            r = J
        elif c in J and rows:
            r = np.sort(rng.choice(inside, 3, replace=False))
        else:
            r = np.union1d(rng.choice(n, 2, replace=False), [c])
        v = np.where(r == c, 4.0, rng.uniform(-1, 1, len(r)))
        cols.append((r, v))
    for c in J[10:10 + zero]:
        cols[c] = (cols[c][0], np.zeros(len(cols[c][0])))
    return from_columns(n, cols), J


# |J| at and around multiples of the panel of 8; |I| ends inside a panel, at its edge, and within the look-ahead
@pytest.mark.parametrize("wide,rows,zero", [(400, 150, 0), (404, 152, 0), (399, 145, 0), (300, 0, 1), (297, 0, 9)])
def test_degenerate_hubs(wide, rows, zero):
    A, J = matrix(wide, rows, zero)
    out = []
    for area in (0, -1):
        with Context(0) as c:
            c.set_tuning(N.PREC_FP64, cta_max_area=area)
            out.append(c.build_h(A, precision=N.PREC_FP64))
    (m, res, info), (m1, res1, info1) = out
    assert info.cols_hub == 1 and info1.cols_hub == 0
    assert info.cols_singular == info1.cols_singular >= 1
    # every column but the hub, and those that meet a zero column, is the same on both paths
    cols = np.repeat(np.arange(A.n), np.diff(A.ptr))
    keep = cols != 0
    fine = np.isfinite(m1) & keep
    assert np.array_equal(np.isfinite(m)[keep], np.isfinite(m1)[keep])
    assert np.array_equal(m[fine], m1[fine])
    assert fine.sum() > A.n
