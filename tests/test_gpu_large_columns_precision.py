"""FP32 builds for FP64 vectors: the columns of the CTA kernel run in FP64 while
there are few entries in all, in FP32 (as the FP32-vector forms') beyond."""
import numpy as np
import pytest

from dcu_b200 import native as N
from dcu_b200 import workloads as W

pytestmark = pytest.mark.gpu


def band(n, deg, width, seed=3):
    """deg random entries a column within `width` of the diagonal, and a dominant diagonal."""
    rng = np.random.default_rng(seed)
    ptr, idx, val = [0], [], []
    for c in range(n):
        lo, hi = max(0, c - width), min(n, c + width + 1)
        rows = np.union1d(rng.choice(np.arange(lo, hi), deg, replace=False), [c])
        idx.append(rows)
        val.append(np.where(rows == c, 2.0 * deg, rng.uniform(-1, 1, len(rows))))
        ptr.append(ptr[-1] + len(rows))
    return W.CSC(n, np.array(ptr, np.int32), np.concatenate(idx).astype(np.int32), np.concatenate(val))


# 30 entries a column: about 30 K queued entries (|I| bound times |J| + 1) each, against 2^25 in all
@pytest.mark.parametrize("prec", [N.PREC_M_FP32, N.PREC_M_BF16])
@pytest.mark.parametrize("n,fp64", [(800, True), (1600, False)])
def test_precision_of_the_cta_columns(ctx, n, fp64, prec):
    A = band(n, 30, 150)
    m, _, info = ctx.build_h(A, precision=prec)
    assert info.cols_large == n and info.cols_singular == 0
    ref, _, _ = ctx.build_h(A, precision=N.PREC_FP64)
    err = np.max(np.abs(m - ref)) / np.max(np.abs(ref))
    # condition numbers below 100: FP64 errors below 1e-11, FP32 ones about 6e-8 and above
    assert err < 1e-11 if fp64 else 1e-9 < err < 1e-4
    if not fp64:
        m32, _, _ = ctx.build_h(A, precision=N.PREC_MIXED_FP32)
        assert np.array_equal(m, m32)
