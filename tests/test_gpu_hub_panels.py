"""Hub columns by panels: widths around multiples of the panel, blocks taller
than the panel kernel takes (the step kernels then run), |I| < |J| and the
forms that share the path, against the oracle and the one-CTA path."""
import numpy as np
import pytest

import oracle
from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context

pytestmark = pytest.mark.gpu


def hubs(n, widths, deg, seed):
    """Column h (h < len(widths)) has widths[h] entries; every other column deg random ones and its diagonal."""
    rng = np.random.default_rng(seed)
    ptr, idx, val = [0], [], []
    for c in range(n):
        k = widths[c] if c < len(widths) else deg + 1
        others = np.setdiff1d(rng.choice(n - len(widths), min(2 * k, n - len(widths)), replace=False) + len(widths), [c])
        rows = np.sort(np.append(others[:k - 1], c))
        idx.append(rows)
        val.append(np.where(rows == c, 4.0 + 0.1 * k, rng.uniform(-1, 1, len(rows))))
        ptr.append(ptr[-1] + len(rows))
    return W.CSC(n, np.array(ptr, np.int32), np.concatenate(idx).astype(np.int32), np.concatenate(val))


def _close(m, m_o, A, tol):
    cols = np.repeat(np.arange(A.n), np.diff(A.ptr))
    scale = np.zeros(A.n)
    np.maximum.at(scale, cols, np.abs(m_o))
    assert np.max(np.abs(m - m_o) / scale[cols]) <= tol


@pytest.mark.parametrize("widths", [(127, 128, 129), (64, 200, 96, 135), (161,)])
def test_widths(ctx, widths):
    A = hubs(900, widths, 3, len(widths))
    m_o, res_o, _, sing = oracle.spai(A, "householder")
    m, res, info = ctx.build_h(A, precision=N.PREC_FP64)
    assert info.cols_hub >= 1 and info.cols_singular == sing == 0
    # condition numbers of these columns are below 100
    _close(m, m_o, A, 1e-11)
    assert np.max(np.abs(res - res_o)) < 1e-11
    with Context(0) as c:
        c.set_tuning(N.PREC_FP64, cta_max_area=-1)
        m1, _, i1 = c.build_h(A, precision=N.PREC_FP64)
    assert i1.cols_hub == 0
    _close(m, m1, A, 1e-11)


def test_taller_than_a_panel(ctx):
    A = hubs(6000, (60, 50), 55, 7)                 # |I| ~ 2400 > 2048 rows
    m_o, _, _, sing = oracle.spai(A, "householder")
    m, _, info = ctx.build_h(A, precision=N.PREC_FP64)
    assert info.cols_hub >= 2 and info.max_ni > 2048 and info.cols_singular == sing == 0
    _close(m, m_o, A, 1e-11)


@pytest.mark.parametrize("prec", [N.PREC_M_FP32, N.PREC_M_BF16, N.PREC_MIXED_FP32])
def test_narrow_forms(ctx, prec):
    A = hubs(900, (130, 150), 3, 9)
    m_o, _, _, _ = oracle.spai(A, "householder")
    m, _, info = ctx.build_h(A, precision=prec)
    assert info.cols_hub >= 1
    _close(m, m_o, A, 2e-3)
    m2, _, _ = ctx.build_h(A, precision=prec)
    assert np.array_equal(m, m2)
