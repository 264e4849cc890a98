"""FP64 builds on the group kernels: columns at the edges of the three sizes
(|J|, |I|, candidates), banded and scattered, sorted and not, both schedules
and a column range, against the Householder oracle."""
import numpy as np
import pytest

import oracle
from dcu_b200 import native as N
from dcu_b200 import workloads as W

pytestmark = pytest.mark.gpu

# backward-stable QR on columns of condition < 1e3: a few thousand roundings
RTOL = 1e-12


def matrix(n, width, reach, seed, shuffle=False):
    """`width` entries a column: the diagonal (dominant) and width - 1 others within `reach` rows of it."""
    rng = np.random.default_rng(seed)
    ptr, idx, val = [0], [], []
    for c in range(n):
        near = np.setdiff1d(np.arange(max(0, c - reach), min(n, c + reach + 1)), [c])
        rows = np.sort(np.append(rng.choice(near, min(width - 1, len(near)), replace=False), c))
        if shuffle:
            rows = rng.permutation(rows)
        idx.append(rows)
        val.append(np.where(rows == c, 1.0 + 0.3 * width, rng.uniform(-1, 1, len(rows))))
        ptr.append(ptr[-1] + len(rows))
    return W.CSC(n, np.array(ptr, np.int32), np.concatenate(idx).astype(np.int32), np.concatenate(val))


def check(ctx, A, **opt):
    m_o, res_o, _, sing = oracle.spai(A, "householder")
    m, res, info = ctx.build_h(A, precision=N.PREC_FP64, **opt)
    assert sing == 0 and info.cols_singular == 0
    assert info.cols_small + info.cols_large == A.n
    cols = np.repeat(np.arange(A.n), np.diff(A.ptr))
    scale = np.zeros(A.n)
    np.maximum.at(scale, cols, np.abs(m_o))
    assert np.max(np.abs(m - m_o) / scale[cols]) <= RTOL
    assert np.max(np.abs(res - res_o)) <= RTOL
    return m, info


# reach = width: dense bands (|I| ~ 4 width); reach large: disjoint columns (|I| ~ width^2)
@pytest.mark.parametrize("width,reach", [(1, 1), (2, 3), (4, 4), (5, 5), (6, 6), (7, 4), (7, 7), (7, 300), (8, 5),
                                         (8, 8), (9, 6), (9, 300), (11, 7), (11, 9), (12, 8), (15, 9), (15, 17),
                                         (16, 16)])
def test_sizes(ctx, width, reach):
    check(ctx, matrix(700, width, reach, width * 31 + reach))


def test_where_columns_go(ctx):
    # 15 entries within 9 rows of the diagonal: at most 37 rows, 225 candidates, all on the groups; 16 entries: none
    _, a = check(ctx, matrix(500, 15, 9, 1))
    assert a.cols_large == 0
    _, b = check(ctx, matrix(500, 16, 16, 1))
    assert b.cols_large == 500


@pytest.mark.parametrize("width", [5, 7, 9, 13])
def test_unsorted_columns_and_schedules(ctx, width):
    A = matrix(333, width, 8, width, shuffle=True)
    m0, _ = check(ctx, A)
    m1, _ = check(ctx, A, schedule=N.SCHED_BALANCED_NNZ)
    assert np.array_equal(m0, m1)
    m2, res, info = ctx.build_h(A, col_start=101, col_end=230)
    s, e = A.ptr[101], A.ptr[230]
    assert np.array_equal(m2[s:e], m0[s:e]) and not m2[:s].any() and not m2[e:].any()
    assert info.cols_total == 129


def test_mixed_widths_share_warps(ctx):
    rng = np.random.default_rng(8)
    parts = [matrix(120, w, r, 50 + w) for w, r in ((3, 3), (7, 40), (8, 8), (14, 12), (20, 30))]
    # interleave the columns of block-diagonal parts so that a warp holds every kind
    n = sum(p.n for p in parts)
    offs = np.cumsum([0] + [p.n for p in parts])
    perm = rng.permutation(n)                       # new number of every old row / column
    cols = {}
    for p, o in zip(parts, offs):
        for c in range(p.n):
            s, e = p.ptr[c], p.ptr[c + 1]
            rows = perm[o + p.idx[s:e]]
            q = np.argsort(rows)
            cols[perm[o + c]] = (rows[q], p.val[s:e][q])
    ptr = np.concatenate([[0], np.cumsum([len(cols[c][0]) for c in range(n)])]).astype(np.int32)
    A = W.CSC(n, ptr, np.concatenate([cols[c][0] for c in range(n)]).astype(np.int32),
              np.concatenate([cols[c][1] for c in range(n)]))
    check(ctx, A)


def test_columns_of_empty_columns(ctx):
    """J columns without entries: |I| = 0, reported singular, the others unharmed."""
    n = 40
    ptr, idx, val = [0], [], []
    for c in range(n):
        if c not in (3, 4):                       # columns 3 and 4 are empty
            rows = [3] if c == 0 else [3, 4] if c == 9 else [c]
            idx += rows
            val += [2.0] * len(rows)
        ptr.append(len(idx))
    A = W.CSC(n, np.array(ptr, np.int32), np.array(idx, np.int32), np.array(val))
    # (no oracle here: it does not take |I| = 0.)  A column that holds only its diagonal: m = 1 / 2
    m, res, info = ctx.build_h(A, precision=N.PREC_FP64)
    assert info.cols_singular == 2 and info.cols_small == n
    alone = np.ones(A.nnz, bool)
    alone[A.ptr[0]:A.ptr[1]] = alone[A.ptr[9]:A.ptr[10]] = False
    assert np.all(m[alone] == 0.5) and not np.any(np.isfinite(m[~alone]))
