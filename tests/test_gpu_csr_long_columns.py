"""CSC -> CSR where a warp shares a column (over 64 entries) or sorts a row (17 to 64 entries)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def pattern(n, lens, symmetric, shuffled, seed=2):
    """Diagonal plus hub columns (or rows and columns) of the given lengths; rows of many lengths from the hubs' overlap."""
    rng = np.random.default_rng(seed)
    M = np.eye(n, dtype=bool)
    for i, length in enumerate(lens):
        c = (37 * i + 5) % n
        r = rng.choice(n, length, replace=False)
        M[:, c] = False
        M[r, c] = True
    for i, length in enumerate((16, 17, 31, 32, 33, 63, 64, 65)):
        r = (53 * i + 11) % n
        M[r] = False
        M[r, rng.choice(n, length, replace=False)] = True
    if symmetric:
        M |= M.T
    cols = [np.flatnonzero(M[:, c]) for c in range(n)]
    if shuffled:
        cols = [rng.permutation(c) for c in cols]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    idx = np.concatenate(cols).astype(np.int32)
    return ptr, idx, rng.standard_normal(len(idx))


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n", [401, 416, 1500])
def test_rows_are_exact(ctx, n, symmetric, shuffled):
    ptr, idx, val = pattern(n, (10, 11, 63, 64, 65, 96, 97, 400), symmetric, shuffled)
    cols = np.repeat(np.arange(n), np.diff(ptr))
    order = np.lexsort((cols, idx))
    d = [torch.from_numpy(a).cuda() for a in (ptr, idx, val)]
    rptr, ridx, rval = torch.empty_like(d[0]), torch.empty_like(d[1]), torch.empty_like(d[2])
    torch.cuda.synchronize()
    ctx.csc_to_csr_d(n, len(idx), *d, rptr, ridx, rval)
    torch.cuda.synchronize()
    assert np.array_equal(rptr.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(idx, minlength=n))]))
    assert np.array_equal(ridx.cpu().numpy(), cols[order])
    assert np.array_equal(rval.cpu().numpy(), val[order])
