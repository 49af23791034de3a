"""The scatter passes over rows by their entries at the edges of the way that short
rows take (at most 64 entries), against numpy in 64 bits."""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a column's sum of up to ~120 positive terms in any order, a row's dot product of up
# to 300 entries, the division and two products
RTOL = 140 * 2.0 ** -24


@pytest.mark.parametrize("m", [1, 40, 20011])
def test_scatter_passes(rlib, m):
    import torch

    rng = np.random.default_rng(m)
    n = 40 * m + 500
    lens = rng.choice([0, 1, 2, 31, 32, 33, 63, 64, 65, 66, 300], m)
    lens[0] = 64
    rp = np.r_[0, np.cumsum(lens)].astype(np.int64)
    row = np.repeat(np.arange(m), lens)
    col = np.concatenate([np.sort(rng.choice(500, k, replace=False)) for k in lens]) + 40 * row  # bands of rows overlap
    val = rng.uniform(0.5, 1.0, col.size).astype(np.float32)
    x, y = rng.uniform(0.5, 1.0, n).astype(np.float32), rng.integers(0, 9, m).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = SimpleNamespace(m=m, n=n, row_ptr=t(rp), col=t(col.astype(np.int32)), val=t(val))
    got = rlib.spmv(rlib.OP_T, m, n, A.row_ptr, A.col, A.val, t(y)).cpu().numpy()
    want = np.bincount(col, val * y.astype(np.float64)[row], minlength=n)
    assert np.max(np.abs(got - want) - RTOL * want) <= 0
    c, ll = torch.zeros(n, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
    rlib.mlem_project(A, t(y), t(x), c, ll=ll)
    ax = np.bincount(row, val * x.astype(np.float64)[col], minlength=m)
    on = (y != 0) & (lens > 0)
    e = np.where(on, y / np.where(on, ax, 1.0), 0.0)
    want = np.bincount(col, val * e[row], minlength=n)
    assert np.max(np.abs(c.cpu().numpy() - want) - RTOL * want) <= 0
    if not np.any((y != 0) & (lens == 0)):  # (log 0)
        assert np.allclose(ll.cpu().numpy(), [np.sum(y[on] * np.log(ax[on])), np.sum(ax[on])], rtol=1e-6)
