"""One iteration of the three resident forms at the numbers of rows where the forward
passes change how warps come by their rows (a stride, draws of a few rows, of 16),
against numpy in 64 bits."""
from types import SimpleNamespace

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

WARPS = 148 * 40
# The ratio's dot product of 3 and its division, a column's sum in which a lane has up
# to ~150 terms of like size, 5 steps between lanes, two products, update and
# normalisation; errors of terms of both signs, so the bound is generous
RTOL = 170 * 2.0 ** -24


# (rows over 600,000 voxels and more are drawn from half as many on)
@pytest.mark.parametrize("m,n", [(WARPS * 16 - 1, 500), (WARPS * 16, 500), (WARPS * 128 - 1, 500), (WARPS * 128, 500),
                                 (WARPS * 128 + 7, 500), (WARPS * 8 - 1, 600000), (WARPS * 8, 600000),
                                 (WARPS * 8, 599999)])
def test_row_draws(rlib, m, n):
    import torch

    rng = np.random.default_rng(m)
    lens = rng.integers(1, 4, m)
    rp = np.r_[0, np.cumsum(lens)].astype(np.int64)
    row = np.repeat(np.arange(m), lens)
    first = np.repeat(rng.integers(0, n - 3, m), lens)
    col = (first + np.arange(row.size) - np.repeat(rp[:-1], lens)).astype(np.int32)  # neighbours: distinct, ascending
    val = rng.uniform(0.5, 1.0, row.size).astype(np.float16)
    y = rng.integers(0, 9, m).astype(np.float32)
    x0 = rng.uniform(0.5, 1.0, n).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = SimpleNamespace(m=m, n=n, row_ptr=t(rp), col=t(col), val=t(val.astype(np.float32)), has_transpose=True,
                        row_rank=None, hval=t(val), rscale=torch.ones(m, device="cuda"))
    A.col_ptr, A.row_idx, A.tval = rlib.csr_transpose(m, n, A.row_ptr, A.col, A.val)
    A.htval = A.tval.half()
    A.pseg, A.panchor, A.pword = rlib.pack_half(A.row_ptr, A.col, A.hval)
    A.tseg, A.tanchor, A.tword = rlib.pack_half(A.col_ptr, A.row_idx, A.htval)
    v = val.astype(np.float64)
    ax = np.bincount(row, v * x0[col], minlength=m)
    want = x0 * np.bincount(col, v * (y / ax)[row], minlength=n)
    want /= want.sum()
    ctx, s = rlib.Context(cfg.SMALL), torch.ones(n, device="cuda")
    for form in (ctx.mlem, ctx.mlem_half, ctx.mlem_packed):
        x = t(x0)
        form(A, t(y), s, x, 1)
        assert np.max(np.abs(x.cpu().numpy() - want) - RTOL * want) <= 0
