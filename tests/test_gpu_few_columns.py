"""The back projection's two ways over the columns, a warp for each and units of
entries, on both sides of their limit (18,944 columns), FP32 and FP16: the same sums
as numpy's in 64 bits."""
from types import SimpleNamespace

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

EACH = 148 * 16 * 8
# a column of at most 3,000 positive entries: as many roundings in a row as a lane
# has entries (94), 5 between lanes, the product, update and normalisation
RTOL = 110 * 2.0 ** -24


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n", [7, 148 * 4 * 8 + 1, EACH - 1, EACH, EACH + 1])
def test_columns_by_either_way(rlib, n, half):
    import torch

    rng = np.random.default_rng(n + half)
    lens = rng.choice([0, 1, 40, 64, 65, 300], n)
    lens[rng.integers(0, n, 3)] = 3000
    cp = np.r_[0, np.cumsum(lens)].astype(np.int64)
    m = max(int(cp[-1]), 1)  # one entry per row, so that the ratios are y / a exactly: a is a power of two
    val = np.ldexp(1.0, rng.integers(-2, 3, m)).astype(np.float16 if half else np.float32)
    y = rng.integers(1, 50, m).astype(np.float32)
    perm = rng.permutation(m)  # entry k lies in row perm[k]; a column's rows ascend
    for j in np.nonzero(lens > 1)[0]:
        perm[cp[j]:cp[j + 1]].sort()
    rowval, rowcol = np.empty_like(val), np.empty(m, np.int32)
    rowval[perm], rowcol[perm] = val, np.repeat(np.arange(n, dtype=np.int32), lens)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = SimpleNamespace(m=m, n=n, row_ptr=t(np.arange(m + 1)), col=t(rowcol), val=t(rowval), has_transpose=True,
                        col_ptr=t(cp), row_idx=t(perm.astype(np.int32)), tval=t(val), row_rank=None, hval=t(rowval),
                        htval=t(val), rscale=torch.ones(m, device="cuda"))
    want = np.zeros(n)
    np.add.at(want, np.repeat(np.arange(n), lens), y[perm].astype(np.float64))
    ctx = rlib.Context(cfg.SMALL)
    if not half:
        out = torch.empty(n, device="cuda")
        rlib.mlem_back(A, t(y / rowval), out)
        assert np.max(np.abs(out.cpu().numpy() - want) - RTOL * want) <= 0
    x = torch.ones(n, device="cuda")
    (ctx.mlem_half if half else ctx.mlem)(A, t(y), torch.ones(n, device="cuda"), x, 1)
    assert np.max(np.abs(x.cpu().numpy() - want / want.sum()) - RTOL * want / want.sum()) <= 0
