"""The batched iteration over more columns than a capped grid of the back pass
could take at 48 columns a warp (148 x 64 blocks x 8 warps x 48 = 3.6M): every
column against the same in FP64, for the whole columns at once and in groups of
row blocks (ratios of a tile above 96 MB)."""
from types import SimpleNamespace

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

K = 4
# Roundings of an image value, 2^-24 each: a row's dot product of up to 200
# entries (as many in a row as a lane has, 25, and 5 between lanes), the ratio's
# division, a column's two products and sum, update and normalisation (5).
RTOL = 40 * 2.0 ** -24


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("m", [100_003, 6_600_001])
def test_batch_with_millions_of_columns(rlib, m, half):
    import torch

    ctx = rlib.Context(cfg.epet_geometry(160, 0.0005, 1, 1.0))
    n = ctx.n_voxels
    assert n > 148 * 64 * 8 * 48
    rng = np.random.default_rng(m + half)
    lens = rng.integers(1, 3, n)
    cp = np.zeros(n + 1, np.int64)
    cp[1:] = np.cumsum(lens)
    col = np.repeat(np.arange(n, dtype=np.int32), lens)
    row = rng.integers(0, m, col.size).astype(np.int32)
    second = cp[1:][lens == 2] - 1  # a column's two rows ascend
    row[second - 1], row[second] = np.minimum(row[second - 1], row[second]), np.maximum(row[second - 1], row[second])
    val = rng.uniform(0.5, 1.0, col.size).astype(np.float32)
    if half:
        val = val.astype(np.float16)
    perm = np.argsort(row, kind="stable")
    rp = np.zeros(m + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(row, minlength=m))
    x0 = rng.uniform(0.5, 1.0, (n, K)).astype(np.float32)
    y = rng.integers(0, 20, (m, K)).astype(np.float32)
    s = rng.uniform(0.5, 1.0, n).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    tv, rv = t(val), t(val[perm])
    A = SimpleNamespace(m=m, n=n, row_ptr=t(rp), col=t(col[perm]), col_ptr=t(cp), row_idx=t(row), has_transpose=True,
                        row_rank=None, val=rv, tval=tv, hval=rv, htval=tv, rscale=torch.ones(m, device="cuda"))
    X = t(x0)
    ctx.mlem_batch(A, t(y), t(s), X, 1, half=half)
    got = X.cpu().numpy()
    v = val.astype(np.float64)
    for f in range(K):
        ax = np.bincount(row, v * x0[col, f], minlength=m)
        e = np.where(y[:, f] == 0, 0.0, y[:, f] / np.where(ax == 0, 1.0, ax))
        want = x0[:, f] * np.bincount(col, v * e[row], minlength=n) / s
        want /= want.sum()
        assert np.max(np.abs(got[:, f] - want) - RTOL * want) <= 0
