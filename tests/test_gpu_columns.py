"""The column loop of the back projections at column lengths around its steps
(empty columns, four short ones at a time, whole and partial 16-byte groups,
long ones), against the same in FP64."""
from types import SimpleNamespace

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 66, 67, 127, 128, 129, 255, 256, 257, 511, 512, 513, 640, 3000]


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n,m", [(1, 4000), (33, 4000), (1000, 4000), (70001, 60001)])
def test_back_projection_by_columns(rlib, n, m, half):
    import torch

    rng = np.random.default_rng(n + half)
    lens = rng.choice(LENGTHS, n, p=None if n < 2000 else np.r_[[0.6], np.full(len(LENGTHS) - 1, 0.4 / 24)])
    lens[0] = 3000 if n == 1 else lens[0]
    cp = np.zeros(n + 1, np.int64)
    cp[1:] = np.cumsum(lens)
    # row 0 has no entries but a count: its ratio is infinite and no column's
    row = rng.integers(1, m, cp[-1]).astype(np.int32)
    val = rng.random(cp[-1]).astype(np.float32)
    order = np.lexsort((np.arange(row.size), row))
    col = np.repeat(np.arange(n), lens).astype(np.int32)[order]
    rp = np.zeros(m + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(row, minlength=m))
    y = rng.poisson(5.0, m).astype(np.float32)
    y[0] = 1.0
    s = rng.random(n).astype(np.float32)
    s[rng.random(n) < 0.1] = 0.0
    x0 = rng.random(n).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = SimpleNamespace(m=m, n=n, row_ptr=t(rp), col=t(col), val=t(val[order]), has_transpose=True, col_ptr=t(cp),
                        row_idx=t(row), tval=t(val), row_rank=None, hval=t(val[order].astype(np.float16)),
                        rscale=torch.ones(m, device="cuda"), htval=t(val.astype(np.float16)))
    v64 = (val.astype(np.float16) if half else val).astype(np.float64)
    ax = np.zeros(m)
    np.add.at(ax, row, v64 * np.repeat(x0.astype(np.float64), lens))
    with np.errstate(divide="ignore", invalid="ignore"):
        e = np.where(y == 0, 0.0, y / ax)
    c = np.zeros(n)
    np.add.at(c, np.repeat(np.arange(n), lens), v64 * e[row])
    if not half:
        e32 = t(e.astype(np.float32))
        out = torch.empty(n, device="cuda")
        rlib.mlem_back(A, e32, out)
        assert np.max(np.abs(out.cpu().numpy() - c) / np.maximum(c, 1e-30) * (c > 0)) <= 1e-5
        assert np.all(out.cpu().numpy()[lens == 0] == 0)
    x = t(x0)
    ctx = rlib.Context(cfg.SMALL)
    (ctx.mlem_half if half else ctx.mlem)(A, t(y), t(s), x, 1)
    want = x0 * c / (s + (s == 0))
    want /= want.sum()
    assert np.max(np.abs(x.cpu().numpy() - want)) <= 1e-5 * want.max()
    assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-5 * np.linalg.norm(want)
