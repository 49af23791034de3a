"""The FP16 back projection's sums over short columns (taken four at a time) are
compensated: columns of large counts that cancel and small ones that remain, in
which plain FP32 sums lose 2^-12 of the large ones."""
from types import SimpleNamespace

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

# The column's sum (one rounding; the compensation's own, 64 * 2^-48 of the sum of
# magnitudes, stay below 2^-26), the normalisation's scale and its product.
RTOL = 4 * 2.0 ** -24


def test_short_columns_are_compensated(rlib):
    import torch

    rng = np.random.default_rng(5)
    n = 6400
    lens = np.tile(np.arange(1, 65), n // 64)
    rng.shuffle(lens)
    cp = np.zeros(n + 1, np.int64)
    cp[1:] = np.cumsum(lens)
    m = int(cp[-1])  # one entry per row: its ratio is y / h, exact for h a power of two
    y = rng.uniform(0.5, 1.0, m).astype(np.float32)
    for j in range(n):
        k = rng.permutation(lens[j])
        pairs = max(int(lens[j]) // 2 - 2, 0)
        big = rng.uniform(2.0 ** 11, 2.0 ** 12, pairs).astype(np.float32)
        y[cp[j] + k[:pairs]] = big
        y[cp[j] + k[pairs:2 * pairs]] = -big
    h = np.ldexp(1.0, rng.integers(-4, 5, m)).astype(np.float16)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    col = np.repeat(np.arange(n, dtype=np.int32), lens)
    A = SimpleNamespace(m=m, n=n, row_ptr=t(np.arange(m + 1)), col=t(col), has_transpose=True, col_ptr=t(cp),
                        row_idx=t(np.arange(m, dtype=np.int32)), row_rank=None, hval=t(h), htval=t(h),
                        rscale=torch.ones(m, device="cuda"))
    x = torch.ones(n, device="cuda")
    rlib.Context(cfg.SMALL).mlem_half(A, t(y), torch.ones(n, device="cuda"), x, 1)
    want = np.add.reduceat(y.astype(np.float64), cp[:-1])
    want /= want.sum()
    assert np.max(np.abs(x.cpu().numpy() - want) / want) <= RTOL
