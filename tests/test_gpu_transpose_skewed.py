"""CSR -> CSC of rows with ascending columns whose entries crowd into few bins (a
piece of the partition is then shared by several warps) or into few long rows.
Exact against numpy: nothing is computed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# pieces of 256 rows (16 warps each), the last of them 5; of 64 rows (4 warps); of a
# few entries above a warp's share; few long rows, one and 9 of a block's eight warps
@pytest.mark.parametrize("m,n,per_row,spread", [(2565, 1 << 20, 1100, 1100), (1001, 2048, 2000, 2048),
                                                 (129, 3000, 300, 320), (64, 200000, 40000, 60000),
                                                 (1, 70000, 65535, 70000), (9, 70000, 30000, 70000)])
def test_skewed_rows(rlib, m, n, per_row, spread):
    import torch

    rng = np.random.default_rng(m)
    lens = rng.integers(max(per_row - 9, 1), per_row + 1, m)
    lens[m // 2] = 0 if m > 1 else per_row
    if n // 1024 * m > lens.sum():
        lens[lens > 0] = per_row
    start = rng.integers(0, n - spread + 1, m) if spread < n and m < 2565 else np.zeros(m, np.int64)
    col = np.concatenate([s + np.sort(rng.choice(spread, k, replace=False)) for s, k in zip(start, lens)]).astype(np.int32)
    rp = np.r_[0, np.cumsum(lens)].astype(np.int64)
    val = rng.standard_normal(col.size).astype(np.float32)
    order = rng.permutation(m).astype(np.int32)
    rank = np.empty(m, np.int64)
    rank[order] = np.arange(m)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    got = rlib.csr_transpose_ordered(m, n, t(rp), t(col), t(val), t(order))
    k = rank[np.repeat(np.arange(m), lens)]
    o = np.lexsort((k, col))
    assert np.array_equal(got[0].cpu().numpy(), np.r_[0, np.cumsum(np.bincount(col, minlength=n))])
    assert np.array_equal(got[1].cpu().numpy(), k[o])
    assert np.array_equal(got[2].cpu().numpy().view(np.uint32), val[o].view(np.uint32))
