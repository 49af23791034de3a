"""CSR -> CSC of rows with ascending columns (partition by bins of 1024 columns)
at the edges of bins, blocks of rows, windows and tiles, and the matrices that it
has to leave to the radix sort.  Exact against numpy: nothing is computed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def csr(rng, m, n, per_row, whole_bin):
    rows = []
    for k in range(m):
        if k % 7 == 3:
            c = np.zeros(0, np.int32)  # no entries
        elif whole_bin and k % 5 == 0:  # all columns of the first bin and of the last
            c = np.r_[np.arange(min(1024, n)), np.arange((n - 1) // 1024 * 1024, n)]
            c = np.unique(c)
        else:
            c = np.sort(rng.choice(n, min(per_row, n), replace=False))
        rows.append(c.astype(np.int32))
    rp = np.r_[0, np.cumsum([len(c) for c in rows])].astype(np.int64)
    col = np.concatenate(rows)
    return rp, col, rng.standard_normal(len(col)).astype(np.float32)


def check(rlib, torch, m, n, rp, col, val, rng):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    row = np.repeat(np.arange(m), np.diff(rp))
    for order in (None, rng.permutation(m).astype(np.int32)):
        if order is None:
            rank = np.arange(m)
            got = rlib.csr_transpose(m, n, t(rp), t(col), t(val))
        else:
            rank = np.empty(m, np.int64)
            rank[order] = np.arange(m)
            got = rlib.csr_transpose_ordered(m, n, t(rp), t(col), t(val), t(order))
        k = rank[row]
        o = np.lexsort((k, col))
        cp = np.r_[0, np.cumsum(np.bincount(col, minlength=n))]
        assert np.array_equal(got[0].cpu().numpy(), cp)
        assert np.array_equal(got[1].cpu().numpy(), k[o])
        assert np.array_equal(got[2].cpu().numpy().view(np.uint32), val[o].view(np.uint32))


# two bins (the second of one column, of all but one, whole); one row and the
# edges of a window of 32 and a block of 1024 rows; bins of several tiles; as many
# bins as there may be, and one more (the radix sort)
@pytest.mark.parametrize("m,n,per_row,whole_bin",
                         [(1, 1025, 1025, False), (32, 2047, 40, True), (33, 2048, 3, True), (1025, 2049, 900, True),
                          (129, 70001, 300, True), (2, 1 << 20, 5000, True), (2, (1 << 20) + 1, 5000, True),
                          (1, 100000, 65535, False), (1, 100000, 65536, False)])
def test_sorted_rows(rlib, torch, m, n, per_row, whole_bin):
    rng = np.random.default_rng(m + n)
    check(rlib, torch, m, n, *csr(rng, m, n, per_row, whole_bin), rng)


@pytest.mark.parametrize("what", ["descending", "equal"])
def test_rows_that_do_not_ascend(rlib, torch, what):
    rng = np.random.default_rng(5)
    m, n = 300, 5000
    rp, col, val = csr(rng, m, n, 100, False)
    e = rp[m - 1]  # the last row's first two entries
    assert rp[m] - e >= 2
    if what == "descending":
        col[e], col[e + 1] = col[e + 1], col[e]
    else:
        col[e + 1] = col[e]
    check(rlib, torch, m, n, rp, col, val, rng)


def test_bad_column_and_order(rlib, torch):
    rng = np.random.default_rng(6)
    m, n = 300, 5000
    rp, col, val = csr(rng, m, n, 100, False)
    t = lambda a: torch.from_numpy(a).cuda()
    for bad in (n, -1, -5000, 2**31 - 1):
        c = col.copy()
        c[rp[m - 1]] = bad
        with pytest.raises(Exception, match="out of range"):
            rlib.csr_transpose(m, n, t(rp), t(c), t(val))
    order = np.arange(m, dtype=np.int32)
    order[-1] = m
    with pytest.raises(Exception, match="out of range"):
        rlib.csr_transpose_ordered(m, n, t(rp), t(col), t(val), t(order))
