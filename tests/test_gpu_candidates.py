"""The candidate search's row intervals at the grids and lines where they can go
wrong, against the oracle's test of every voxel: candidates and counts
bit-exact."""
import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu


def grid(n, d=(0.002, 0.002, 0.002), shift=(0.0, 0.0, 0.0), na=8, da=45.0):
    o = tuple(-0.5 * n[k] * d[k] + shift[k] for k in range(3))
    return cfg.Geometry(grid_o=o, grid_d=d, grid_n=n, pos0x=-0.240, pos1x=0.240, na=na, n0z=13, n0y=13, n1z=13,
                        n1y=13, da=da, segx=0.020, segy=0.004, segz=0.004)


@pytest.mark.parametrize("name,g", [
    ("one row", grid((1, 1, 50))),
    ("one column", grid((50, 1, 1))),
    # more slabs, and more rows of the cylinder, than the block has threads
    ("300 slabs", grid((300, 30, 20), d=(0.0005, 0.002, 0.002))),
    ("fine rows", grid((20, 200, 20), d=(0.002, 0.0005, 0.002))),
    # long rows: a step's candidates do not fit the stage
    ("400 along z", grid((24, 24, 400), d=(0.002, 0.002, 0.0004))),
    ("off centre", grid((40, 40, 40), shift=(0.05, -0.03, 0.04))),
    ("coarse", grid((12, 12, 12), d=(0.012, 0.009, 0.011))),
])
def test_candidates_match_oracle(rlib, oracle, name, g):
    rng = np.random.default_rng(7)
    per = 13 ** 4
    same = [v * per + (6 * 13 + 6) * 170 for v in range(g.na)]  # both crystals in the middle: lines along x, z, 45 degrees
    lst = np.sort(np.r_[rng.integers(0, g.n_channels, 40), same]).astype(np.int32)
    ctx = rlib.Context(g)
    co, vo, cur = oracle.workqueue(g, lst)
    c, v, cur_g = ctx.workqueue(lst, max_out=co.size + 10)
    assert np.array_equal(c.cpu().numpy(), co) and np.array_equal(v.cpu().numpy(), vo) and cur_g == cur
    assert int(ctx.candidate_counts(lst).sum().item()) == co.size
    # in chunks, from cursors inside rows
    done, cur = 0, (0, 0)
    step = max(1, co.size // 3 + 1)
    while done < co.size:
        c, v, cur = ctx.workqueue(lst, cursor=cur, max_out=step)
        assert np.array_equal(v.cpu().numpy(), vo[done:done + step])
        done += c.numel()
        if c.numel() == 0:
            break
    assert done == co.size
