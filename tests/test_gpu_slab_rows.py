"""Rows built by the slab kernel (one thread per few slabs of the grid) at the
shapes where it can go wrong, against the oracle: structure bit-exact, values
within 1e-5 (the order in which rays are summed)."""
import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

SEED = 77


def grid(n, d=(0.002, 0.002, 0.002), shift=(0.0, 0.0, 0.0), na=16, da=22.5):
    o = tuple(-0.5 * n[k] * d[k] + shift[k] for k in range(3))
    return cfg.Geometry(grid_o=o, grid_d=d, grid_n=n, pos0x=-0.240, pos1x=0.240, na=na, n0z=13, n0y=13, n1z=13,
                        n1y=13, da=da, segx=0.020, segy=0.004, segz=0.004)


@pytest.mark.parametrize("name,g,nrays", [
    ("one slab", grid((1, 9, 1)), 50),
    ("two and three slabs", grid((2, 20, 3)), 50),
    # slabs that are no multiple of a thread's, x and z differ
    ("31 x 17 x 47", grid((31, 17, 47)), 129),
    # more z planes than three mask words hold
    ("20 x 20 x 130", grid((20, 20, 130), d=(0.002, 0.002, 0.001)), 100),
    # most slabs a row can have, and one more (hash table along that axis)
    ("256 slabs", grid((256, 12, 40), d=(0.0005, 0.002, 0.002)), 65),
    ("257 slabs", grid((257, 12, 40), d=(0.0005, 0.002, 0.002)), 65),
    # several planes of another axis inside a slab
    ("steep", grid((18, 90, 90), d=(0.005, 0.001, 0.001)), 200),
    ("flat", grid((80, 12, 12), d=(0.001, 0.006, 0.006)), 200),
    # rays that enter and leave through the sides
    ("off centre", grid((30, 30, 30), shift=(0.01, 0.015, -0.02)), 192),
    # one ray, and one more than a staged batch
    ("one ray", grid((40, 40, 40)), 1),
    ("193 rays", grid((40, 40, 40)), 193),
    # 45 degrees: as many planes of the other axis as slabs
    ("45 degrees", grid((70, 70, 70), na=8, da=45.0), 1000),
])
def test_slab_rows_match_oracle(rlib, oracle, name, g, nrays):
    rng = np.random.default_rng(3)
    lst = np.sort(rng.integers(0, g.n_channels, 150)).astype(np.int32)
    rp, col, val = rlib.Context(g, 0).build(lst, nrays, SEED).to_numpy()
    rp_o, col_o, val_o = oracle.sysmat(g, lst, nrays, SEED, method=1)
    assert np.array_equal(rp, rp_o) and np.array_equal(col, col_o)
    if val_o.size:
        assert np.max(np.abs(val - val_o) / val_o) <= 1e-5
