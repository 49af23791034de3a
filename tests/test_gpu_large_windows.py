"""Rows of crystals that cover many voxels: windows too large for sums of each
thread's own are walked into shared ones, not into the hash table (the build's
trace counts those rows), against the oracle: structure bit-exact, values within
1e-5 (the order in which rays are summed)."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

SEED = 78
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def grid(n, pitch, seg):
    o = tuple(-0.5 * v * pitch for v in n)
    return cfg.Geometry(grid_o=o, grid_d=(pitch,) * 3, grid_n=n, pos0x=-0.240, pos1x=0.240, na=16, n0z=5, n0y=3,
                        n1z=4, n1y=5, da=22.5, segx=0.020, segy=seg, segz=seg)


CASES = {
    # by rows' most entries: 2048, 4096, 8192
    "12 mm on 2 mm": (grid((40, 40, 40), 0.002, 0.012), 100),
    "10 mm on 2 mm": (grid((70, 70, 70), 0.002, 0.010), 200),
    "9 mm on 1.5 mm": (grid((100, 90, 100), 0.0015, 0.009), 150),
    # z slabs whose masks do not fit behind the sums
    "5 mm on 1 mm, 130 planes": (grid((60, 60, 130), 0.001, 0.005), 128),
}


# rows that overflow the tables of two levels: their chunk is built again
OVERFLOW = "20 mm on 2 mm"
CASES_ALL = dict(CASES, **{OVERFLOW: (grid((70, 70, 70), 0.002, 0.020), 300)})


def channels(g, rows=60):
    return np.sort(np.random.default_rng(4).integers(0, g.n_channels, rows)).astype(np.int32)


def build(name, rows, tmp_path):
    out = str(tmp_path / "rows.npz")
    r = subprocess.run([sys.executable, os.path.abspath(__file__), name, str(rows), out], cwd=ROOT,
                       capture_output=True, text=True, env=dict(os.environ, RAPTR_TRACE="1", PYTHONPATH=ROOT),
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    by_table = re.findall(r"(\d+) with windows over the slot limit, (\d+) with a ray outside", r.stderr)
    assert len(by_table) == 1
    return np.load(out), int(by_table[0][0]), int(by_table[0][1])


@pytest.mark.parametrize("name", CASES)
def test_large_windows(rlib, oracle, tmp_path, name):
    g, nrays = CASES[name]
    got, over_limit, outside = build(name, 60, tmp_path)
    assert (over_limit, outside) == (0, 0)
    rp, col, val = oracle.sysmat(g, channels(g), nrays, SEED, method=1)
    assert np.array_equal(got["rp"], rp) and np.array_equal(got["col"], col)
    assert np.max(np.abs(got["val"] - val) / val) <= 1e-5


def test_an_overflow_ends_its_level(rlib, oracle, tmp_path):
    """Once a row has overflowed its level's table, the level's other rows are not
    tried (each block of the table kernel, of which there are 592, ends the row it
    is at)."""
    g, nrays = CASES_ALL[OVERFLOW]
    rows = 3000
    got, over_limit, _ = build(OVERFLOW, rows, tmp_path)
    assert over_limit < rows
    pick = np.linspace(0, rows - 1, 25).astype(int)
    lst = channels(g, rows)[pick]
    rp, col, val = oracle.sysmat(g, lst, nrays, SEED, method=1)
    assert np.max(np.diff(rp)) > 4096
    for k, i in enumerate(pick):
        sl, so = slice(got["rp"][i], got["rp"][i + 1]), slice(rp[k], rp[k + 1])
        assert np.array_equal(got["col"][sl], col[so])
        assert np.max(np.abs(got["val"][sl] - val[so]) / val[so]) <= 1e-5


if __name__ == "__main__":
    import raptr_b200

    g, nrays = CASES_ALL[sys.argv[1]]
    rp, col, val = raptr_b200.Context(g, 0).build(channels(g, int(sys.argv[2])), nrays, SEED).to_numpy()
    np.savez(sys.argv[3], rp=rp, col=col, val=val)
