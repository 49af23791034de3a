"""The batched iteration where the library's memory is capped: 64 frames at the
default tile in the memory that two tiles of 32 need, and in narrower tiles where
the widest does not fit.  The image is that of the uncapped call."""
import os
import subprocess
import sys

import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
K = 64
RTOL = 1e-5  # other tiles and groups of rows sum in another order


def run(rlib, m):
    from types import SimpleNamespace

    import torch

    g = cfg.FULL
    ctx = rlib.Context(g, 0)
    n = ctx.n_voxels
    rng = np.random.default_rng(m)
    lens = np.full(m, 3)
    rp = np.r_[0, np.cumsum(lens)].astype(np.int64)
    col = (np.repeat(rng.integers(0, n - 3, m), lens) + np.tile(np.arange(3), m)).astype(np.int32)
    row = np.repeat(np.arange(m, dtype=np.int32), lens)
    val = rng.uniform(0.5, 1.0, col.size).astype(np.float32)
    o = np.argsort(col, kind="stable")
    cp = np.r_[0, np.cumsum(np.bincount(col, minlength=n))].astype(np.int64)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = SimpleNamespace(m=m, n=n, row_ptr=t(rp), col=t(col), val=t(val), col_ptr=t(cp), row_idx=t(row[o]), tval=t(val[o]),
                        has_transpose=True, row_rank=None)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m)
    Y = torch.randint(0, 9, (m, K), device="cuda", generator=gen).float()
    X = torch.rand((n, K), device="cuda", generator=gen) + 0.5
    ctx.mlem_batch(A, Y, torch.ones(n, device="cuda"), X, 2, half=False)
    return X.cpu().numpy()


# rows, cap (MiB).  100 rows: the images' buffer (88 MB) and the list of columns; without
# them, tiles of 32 once took 168 MiB.  400,000 rows: ratios (102 MB), images, partial
# sums (88 MB in one tile, 22 + 22 with a compact copy in tiles of 16), row blocks (23)
@pytest.mark.parametrize("m,cap_mb", [(100, 177), (400_000, 260)])
def test_capped(rlib, tmp_path, m, cap_mb):
    out = str(tmp_path / "x.npy")
    env = dict(os.environ, RAPTR_DEVICE_MEMORY_LIMIT=str(cap_mb << 20), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), str(m), out], cwd=ROOT, capture_output=True,
                       text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    want, got = run(rlib, m), np.load(out)
    assert np.linalg.norm(got - want) <= RTOL * np.linalg.norm(want)


if __name__ == "__main__":
    import raptr_b200

    np.save(sys.argv[2], run(raptr_b200, int(sys.argv[1])))
