"""An iteration of a served batch launches its passes and nothing that could be
done once per matrix: beside batches of large geometries every launch waits for its
turn."""
import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu


def test_launches_of_a_served_iteration(rlib):
    g = cfg.epet_geometry(30, 0.002, 4, 45.0)
    srv = rlib.Server(0, hbm_budget_bytes=4 << 30)
    y = np.random.default_rng(1).poisson(3.0, g.n_channels).astype(np.float32)

    def launches(n_iter):
        before = rlib.kernel_launches()
        x, _ = srv.wait(srv.submit(g, y, n_iter, 50, 7), g.n_voxels)
        assert np.isfinite(x).all() and abs(float(x.sum()) - 1.0) < 1e-5
        return rlib.kernel_launches() - before

    launches(2)  # builds the matrix
    few, many = launches(10), launches(60)
    srv.close()
    assert many - few == 50 * 3  # forward, back, normalisation


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_columns_without_entries(rlib, half, bad):
    """Columns no row sees become 0, or make the image's sum what an infinite or
    undefined start value there makes it (each frame by itself)."""
    import torch

    g, K = cfg.epet_geometry(24, 0.002, 3, 60.0), 12
    ctx = rlib.Context(g, 0)
    A = ctx.build(np.arange(0, 200, dtype=np.int32), 50, 7)
    A.to_half()
    seen = (A.col_ptr[1:] > A.col_ptr[:-1]).cpu().numpy()
    assert 0 < seen.sum() < seen.size
    rng = np.random.default_rng(2)
    y = rng.integers(1, 9, (A.m, K)).astype(np.float32)
    x0 = rng.uniform(0.5, 1.0, (A.n, K)).astype(np.float32)
    x0[np.nonzero(~seen)[0][3], 5] = bad
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X, s = t(x0), torch.full((A.n,), 1.0, device="cuda")
    ctx.mlem_batch(A, t(y), s, X, 1, frame_tile=8, half=half)
    X = X.cpu().numpy()
    others = np.delete(np.arange(K), 5)
    assert np.all(X[~seen][:, others] == 0)
    assert np.all(X[seen][:, others] > 0) and np.allclose(X[:, others].sum(0), 1.0, atol=1e-5)
    assert np.isnan(X[:, 5]).all()
