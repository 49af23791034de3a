"""The iterations as launches of the caller's stream: queued on a stream of its own
without a wait, and captured by the caller in a CUDA graph, they give the image of a
call that waits."""
import numpy as np
import pytest

from raptr_b200 import config as cfg

pytestmark = pytest.mark.gpu

RTOL = 1e-6  # the order in which blocks add the image's sum


@pytest.mark.parametrize("form", ["gather", "half", "batch"])
def test_queued_and_captured_iterations(rlib, form):
    import torch

    g = cfg.epet_geometry(30, 0.002, 4, 45.0)
    ctx = rlib.Context(g, 0)
    A = ctx.build(np.arange(g.n_channels, dtype=np.int32), 50, 7)
    A.to_half()
    K = 8 if form == "batch" else 1
    rng = np.random.default_rng(3)
    y = torch.from_numpy(rng.poisson(3.0, (A.m, K)).astype(np.float32)).cuda()
    s = rlib.sensitivity(A)[1]
    x0 = torch.full((A.n, K), 1.0 / A.n, device="cuda")
    if form != "batch":
        y, x0 = y[:, 0].contiguous(), x0[:, 0].contiguous()

    def run(x, **kw):
        {"gather": ctx.mlem, "half": ctx.mlem_half, "batch": ctx.mlem_batch}[form](A, y, s, x, 4, **kw)

    want = x0.clone()
    run(want, use_graph=True)
    rel = lambda x: float((x - want).norm() / want.norm())

    side = torch.cuda.Stream()
    x = x0.clone()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run(x, use_graph=False)
        after = x + 0.0  # ordered after the iterations
    torch.cuda.current_stream().wait_stream(side)
    assert rel(after) <= RTOL

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        run(x, use_graph=False)
    for _ in range(2):
        x.copy_(x0)
        graph.replay()
        assert rel(x) <= RTOL
