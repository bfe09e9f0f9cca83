"""Batches of one and a quarter to one and three quarters of the resident warps' first runs, whose second runs
are dealt out by index without a cursor: the rule's edges against the oracle bit for bit, plain and captured,
and the launch's shape."""
import numpy as np
import pytest
import torch

from rbr_b200 import scenes

pytestmark = pytest.mark.gpu

RESIDENT = 148 * 8 * 128
EDGES = [RESIDENT + RESIDENT // 4 + k for k in (-1, 0, 33)] + [RESIDENT + RESIDENT // 4 * 3 + k for k in (-1, 0, 1)]


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("kernel,order", [(0, 0), (1, 0), (1, 5)])
@pytest.mark.parametrize("n", EDGES)
def test_edges_match_the_oracle(ctx, restatement, kernel, order, n, any_hit):
    w = scenes.random_world(60, 400, True, seed=5, flat_triangles=4)
    ctx.upload(w)
    assert ctx.stats().num_wide_nodes > 64
    rays = scenes.random_test_rays(2 * n, seed=n)[:n]
    dev = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
    outs = [torch.full((n * (1 if any_hit else 8),), 0xAA, dtype=torch.uint8, device="cuda") for _ in range(2)]
    call = ctx.trace_any_dev if any_hit else ctx.trace_closest_dev
    ctx.set_param("trace.kernel", kernel)
    ctx.set_param("trace.order", order)
    try:
        call(dev.data_ptr(), n, outs[0].data_ptr())
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(dev.data_ptr(), n, outs[1].data_ptr(), torch.cuda.current_stream().cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        ctx.set_param("trace.kernel", 0)
        ctx.set_param("trace.order", 0)
    assert torch.equal(outs[0], outs[1])
    h = restatement.scene(w)
    got = outs[0].cpu().numpy()
    if any_hit:
        assert np.array_equal(got, restatement.trace_any(h, rays))
    else:
        want = restatement.trace_closest(h, rays)
        assert np.array_equal(got.view(np.uint32)[0::2], want["prim"].view(np.uint32))
        assert np.array_equal(got.view(np.uint32)[1::2], want["t"].view(np.uint32))


def test_second_runs_take_the_resident_grid(ctx):
    driver = pytest.importorskip("cuda.bindings.driver")
    ctx.upload(scenes.random_world(60, 400, True, seed=5, flat_triangles=4))
    n = RESIDENT + RESIDENT // 2
    rays = scenes.random_test_rays(2 * n, seed=3)[:n]
    dev = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
    out = torch.zeros(n * 8, dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        ctx.trace_closest_dev(dev.data_ptr(), n, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    g = driver.CUgraph(graph.raw_cuda_graph())
    _, nodes, _ = driver.cuGraphGetNodes(g, 8)
    params = [driver.cuGraphKernelNodeGetParams(x)[1] for x in nodes[:1]]
    assert len(params) == 1 and params[0].gridDimX == RESIDENT // 128
