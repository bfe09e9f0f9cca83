"""Ray queries beside one another on several streams: launches that claim their rays from a cursor of
the context's ring while many later calls go round the ring, and calls captured into a graph that is
replayed beside others. Every answer equals that of the same call alone."""
import numpy as np
import pytest
import torch

from rbr_b200 import scenes

pytestmark = pytest.mark.gpu

RING = 64


class Query:
    def __init__(self, ctx, rays, any_hit):
        self.ctx, self.n, self.any_hit = ctx, len(rays), any_hit
        self.rays = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
        self.out = torch.zeros(self.n * (1 if any_hit else 8), dtype=torch.uint8, device="cuda")
        self.run(torch.cuda.current_stream())
        torch.cuda.synchronize()
        self.want = self.out.clone()
        self.out.fill_(0xAA)
        torch.cuda.synchronize()

    def run(self, stream):
        f = self.ctx.trace_any_dev if self.any_hit else self.ctx.trace_closest_dev
        f(self.rays.data_ptr(), self.n, self.out.data_ptr(), stream.cuda_stream)


# kernel 2's first runs end at 4 rays a warp, the others' at 32: each size is past its kernel's
@pytest.mark.parametrize("kernel,small", [(0, 400_003), (1, 400_003), (2, 60_001)])
@pytest.mark.parametrize("any_hit", [False, True])
def test_calls_on_two_streams(ctx, kernel, small, any_hit):
    ctx.upload(scenes.random_world(60, 300, True, seed=5, flat_triangles=4))
    ctx.set_param("trace.kernel", kernel)
    try:
        pool = scenes.random_test_rays(1_000_000, seed=9)
        long = Query(ctx, np.resize(pool, 6_000_001), any_hit)
        short = [Query(ctx, pool[k:k + small + k], any_hit) for k in (0, 1, 2)]
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        long.run(a)
        for i in range(RING + 2):
            short[i % 3].run(b)
        torch.cuda.synchronize()
    finally:
        ctx.set_param("trace.kernel", 0)
    for q in [long, *short]:
        assert torch.equal(q.out, q.want)


@pytest.mark.parametrize("kernel", [0, 1, 2])
@pytest.mark.parametrize("n", [60_001, 700_001])
def test_captured_call_beside_others(ctx, kernel, n):
    ctx.upload(scenes.random_world(60, 300, True, seed=6, flat_triangles=4))
    ctx.set_param("trace.kernel", kernel)
    try:
        pool = scenes.random_test_rays(1_000_000, seed=10)
        captured, other = Query(ctx, pool[:n], False), Query(ctx, pool[7:500_010], False)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured.run(torch.cuda.current_stream())
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        for _ in range(2):
            for _ in range(RING + 2):
                graph.replay()
                other.run(side)
        torch.cuda.synchronize()
    finally:
        ctx.set_param("trace.kernel", 0)
    assert torch.equal(captured.out, captured.want) and torch.equal(other.out, other.want)
