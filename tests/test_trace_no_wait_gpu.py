"""Ray queries on one stream never wait for another stream's: with a long wait and a query queued behind it
on stream a, more queries than the context has claim cursors finish on stream b first, with right answers."""
import numpy as np
import pytest
import torch

from rbr_b200 import Context, scenes

pytestmark = pytest.mark.gpu

RING = 64
CYCLES = 2_000_000_000  # of the wait on stream a: a second, and ends by itself


@pytest.mark.parametrize("kernel,n", [(0, 400_003), (1, 400_003), (2, 60_001)])
@pytest.mark.parametrize("any_hit", [False, True])
def test_queries_do_not_wait_for_another_stream(kernel, n, any_hit):
    with Context(0) as ctx:
        ctx.upload(scenes.random_world(400, 1500, False, seed=5))
        ctx.set_param("trace.kernel", kernel)
        rays = scenes.random_test_rays(2 * n, seed=9)[:n]
        dev = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
        call = ctx.trace_any_dev if any_hit else ctx.trace_closest_dev
        outs = [torch.zeros(n * (1 if any_hit else 8), dtype=torch.uint8, device="cuda") for _ in range(3)]
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        call(dev.data_ptr(), n, outs[0].data_ptr())
        call(dev.data_ptr(), n, outs[1].data_ptr(), b.cuda_stream)
        graph = torch.cuda.CUDAGraph()  # loads the kernel that calls without a cursor run (a load may wait for the GPU)
        with torch.cuda.graph(graph):
            call(dev.data_ptr(), n, outs[2].data_ptr(), torch.cuda.current_stream().cuda_stream)
        graph.replay()
        outs[1].zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            torch.cuda._sleep(CYCLES)
        call(dev.data_ptr(), n, outs[2].data_ptr(), a.cuda_stream)
        last = torch.cuda.Event()
        last.record(a)
        for _ in range(RING + 2):
            call(dev.data_ptr(), n, outs[1].data_ptr(), b.cuda_stream)
        b.synchronize()
        waited = last.query()
        torch.cuda.synchronize()
        assert not waited
        assert torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])
