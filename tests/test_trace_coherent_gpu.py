"""Kernel 0 on camera rays around the rule that lets a warp trace coherent rays one thread per ray: batches
on both sides of 1,024 rays a node and of 2^20 rays, against the oracle bit for bit, and their time, which
must not be the warp traversal's (kernel 1) where the rule holds."""
import numpy as np
import pytest
import torch

from rbr_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def camera_rays(n):
    w = max(1, int(np.sqrt(n)))
    k = np.arange(n)
    d = np.stack([((k % w) / w - 0.5) * 0.7, ((k // w) / w - 0.5) * 0.7, np.full(n, -1.0)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return abi.make_rays(np.tile(np.array([[0.0, 0.5, 25.0]], np.float32), (n, 1)), d.astype(np.float32))


def world():
    return scenes.random_world(60, 400, False, seed=5, flat_triangles=4)


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("rays", ["below", "at", "million"])
def test_rule_edges_match_the_oracle(ctx, restatement, rays, any_hit):
    w = world()
    ctx.upload(w)
    nodes = ctx.stats().num_wide_nodes
    assert 64 < nodes < 512
    n = {"below": 1024 * nodes - 1, "at": 1024 * nodes, "million": (1 << 20) + 33}[rays]
    r = camera_rays(n)
    chunk = ctx.get_param("trace.host_chunk")
    ctx.set_param("trace.host_chunk", 0)
    try:
        got = ctx.trace_host(r, any_hit=any_hit)
    finally:
        ctx.set_param("trace.host_chunk", chunk)
    h = restatement.scene(w)
    if any_hit:
        assert np.array_equal(got, restatement.trace_any(h, r))
    else:
        want = restatement.trace_closest(h, r)
        assert np.array_equal(got["prim"], want["prim"])
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))


def test_coherent_rays_through_a_small_tree_are_not_warp_traversed(ctx):
    """2^18 rays through 109 nodes: 34 us one thread per ray, 47 by warp traversal."""
    ctx.upload(world())
    n = 1 << 18
    r = camera_rays(n)
    dev = torch.from_numpy(np.frombuffer(r.tobytes(), np.uint8).copy()).cuda()
    out = torch.zeros(n * 8, dtype=torch.uint8, device="cuda")
    best = {}
    for _ in range(5):
        for kernel in (0, 1):
            ctx.set_param("trace.kernel", kernel)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ctx.trace_closest_dev(dev.data_ptr(), n, out.data_ptr())
            a.record()
            for _ in range(8):
                ctx.trace_closest_dev(dev.data_ptr(), n, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
            b.record()
            b.synchronize()
            best[kernel] = min(best.get(kernel, 1e9), a.elapsed_time(b))
    ctx.set_param("trace.kernel", 0)
    assert best[0] < 0.9 * best[1]
