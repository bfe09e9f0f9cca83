"""The persistent ray-query kernel where it can go wrong, against the oracle bit for bit: batches
around its 32-ray runs, its blocks and the resident warps' first runs (the cursor takes over after
them), coherent and incoherent rays on both sides of the rule that chooses between them, planes (rays
finished before they start), and nodes of many records (more than one window of the record queue)."""
import numpy as np
import pytest

from rbr_b200 import abi, scenes

pytestmark = pytest.mark.gpu

RESIDENT = 148 * 8 * 128  # rays of the first runs at 8 blocks per SM


def camera_rays(n):
    """A fan of nearly parallel rays from one point, in scanline order."""
    w = max(1, int(np.sqrt(n)))
    k = np.arange(n)
    d = np.stack([(k % w) / w - 0.5, (k // w) / w - 0.5, np.full(n, -1.5)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return abi.make_rays(np.tile(np.array([[0.3, 0.2, 13.5]], np.float32), (n, 1)), d.astype(np.float32))


def check(ctx, restatement, world, rays, kernel, refill=1):
    ctx.upload(world)
    h = restatement.scene(world)
    ctx.set_param("trace.kernel", kernel)
    ctx.set_param("trace.refill_min", refill)
    try:
        got, occ = ctx.trace_host(rays), ctx.trace_host(rays, any_hit=True)
    finally:
        ctx.set_param("trace.kernel", 0)
        ctx.set_param("trace.refill_min", 1)
    want = restatement.trace_closest(h, rays)
    assert np.array_equal(got["prim"], want["prim"])
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
    assert np.array_equal(occ, restatement.trace_any(h, rays))


@pytest.mark.parametrize("kernel,refill", [(0, 1), (1, 1), (1, 32)])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, RESIDENT - 1, RESIDENT + 1, RESIDENT + 4097])
@pytest.mark.parametrize("coherent", [False, True])
def test_batch_edges(ctx, restatement, kernel, refill, n, coherent):
    # one chunk per call, so that the batch sizes are the kernel's
    chunk = ctx.get_param("trace.host_chunk")
    ctx.set_param("trace.host_chunk", 0)
    try:
        w = scenes.random_world(6, 8, True, seed=3, flat_triangles=4)
        rays = camera_rays(n) if coherent else scenes.random_test_rays(2 * n + 16, seed=n)[:n]
        check(ctx, restatement, w, rays, kernel, refill)
    finally:
        ctx.set_param("trace.host_chunk", chunk)


def test_nodes_of_many_records(ctx, restatement):
    """A pile of coincident small triangles: leaf-only nodes of up to 32 records, all hit by every
    ray of a warp, so a step queues up to 1,024 records (16 windows)."""
    w = scenes.Scene()
    m = w.diffuse((0.5, 0.5, 0.5))
    rng = np.random.default_rng(8)
    base = np.array([-1, -1, 0, 1, -1, 0, 0, 1, 0], np.float32)
    w.triangles = (base + rng.uniform(-0.05, 0.05, (96, 9))).astype(np.float32)
    w.triangle_materials = np.full(96, m, np.uint32)
    o = rng.uniform(-0.2, 0.2, (4000, 3)).astype(np.float32)
    o[:, 2] = 3.0
    d = rng.uniform(-0.05, 0.05, (4000, 3)).astype(np.float32)
    d[:, 2] = -1.0
    rays = abi.make_rays(o, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    for kernel in (0, 1, 2):
        check(ctx, restatement, w, rays, kernel)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 17, 148 * 112, 148 * 112 + 1])
def test_small_batches_by_groups(ctx, restatement, n):
    """Kernel 0 on both sides of the rule that hands small batches over larger trees to groups of 8
    lanes, and around a group's and a warp's share."""
    w = scenes.random_world(400, 1500, False, seed=5)
    ctx.upload(w)
    assert ctx.stats().num_wide_nodes > 64
    check(ctx, restatement, w, scenes.random_test_rays(2 * n + 16, seed=n)[:n], 0)
