"""Ray queries captured into a CUDA graph where their hand-out of rays can go wrong: batches around the
resident blocks' first runs and around the ends of a block's own chunk, against the oracle bit for bit, and
the captured launch's shape (its blocks claim rays past their first runs, as a plain call's do)."""
import numpy as np
import pytest
import torch

from rbr_b200 import Context, scenes

pytestmark = pytest.mark.gpu

RESIDENT = 148 * 8 * 128  # rays of the first runs of kernels 0 and 1 at 8 blocks per SM
RESIDENT2 = 148 * 9 * 16  # and of kernel 2 at 9


def capture(ctx, rays, any_hit):
    """The captured graph of one call, and its output buffer (after a plain call that fills it)."""
    dev = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
    out = torch.zeros(len(rays) * (1 if any_hit else 8), dtype=torch.uint8, device="cuda")
    call = ctx.trace_any_dev if any_hit else ctx.trace_closest_dev
    call(dev.data_ptr(), len(rays), out.data_ptr())
    torch.cuda.synchronize()
    plain = out.clone()
    out.fill_(0xAA)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call(dev.data_ptr(), len(rays), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    graph.instantiate()
    return graph, dev, out, plain


def kernel_nodes(graph):
    driver = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS
        return r[1]

    g = driver.CUgraph(graph.raw_cuda_graph())
    _, _, count = driver.cuGraphGetNodes(g)
    nodes = ok(driver.cuGraphGetNodes(g, count))
    return [(n, ok(driver.cuGraphKernelNodeGetParams(n))) for n in nodes
            if ok(driver.cuGraphNodeGetType(n)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("kernel,n", [(k, n) for k in (0, 1) for n in (RESIDENT, RESIDENT + 1, 2 * RESIDENT - 1, 2 * RESIDENT + 1,
                                                                       3 * RESIDENT + 129, 5 * RESIDENT + 511)]
                         + [(2, n) for n in (RESIDENT2, RESIDENT2 + 1, 2 * RESIDENT2 + 17, 40 * RESIDENT2 + 255)])
def test_captured_batches_match_the_oracle(ctx, restatement, kernel, n, any_hit):
    w = scenes.random_world(30, 150, True, seed=6, flat_triangles=4)
    ctx.upload(w)
    rays = scenes.random_test_rays(2 * n + 16, seed=n)[:n]
    ctx.set_param("trace.kernel", kernel)
    try:
        graph, dev, out, plain = capture(ctx, rays, any_hit)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        ctx.set_param("trace.kernel", 0)
    assert torch.equal(out, plain)
    h = restatement.scene(w)
    got = out.cpu().numpy()
    if any_hit:
        assert np.array_equal(got, restatement.trace_any(h, rays))
    else:
        want = restatement.trace_closest(h, rays)
        assert np.array_equal(got.view(np.uint32).reshape(-1, 2)[:, 0], want["prim"].view(np.uint32))
        assert np.array_equal(got.view(np.uint32).reshape(-1, 2)[:, 1], want["t"].view(np.uint32))


@pytest.mark.parametrize("kernel,first_run", [(0, 128), (1, 128), (2, 16)])
def test_captured_blocks_claim_past_their_first_runs(ctx, kernel, first_run):
    ctx.upload(scenes.random_world(400, 1500, False, seed=5))
    n = 1_000_003
    ctx.set_param("trace.kernel", kernel)
    try:
        graph, _, _, _ = capture(ctx, scenes.random_test_rays(2 * n, seed=3)[:n], False)
        (node, params), = kernel_nodes(graph)
    finally:
        ctx.set_param("trace.kernel", 0)
    assert params.blockDimX == 128 and params.gridDimX * first_run < n


@pytest.mark.parametrize("kernel,n", [(0, 1000), (0, 300_001), (1, 300_001), (2, 1000), (2, 300_001)])
@pytest.mark.parametrize("any_hit", [False, True])
def test_l2_persist_marks_every_launch(kernel, n, any_hit):
    """trace.l2_persist reaches small batches (groups of 8 lanes) as it does large ones."""
    driver = pytest.importorskip("cuda.bindings.driver")
    with Context(0) as ctx:
        ctx.upload(scenes.random_world(400, 1500, False, seed=5))
        ctx.set_param("trace.kernel", kernel)
        rays = scenes.random_test_rays(2 * n, seed=3)[:n]
        windows = []
        for on in (0, 1):
            ctx.set_param("trace.l2_persist", on)
            graph, _, _, _ = capture(ctx, rays, any_hit)
            (node, _), = kernel_nodes(graph)
            err, value = driver.cuGraphKernelNodeGetAttribute(
                node, driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_ACCESS_POLICY_WINDOW)
            assert err == driver.CUresult.CUDA_SUCCESS
            windows.append(value.accessPolicyWindow.num_bytes)
        ctx.set_param("trace.l2_persist", 0)
    assert windows[0] == 0 and windows[1] > 0


@pytest.mark.parametrize("ns,nt,n", [(1, 0, 1_000_003), (3, 4, 3_000_001), (10, 30, 1_000_003), (40, 200, 700_001)])
def test_small_trees_take_one_thread_per_ray(ctx, ns, nt, n):
    """Over trees of few nodes kernel 0 has a thread for every ray, whatever the batch."""
    w = scenes.random_world(ns, nt, False, seed=5, flat_triangles=4)
    ctx.upload(w)
    nodes = ctx.stats().num_wide_nodes
    assert nodes <= 8 or (nodes <= 64 and n * nodes <= 1 << 26)
    graph, _, _, _ = capture(ctx, scenes.random_test_rays(2 * n, seed=3)[:n], False)
    (_, params), = kernel_nodes(graph)
    assert params.gridDimX == (n + 127) // 128


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("past", [0, 1])
def test_small_tree_rule_edge_matches_the_oracle(ctx, restatement, past, any_hit):
    """On both sides of the batch size from which a tree of some 60 nodes goes to warp traversal."""
    w = scenes.random_world(40, 200, True, seed=5, flat_triangles=4)
    ctx.upload(w)
    n = (1 << 26) // ctx.stats().num_wide_nodes + past
    rays = scenes.random_test_rays(2 * n, seed=7)[:n]
    chunk = ctx.get_param("trace.host_chunk")
    ctx.set_param("trace.host_chunk", 0)
    try:
        got = ctx.trace_host(rays, any_hit=any_hit)
    finally:
        ctx.set_param("trace.host_chunk", chunk)
    h = restatement.scene(w)
    if any_hit:
        assert np.array_equal(got, restatement.trace_any(h, rays))
    else:
        want = restatement.trace_closest(h, rays)
        assert np.array_equal(got["prim"], want["prim"])
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))


@pytest.mark.parametrize("ns,nt", [(40, 200), (400, 1500)])
def test_kernel_1_takes_kernel_0s_ways_for_small_batches(ctx, ns, nt):
    """A batch that never refills a lane runs the same kernel whether kernel 0 or 1 is chosen (by the autotuner)."""
    driver = pytest.importorskip("cuda.bindings.driver")
    ctx.upload(scenes.random_world(ns, nt, False, seed=5))
    names = {}
    try:
        for n in (33, 1000, 40_000, RESIDENT, 4 * RESIDENT):
            rays = scenes.random_test_rays(2 * n + 16, seed=3)[:n]
            for kernel, per_sm in ((0, 0), (1, 0), (1, 8)):
                ctx.set_param("trace.kernel", kernel)
                ctx.set_param("trace.blocks_per_sm", per_sm)
                graph, _, _, _ = capture(ctx, rays, False)
                (_, params), = kernel_nodes(graph)
                names[n, kernel, per_sm] = driver.cuFuncGetName(params.func)[1]
    finally:
        ctx.set_param("trace.kernel", 0)
        ctx.set_param("trace.blocks_per_sm", 0)
    for n in (33, 1000, 40_000, RESIDENT):
        assert names[n, 1, 0] == names[n, 0, 0] != names[n, 1, 8]
    assert names[4 * RESIDENT, 1, 0] != names[4 * RESIDENT, 0, 0]
