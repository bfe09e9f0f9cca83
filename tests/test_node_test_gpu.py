"""The wide-node test at the edges of its arithmetic, against the brute-force oracle: rays of every
direction octant, zero and tiny direction components, limits from 0 to infinity, directions that
are shorter than unit vectors, origins outside the scene, and scenes of one to a few primitives
(nodes with empty slots). Every traversal kernel, bit for bit: the node test only ever has to be
conservative, so no tolerance applies."""
import numpy as np
import pytest

from rbr_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def edge_rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-14.0, 14.0, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d *= np.where(np.arange(n)[:, None] >> np.arange(3) & 1, -1, 1)  # octants in turn
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k = rng.integers(0, 3, n)
    kind = rng.integers(0, 5, n)
    rows = np.arange(n)
    d[rows[kind == 0], k[kind == 0]] = 0.0
    d[rows[kind == 1], k[kind == 1]] = -0.0
    d[rows[kind == 2], k[kind == 2]] = 1e-25
    o[kind == 3] -= d[kind == 3] * np.float32(20.0)  # aimed back at the scene from outside
    d[kind == 4] *= np.float32(1e-3)
    tmax = rng.choice(np.array([0.0, 1e-4, 0.3, 5.0, 40.0, 1e20, np.inf], np.float32), n)
    return abi.make_rays(o, d.astype(np.float32), tmax)


@pytest.mark.parametrize("kernel,order", [(0, 0), (0, 5), (1, 0), (2, 0)])
@pytest.mark.parametrize("ns,nt", [(1, 0), (3, 4), (60, 300)])
def test_node_test_edges_match_bruteforce(ctx, restatement, kernel, order, ns, nt):
    w = scenes.random_world(ns, nt, False, seed=41 + ns, flat_triangles=1 if nt == 0 else 20)
    rays = edge_rays(20000, 43 + nt)
    ctx.upload(w)
    h = restatement.scene(w)
    want = restatement.trace_closest(h, rays)
    want_any = restatement.trace_any(h, rays)
    ctx.set_param("trace.kernel", kernel)
    ctx.set_param("trace.order", order)
    try:
        got = ctx.trace_host(rays)
        got_any = ctx.trace_host(rays, any_hit=True)
    finally:
        ctx.set_param("trace.kernel", 0)
        ctx.set_param("trace.order", 0)
    assert np.array_equal(got["prim"], want["prim"])
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
    assert np.array_equal(got_any, want_any)
