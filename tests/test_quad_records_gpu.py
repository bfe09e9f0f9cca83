"""Quad records on the device (host-computed normals, edge tests without divisions) against the oracle,
bit for bit: rays at corners, along edges and just past them, axis-aligned and tilted quads of sizes
from 1e-3 to 1e3, and degenerate ones (a zero edge, parallel edges)."""
import numpy as np
import pytest

from rbr_b200 import abi, scenes

pytestmark = pytest.mark.gpu

F32 = np.float32


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3])
@pytest.mark.parametrize("tilted", [False, True])
def test_quad_edges_match_bruteforce(ctx, restatement, scale, tilted):
    rng = np.random.default_rng(17)
    n = 24
    o = rng.uniform(-5, 5, (n, 3)).astype(F32)
    u, v = np.zeros((n, 3), F32), np.zeros((n, 3), F32)
    a, b = rng.integers(0, 3, n), rng.integers(1, 3, n)
    u[np.arange(n), a] = rng.uniform(0.5, 2.0, n)
    v[np.arange(n), (a + b) % 3] = rng.uniform(0.5, 2.0, n)
    if tilted:
        u += rng.uniform(-0.4, 0.4, (n, 3)).astype(F32)
        v += rng.uniform(-0.4, 0.4, (n, 3)).astype(F32)
    u[0] = 0.0           # a zero edge
    v[1] = u[1]          # parallel edges
    o, u, v = (x * F32(scale) for x in (o, u, v))
    s = scenes.Scene()
    m = s.diffuse((0.5, 0.5, 0.5))
    s.quads = np.ascontiguousarray(np.concatenate([o, u, v], 1).astype(F32))
    s.quad_materials = np.full(n, m, np.uint32)
    # targets on the quads: corners, edges, and points a few ulps or a little off them
    q = rng.integers(0, n, 12000)
    grid = np.array([0.0, 1.0, 0.5, -1e-7, 1.0 + 1.2e-7, 1e-7, 1.0 - 6e-8, -0.01, 1.01], F32)
    cu, cv = rng.choice(grid, len(q)), rng.choice(grid, len(q))
    tgt = (o[q] + u[q] * cu[:, None] + v[q] * cv[:, None]).astype(F32)
    org = (tgt + rng.normal(size=tgt.shape).astype(F32) * F32(4 * scale)).astype(F32)
    half = np.arange(len(q)) % 2 == 0  # half of the rays straight along an axis
    k = rng.integers(0, 3, len(q))
    ax = tgt.copy()
    ax[np.arange(len(q)), k] += F32(3 * scale)
    org[half] = ax[half]
    d = tgt - org
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-20)
    rays = abi.make_rays(org, d.astype(F32))
    ctx.upload(s)
    h = restatement.scene(s)
    want = restatement.trace_closest(h, rays)
    got = ctx.trace_host(rays)
    assert np.array_equal(got["prim"], want["prim"])
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
    assert np.array_equal(ctx.trace_host(rays, any_hit=True), restatement.trace_any(h, rays))
