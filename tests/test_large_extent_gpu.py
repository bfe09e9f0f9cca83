"""A finely meshed object of unit size in a scene thousands of times its extent (a ground, a sky, one far
object). A ray without a limit must not visit more of the object than the same ray limited to a few units
around it: what lies beyond is a ground of one primitive. Answers are the oracle's bit for bit.

Bound: the limit's end lies past every box of the object, so both rays meet the same boxes; only roundings
of the slab distances (2^-22 of them) differ, far fewer than a tenth of the nodes."""
import numpy as np
import pytest

from rbr_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def world(half, level):
    pos, f = scenes.displaced_icosphere(level=level, radius=1.0, seed=3)
    s = scenes.Scene()
    m = s.diffuse((0.7, 0.7, 0.7))
    s.triangles = np.ascontiguousarray(pos[f].reshape(-1, 9))
    s.triangle_materials = np.full(len(f), m, np.uint32)
    s.quads = np.array([[-half, -1.2, -half, 2 * half, 0, 0, 0, 0, 2 * half]], np.float32)
    s.quad_materials = np.array([m], np.uint32)
    return s


def surface_rays(n, seed, tmax=np.inf):
    """From just above the object upwards and away from it: they hit nothing."""
    rng = np.random.default_rng(seed)
    p = rng.normal(size=(n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    d = rng.normal(size=(n, 3))
    d[(d * p).sum(1) < 0] *= -1
    d[:, 1] = np.abs(d[:, 1])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return abi.make_rays((1.15 * p).astype(np.float32), d.astype(np.float32), tmax)


def camera_rays(n, seed, tmax=np.inf):
    rng = np.random.default_rng(seed)
    d = np.concatenate([rng.uniform(-0.4, 0.4, (n, 2)), np.full((n, 1), -1.0)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return abi.make_rays(np.tile(np.array([[0.0, 0.3, 4.0]], np.float32), (n, 1)), d.astype(np.float32), tmax)


@pytest.mark.parametrize("make", [surface_rays, camera_rays])
@pytest.mark.parametrize("half", [20.0, 2000.0, 20000.0])
def test_object_nodes_do_not_grow_with_the_limit(ctx, make, half):
    torch = pytest.importorskip("torch")
    ctx.upload(world(half, 6))
    for any_hit in (False, True):
        nodes = []
        for tmax in (10.0, np.inf):
            rays = make(20000, 7, tmax)
            dev = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
            nodes.append(ctx.trace_counts_dev(dev.data_ptr(), len(rays), any_hit)[0])
        assert nodes[1] <= 1.1 * nodes[0]


@pytest.mark.parametrize("kernel,order", [(0, 0), (0, 5), (1, 0), (2, 0)])
@pytest.mark.parametrize("half", [2000.0, 20000.0])
def test_answers_match_bruteforce(ctx, restatement, kernel, order, half):
    w = world(half, 5)
    ctx.upload(w)
    h = restatement.scene(w)
    ctx.set_param("trace.kernel", kernel)
    ctx.set_param("trace.order", order)
    try:
        for rays in (surface_rays(2000, 8), camera_rays(2000, 9)):
            got, occ = ctx.trace_host(rays), ctx.trace_host(rays, any_hit=True)
            want = restatement.trace_closest(h, rays)
            assert np.array_equal(got["prim"], want["prim"])
            assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
            assert np.array_equal(occ, restatement.trace_any(h, rays))
    finally:
        ctx.set_param("trace.kernel", 0)
        ctx.set_param("trace.order", 0)
