"""A scene of one light before a background that is not black: every path's light is summed in one order
(its depths', the background last), so a render repeats bit for bit, whatever its waves and streams, alone
or in a batch, and through the radiance cache."""
import numpy as np
import pytest

from rbr_b200 import Batch, Context, render_params, scenes

pytestmark = pytest.mark.gpu

SIZE = 192


def lit_scene():
    s = scenes.cornell_box(SIZE, SIZE)
    assert len(s.lights) == 1
    s.background = (0.3, 0.2, 0.1)
    s.camera = scenes.look_at_camera(SIZE, SIZE, (0.0, 1.0, 6.0), (0.0, 1.0, 0.0), (0.0, 1.0, 0.0), 40.0)
    return s


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32).reshape(-1)


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("depth", [1, 2, 6])
def test_renders_repeat_bit_for_bit(depth, split):
    s = lit_scene()
    p = render_params(spp=16, max_depth=depth, seed=5)
    with Context(0) as c:
        c.upload(s)
        c.set_param("pt.shade_split", split)
        films = []
        for wave, streams in [(1 << 23, 2)] * 4 + [(1 << 23, 1), (20000, 2), (20000, 1)]:
            c.set_param("pt.wave_paths", wave)
            c.set_param("pt.streams", streams)
            films.append(bits(c.render_host(s.camera, p)))
    assert films[0].any()
    for f in films[1:]:
        assert np.array_equal(f, films[0])


@pytest.mark.parametrize("cfg", [dict(), dict(wave_paths=20000), dict(persistent=1), dict(persistent=1, wave_paths=20000)])
def test_batch_equals_the_render(cfg):
    torch = pytest.importorskip("torch")
    s = lit_scene()
    p = render_params(spp=16, max_depth=6, seed=5)
    with Context(0) as c:
        c.upload(s)
        want = bits(c.render_host(s.camera, p))
        b = Batch(c, **cfg)
        sid = b.add_scene(s)
        for _ in range(3):
            f = torch.zeros(SIZE * SIZE * 3, device="cuda")
            b.submit(sid, s.camera, p, f.data_ptr())
            b.run()
            torch.cuda.synchronize()
            assert np.array_equal(bits(f.cpu().numpy()), want)
        b.close()


def test_cached_frames_repeat_bit_for_bit():
    torch = pytest.importorskip("torch")
    s = lit_scene()
    with Context(0) as c:
        c.upload(s)
        c.cache_create(seed=1)
        films = []
        for _ in range(4):
            f = torch.zeros(SIZE * SIZE * 3, device="cuda")
            c.cache_render_dev(s.camera, render_params(spp=8, max_depth=6, seed=5), 1, f.data_ptr(), 0, False)
            torch.cuda.synchronize()
            films.append(bits(f.cpu().numpy()))
    for f in films[1:]:
        assert np.array_equal(f, films[0])
