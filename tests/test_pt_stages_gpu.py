"""The path tracer's launches where they can go wrong: depths 0 to 6 (the counter sets of four depths in
turn), many small waves on the same counters against one wave, one and two waves in flight, a lit
background (added beside the paths' shadow rays), and queues around a warp's 32 entries.

Tolerance: the same paths on both sides, so only the order in which a path's at most 6 * 2 light
samples and its background are added differs: 13 roundings of 2^-24 of the sum, 8e-7 relative."""
import numpy as np
import pytest

from rbr_b200 import Context, abi, render_params, scenes

pytestmark = pytest.mark.gpu


def lit_scene(width, height, fog):
    s = (scenes.foggy_cornell_box if fog else scenes.cornell_box)(width, height)
    s.point_light((0.0, 1.2, 0.6), (1.0, 0.9, 0.8), 0.5)
    s.background = (0.3, 0.2, 0.1)
    s.camera = scenes.look_at_camera(width, height, (0.0, 1.0, 6.0), (0.0, 1.0, 0.0), (0.0, 1.0, 0.0), 40.0)
    return s


@pytest.mark.parametrize("fog", [False, True])
@pytest.mark.parametrize("depth", [0, 1, 2, 3, 6])
def test_small_waves_equal_one_wave(fog, depth):
    s = lit_scene(67, 45, fog)
    p = render_params(spp=3, max_depth=depth, seed=5, flags=abi.RBR_RENDER_VOLUMETRIC if fog else 0)
    with Context(0) as c:
        c.upload(s)
        films = []
        for wave, streams in ((1 << 23, 1), (1 << 23, 2), (1024, 2), (1024, 1)):
            c.set_param("pt.wave_paths", wave)
            c.set_param("pt.streams", streams)
            films.append(c.render_host(s.camera, p, out=np.full(67 * 45 * 3, 7.0, np.float32)))
            st = c.render_stats()
            assert st.paths == 67 * 45 * 3 and st.waves == (1 if (wave, streams) == (1 << 23, 1) else 2 if wave > 1024 else 9)
    if depth == 0:
        assert not films[0].any()
    else:
        assert films[0].any()
    for f in films[1:]:
        np.testing.assert_allclose(f, films[0], rtol=8e-7, atol=1e-9)


@pytest.mark.parametrize("width,height", [(1, 1), (31, 1), (33, 1), (16, 8)])
def test_tiny_images_match_the_oracle(restatement, width, height):
    s = lit_scene(width, height, False)
    p = render_params(spp=1, max_depth=4, seed=9)
    with Context(0) as c:
        c.upload(s)
        gpu = c.render_host(s.camera, p)
    cpu = restatement.render(restatement.scene(s), s.camera, p)
    # the same random numbers; a sine or cosine an ulp off may flip a decision of a path
    assert np.isclose(gpu, cpu, rtol=1e-4, atol=1e-5).all(-1).mean() >= 0.95
