"""The film export's single-precision estimate against double precision: every byte must be the one
float32(pow(double(v), double(1 / gamma))) gives, above all next to the byte boundaries, for values
outside [0, 1], and for sizes and addresses that the four-value loads and stores do not divide."""
import ctypes as C

import numpy as np
import pytest

from rbr_b200 import abi

pytestmark = pytest.mark.gpu

F32 = np.float32


def expected(film, gamma, tonemap, exposure):
    v = film.astype(F32)
    with np.errstate(all="ignore"):
        if tonemap:
            v = v * F32(exposure)
            v = v / (v + F32(1))
        g = F32(1) / F32(gamma)
        p = np.power(v.astype(np.float64), np.float64(g)).astype(F32)
    c = np.where(np.isnan(p), F32(1), np.clip(p, F32(0), F32(1)))
    return (c * F32(255) + F32(0.5)).astype(np.uint8)


def values(n, gamma, seed):
    """Random radiance with values a few ulps around the byte boundaries, and special ones."""
    rng = np.random.default_rng(seed)
    v = (rng.random(n) ** 3 * 4.0).astype(F32)
    edge = (((np.arange(1, 256) - 0.5) / 255.0) ** gamma).astype(F32)
    near = np.concatenate([(edge.view(np.int32) + k).view(F32) for k in range(-3, 4)])
    m = min(n, len(near))
    v[:m] = near[:m]
    special = np.array([0.0, -0.0, 1.0, 1.0000001, 0.9999999, 1e-30, 1e-45, 7.0, np.inf, -0.25, -np.inf, np.nan], F32)
    k = min(len(special), n)
    v[n - k:] = special[:k]
    return v


@pytest.mark.parametrize("gamma,tonemap,exposure", [(2.2, False, 1.0), (2.2, True, 1.5), (1.0, False, 1.0), (0.5, True, 0.3),
                                                    (2.4, False, 1.0), (100.0, False, 1.0), (100.0, True, 1.0), (0.2, False, 1.0)])
@pytest.mark.parametrize("width,height,shift", [(1, 1, 0), (3, 5, 0), (641, 479, 0), (512, 256, 1), (64, 64, 4)])
def test_bytes_equal_double_precision(ctx, gamma, tonemap, exposure, width, height, shift):
    torch = pytest.importorskip("torch")
    n = width * height * 3
    film = values(n, gamma, 11)
    buf = torch.zeros(n + 8, dtype=torch.float32, device="cuda")
    buf[shift:shift + n] = torch.from_numpy(film).cuda()
    out = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    st = ctx.lib.rbr_film_to_rgb8(ctx.h, C.c_void_p(buf.data_ptr() + 4 * shift), width, height, exposure, gamma, int(tonemap),
                                  C.c_void_p(out.data_ptr() + shift), None)
    assert st == abi.RBR_OK, ctx.last_error()
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(got[shift:shift + n], expected(film, gamma, tonemap, exposure))
    assert (got[:shift] == 7).all() and (got[shift + n:] == 7).all()
