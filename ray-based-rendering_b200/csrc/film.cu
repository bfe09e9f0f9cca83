// Film export on the device: Film::toRGB8 and Film::toRGB8ToneMapped (src/core/film.cpp:34-62)
// over a film of per-pixel means (what Film::getPixel returns after one averaged sample).
#include "rbr_bsdf.cuh"
#include <algorithm>
#include "rbr_context.h"

namespace rbr {
namespace {

// encode(): gamma, clamp to [0, 1] as std::max(0, std::min(1, v)), * 255 + 0.5, truncated.
__device__ __forceinline__ uint8_t encode8(float v, float inv_gamma) {
    const float p = static_cast<float>(pow(static_cast<double>(v), static_cast<double>(inv_gamma)));
    // std::max(0, std::min(1, p)) sends NaN (a negative value's power) to 1; a saturating
    // clamp would send it to 0, so NaN is handled before clamping.
    const float c = (p != p) ? 1.0f : fminf(fmaxf(p, 0.0f), 1.0f);
    return static_cast<uint8_t>(__float2uint_rz(fa(fm(c, 255.0f), 0.5f)));
}

__device__ __forceinline__ float exp2f_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Half-width of the band around a byte boundary within which the single-precision estimate below may
// round the other way. The approximate logarithm is off by 2^-22 of itself or, for v within [1/2, 2], of
// 1, so with g <= 4 the exponent g log2 v by 4 x 2^-22 and 5/4 x 2^-22 of itself; the tone map's approximate
// quotient is off by 2 ulp, at most 2^-22 of v, 5.8 x 2^-22 in the exponent; the power by 2^-22 of itself.
// A byte x has |g log2 v| = log2(255 / x), and x times the sum (the exponent's by ln 2) is largest at 255:
// 4.8e-4. 255 p + 0.5 in floats adds half an ulp of 256 twice on either side, 6e-5.
constexpr float kByteBand = 8e-4f;
constexpr float kMostInvGamma = 4.0f;

// encode8 of the (tone-mapped) value from approximate functions, for inv_gamma <= kMostInvGamma, or -1
// where only the double-precision power decides: within the band of a boundary, for negative values and NaN.
__device__ __forceinline__ int encode8_fast(float v, float exposure, float inv_gamma, int tonemap) {
    if (tonemap) {
        v *= exposure;
        // below 1e-7 the quotient is v to 2^-23, and the approximate one might flush a subnormal
        v = v < 1e-7f ? v : v < 1e30f ? __fdividef(v, v + 1.0f) : -1.0f;
    }
    const float p = fminf(exp2f_approx(inv_gamma * __log2f(v)), 1.0f);
    const float x = fmaf(p, 255.0f, 0.5f), f = floorf(x), r = x - f;
    return v >= 0.0f && r > kByteBand && r < 1.0f - kByteBand ? static_cast<int>(f) : -1;
}

// Every value of the film on its own: kPer values a thread, as one load and one store where kPer is 4.
// The double-precision power of every value bound the export (1080p 56 us, 12 times its memory time);
// with the estimate above (kFast) one value in 600 still takes it: 17.6 us (22.4 with log2f, exp2f and the
// exact quotient for every value), bound by the warps in which some value does.
template <int kPer, bool kFast>
__global__ void __launch_bounds__(256) k_film_rgb8(const float* __restrict__ film, uint64_t count, float exposure,
                                                   float inv_gamma, int tonemap, uint8_t* __restrict__ out) {
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count / kPer; i += stride) {
        float v[kPer];
        if constexpr (kPer == 4) {
            const float4 q = __ldcs(reinterpret_cast<const float4*>(film) + i);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else {
            v[0] = film[i];
        }
        uint32_t word = 0, open = 0;  // bytes, and the values still to encode
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int e = kFast ? encode8_fast(v[k], exposure, inv_gamma, tonemap) : -1;
            if (e < 0) open |= 1u << k;
            else word |= static_cast<uint32_t>(e) << (8 * k);
        }
        while (open != 0) {
            const int k = __ffs(static_cast<int>(open)) - 1;
            open &= open - 1;
            float x = v[0];
#pragma unroll
            for (int m = 1; m < kPer; ++m) x = k == m ? v[m] : x;
            if (tonemap) {  // Reinhard: c = c * exposure; c = c / (c + 1)
                x = fm(x, exposure);
                x = fd(x, fa(x, 1.0f));
            }
            word |= static_cast<uint32_t>(encode8(x, inv_gamma)) << (8 * k);
        }
        if constexpr (kPer == 4) reinterpret_cast<uint32_t*>(out)[i] = word;
        else out[i] = static_cast<uint8_t>(word);
    }
}

}  // namespace
}  // namespace rbr

using namespace rbr;

extern "C" {

rbr_status rbr_film_to_rgb8(rbr_ctx* ctx, const float* film, int32_t width, int32_t height, float exposure, float gamma,
                            int tonemap, uint8_t* out, void* stream) {
    if (!ctx || !film || !out || width <= 0 || height <= 0 || !(gamma > 0.0f)) return RBR_ERR_INVALID_ARGUMENT;
    const DeviceScope scope(ctx->device);
    const uint64_t count = uint64_t(width) * uint64_t(height) * 3;
    const float inv_gamma = 1.0f / gamma;
    const auto s = static_cast<cudaStream_t>(stream);
    const uint64_t most = uint64_t(ctx->num_sms) * 32;
    // Four values a thread where the buffers are aligned for it, the last count % 4 one by one. One value a
    // thread for small films, which one round of resident threads covers: without a second launch for the
    // remainder (7x5 16.1 us with it, 11.2 without; no slower at 64x48 to 400x300). Without the estimate for
    // exponents it does not cover (1080p, gamma 0.2: 58.5 us with it for nothing, 52.4 without).
    const bool fast = inv_gamma <= kMostInvGamma;
    const bool wide = fast && count > uint64_t(ctx->num_sms) * 2048 && (reinterpret_cast<uintptr_t>(film) & 15u) == 0 &&
                      (reinterpret_cast<uintptr_t>(out) & 3u) == 0;
    const uint64_t head = wide ? count & ~uint64_t(3) : 0;
    if (head)
        k_film_rgb8<4, true><<<static_cast<uint32_t>(std::min((head / 4 + 255) / 256, most)), 256, 0, s>>>(
            film, head, exposure, inv_gamma, tonemap, out);
    if (head < count) {
        auto k = fast ? k_film_rgb8<1, true> : k_film_rgb8<1, false>;
        k<<<static_cast<uint32_t>(std::min((count - head + 255) / 256, most)), 256, 0, s>>>(
            film + head, count - head, exposure, inv_gamma, tonemap, out + head);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "film export");
    return RBR_OK;
}

rbr_status rbr_film_to_rgb8_host(rbr_ctx* ctx, const float* film, int32_t width, int32_t height, float exposure,
                                 float gamma, int tonemap, uint8_t* out) {
    if (!ctx || !film || !out || width <= 0 || height <= 0) return RBR_ERR_INVALID_ARGUMENT;
    const DeviceScope scope(ctx->device);
    const size_t npix = size_t(width) * size_t(height);
    rbr_status st = ensure(ctx, ctx->stage_in, npix * 12, "film staging");
    if (st == RBR_OK) st = ensure(ctx, ctx->stage_out, npix * 3, "film staging");
    if (st != RBR_OK) return st;
    cudaError_t e = cudaMemcpyAsync(ctx->stage_in.ptr, film, npix * 12, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "film export");
    st = rbr_film_to_rgb8(ctx, static_cast<const float*>(ctx->stage_in.ptr), width, height, exposure, gamma, tonemap,
                          static_cast<uint8_t*>(ctx->stage_out.ptr), ctx->stream);
    if (st != RBR_OK) return st;
    e = cudaMemcpyAsync(out, ctx->stage_out.ptr, npix * 3, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "film export");
    return RBR_OK;
}

}  // extern "C"
