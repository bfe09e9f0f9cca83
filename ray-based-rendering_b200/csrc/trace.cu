// Ray-query kernels: closest hit and any hit for a batch of rbr_ray records.
//
// Rays are read as two 16 B words (origin+tmax, direction+pad), answers
// written as one 8 B word (closest) or one byte (any). The traversal itself is in
// rbr_device.cuh.
#include <algorithm>
#include <cmath>

#include <cub/device/device_radix_sort.cuh>

#include "rbr_context.h"
#include "rbr_device.cuh"
#include "rbr_sort.cuh"

namespace rbr {

namespace {

constexpr int kTraceBlock = 128;

// Ray loads and hit stores: with kStream, evict-first (streaming) hints, since every ray and
// hit is touched once and the L2 is better spent on the BVH.
template <bool kStream>
__device__ __forceinline__ float4 ray_word(const float4* p) { return kStream ? __ldcs(p) : __ldg(p); }
template <bool kStream>
__device__ __forceinline__ void put_hit(uint2* p, uint2 h) {
    if (kStream) __stcs(p, h);
    else *p = h;
}

// One thread per ray in the order `perm` (a permutation of 0..n-1): rays that start close together
// with directions of the same octant share warps, so they walk the same nodes. Answers go to the
// rays' own positions. kMinBlocks: resident blocks per SM the register allocation must allow (8:
// up to 64 registers a thread, 10: 48, 12: 40) -- occupancy against register spills, picked by
// tuning.
template <int kMinBlocks, bool kStream>
__global__ void __launch_bounds__(kTraceBlock, kMinBlocks)
    k_trace_closest_perm(DeviceScene s, const float4* __restrict__ rays, uint32_t n, const uint32_t* __restrict__ perm,
                         uint2* __restrict__ hits, int* err) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t i = kStream ? __ldcs(perm + j) : __ldg(perm + j);
    const float4 a = ray_word<kStream>(rays + 2 * static_cast<size_t>(i));
    const float4 b = ray_word<kStream>(rays + 2 * static_cast<size_t>(i) + 1);
    float t = 0.0f;
    const uint32_t prim = traverse<false>(s, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, t, err);
    put_hit<kStream>(hits + i, make_uint2(prim, prim == 0xFFFFFFFFu ? 0u : __float_as_uint(t)));
}

// Launches a ray-query kernel; with trace.l2_persist the BVH's address range (nodes and leaf
// records) is marked persisting in L2 for this launch only (a launch attribute: the caller's
// stream keeps its own attributes).
template <typename... Params, typename... Args>
cudaError_t launch_query(const rbr_ctx* ctx, void (*kernel)(Params...), uint32_t blocks, cudaStream_t stream,
                         Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kTraceBlock);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (ctx->trace_l2_persist && ctx->bvh_bytes && ctx->l2_persist_bytes) {
        attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
        attr[0].val.accessPolicyWindow.base_ptr = const_cast<void*>(ctx->bvh_base);
        attr[0].val.accessPolicyWindow.num_bytes = ctx->bvh_bytes;
        attr[0].val.accessPolicyWindow.hitRatio =
            static_cast<float>(std::min(1.0, double(ctx->l2_persist_bytes) / double(ctx->bvh_bytes)));
        attr[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        attr[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

__global__ void __launch_bounds__(kTraceBlock) k_trace_any_perm(DeviceScene s, const float4* __restrict__ rays, uint32_t n,
                                                                const uint32_t* __restrict__ perm,
                                                                uint8_t* __restrict__ occ, int* err) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t i = __ldg(perm + j);
    const float4 a = __ldg(rays + 2 * static_cast<size_t>(i));
    const float4 b = __ldg(rays + 2 * static_cast<size_t>(i) + 1);
    float t;
    occ[i] = static_cast<uint8_t>(traverse<true>(s, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, t, err));
}

// Sort keys from the direction octant (3 bits) and a Morton code of the origin's cell over the
// scene box. order 1: octant, then 27-bit Morton code of 512^3 cells (30 key bits); order 2:
// octant, then 18-bit code of 64^3 cells (21 bits, one radix pass fewer); order 3: the 64^3
// cell first, octant last (21 bits), so consecutive warps stay in one region of the scene.
// Orders 4 and 5 bin the direction finely and the origin coarsely (16 bits, two radix passes):
// the direction's octahedral map onto the unit square in 16 x 8 cells (7 bits) and a Morton
// code of 8^3 origin cells (9 bits); order 4 direction first, order 5 origin first. Rays of one
// direction cell from nearby origins diverge less than rays of one octant, whose directions
// span 90 degrees.
__device__ __forceinline__ uint32_t spread3(uint32_t x) {  // 9 bits -> every third of 27
    x &= 0x1FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// Sort key of one ray (a = origin and tmax, b = direction). Orders 1-3: direction octant and
// Morton code of the origin cell (64^3 or 512^3 cells); orders 4 and 5: octahedral direction
// cell of 16 x 8 and origin cell of 8^3, 16 bits.
__device__ __forceinline__ uint32_t ray_key(float4 a, float4 b, float3 lo, float3 scale, int order) {
    const uint32_t oct = (signbit(b.x) ? 4u : 0u) | (signbit(b.y) ? 2u : 0u) | (signbit(b.z) ? 1u : 0u);
    auto cell = [](float v, float l, float sc) {
        const float c = (v - l) * sc;  // NaN and out-of-box origins clamp to the box
        return static_cast<uint32_t>(fminf(fmaxf(c, 0.0f), 511.0f));
    };
    const uint32_t m = spread3(cell(a.x, lo.x, scale.x)) << 2 | spread3(cell(a.y, lo.y, scale.y)) << 1 |
                       spread3(cell(a.z, lo.z, scale.z));
    if (order >= 4) {
        // octahedral map: (x, y) / (|x| + |y| + |z|), the lower hemisphere folded outwards
        const float l1 = fabsf(b.x) + fabsf(b.y) + fabsf(b.z);
        float u = l1 > 0.0f ? b.x / l1 : 0.0f, v = l1 > 0.0f ? b.y / l1 : 0.0f;
        if (b.z < 0.0f) {
            const float uu = (1.0f - fabsf(v)) * (u < 0.0f ? -1.0f : 1.0f);
            v = (1.0f - fabsf(u)) * (v < 0.0f ? -1.0f : 1.0f);
            u = uu;
        }
        const uint32_t du = static_cast<uint32_t>(fminf(fmaxf((u + 1.0f) * 8.0f, 0.0f), 15.0f));  // NaN -> 0
        const uint32_t dv = static_cast<uint32_t>(fminf(fmaxf((v + 1.0f) * 4.0f, 0.0f), 7.0f));
        const uint32_t dir = (du << 3) | dv;
        const uint32_t c = m >> 18;  // 8^3 cells: the top 9 bits of the 27-bit code
        return order == 4 ? (dir << 9) | c : (c << 7) | dir;
    }
    return order == 1 ? (oct << 27) | m : order == 2 ? (oct << 18) | (m >> 9) : ((m >> 9) << 3) | oct;
}

__global__ void k_ray_keys(const float4* __restrict__ rays, uint32_t n, float3 lo, float3 scale, int order,
                           uint32_t* keys, uint32_t* idx) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = __ldg(rays + 2 * static_cast<size_t>(i));
        const float4 b = __ldg(rays + 2 * static_cast<size_t>(i) + 1);
        keys[i] = ray_key(a, b, lo, scale, order);
        idx[i] = i;
    }
}

// Orders 4 and 5 (16-bit keys) use the counting sort of rbr_sort.cuh: 65,536 key values in 64
// chunks.
constexpr uint32_t kKeyValues = 1u << 16;
constexpr uint32_t kScanChunks = kKeyValues / kScanThreads;

__global__ void k_ray_keys16(const float4* __restrict__ rays, uint32_t n, float3 lo, float3 scale, int order,
                             uint16_t* __restrict__ keys, uint32_t* __restrict__ counts) {
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        uint32_t k = kNoKey;
        if (i < n) {
            const float4 a = __ldg(rays + 2 * static_cast<size_t>(i));
            const float4 b = __ldg(rays + 2 * static_cast<size_t>(i) + 1);
            k = ray_key(a, b, lo, scale, order);
            keys[i] = static_cast<uint16_t>(k);
        }
        count_key(counts, k);
    }
}

__global__ void k_ray_scatter16(const uint16_t* __restrict__ keys, uint32_t n, uint32_t* __restrict__ offsets,
                                const uint32_t* __restrict__ chunk_sum, uint32_t* __restrict__ perm) {
    scatter_keys<kScanChunks>(keys, n, offsets, chunk_sum, perm);
}

// Same traversal, counting wide nodes fetched and leaf records tested (summed over the batch).
template <bool kAny>
__global__ void __launch_bounds__(kTraceBlock) k_trace_count(DeviceScene s, const float4* __restrict__ rays,
                                                             uint32_t n, unsigned long long* totals, int* err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint2 c = make_uint2(0, 0);
    if (i < n) {
        const float4 a = __ldg(rays + 2 * static_cast<size_t>(i));
        const float4 b = __ldg(rays + 2 * static_cast<size_t>(i) + 1);
        float t;
        traverse<kAny, true>(s, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, t, err, &c);
    }
    unsigned long long nodes = c.x, recs = c.y;
    for (int off = 16; off > 0; off >>= 1) {
        nodes += __shfl_down_sync(0xFFFFFFFFu, nodes, off);
        recs += __shfl_down_sync(0xFFFFFFFFu, recs, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(totals, nodes);
        atomicAdd(totals + 1, recs);
    }
}

__device__ __forceinline__ uint32_t lane_mask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Persistent warps: each warp starts with the 32 rays of its own index and claims the next 32 from
// a global cursor when it needs more. Incoherent rays were bound by instruction issue at 8 to 12 of
// 32 lanes active: some rays of a warp end long before others, and few lanes test leaf records at
// once. A warp looks at its first rays and keeps to one of two ways:
//   - Warp traversal (rbr_device.cuh), and the next rays go to lanes whose ray is done while the
//     others are still traversing: 29 of 32 lanes busy in the node test, one round of record tests
//     a step. 2^22 uniform rays through 1.3M triangles 1,620 -> 1,068 us (sorted first, one thread
//     per ray: 1,380), any hit 1,240 -> 871; 2^22 shadow segments over 2M triangles 838 -> 501;
//     1,024 to 2^16 rays, bound by the longest traversals, unchanged to 20 % faster.
//   - Coherent rays (neighbouring origins, nearly the same direction: camera rays in scanline
//     order) walk the same nodes and finish together: one thread per ray, 32 new rays when all are
//     done, where coherent_pays().
// A claim is 32 rays whatever the batch: with claims of up to 256 the warps that drew the long
// traversals of a camera image kept a launch alive behind the others (2^22 rays 1,701 us, 764 at
// 32). Not kept: claiming the next run ahead of a traversal (679 us instead of 591: a held run
// waits behind a long one), records tested by their own lane where many lanes have one.
// An any-hit claim is 64 rays while there are plenty and the last run was quick, since claims on one cursor
// are served 0.85 ns apart: 2^22 rays that hit the first primitive they meet 106 -> 75 us (20 K triangles,
// one thread per ray) and 108 -> 90 (2 M, warp traversal), that miss the tree 106 -> 84. It costs other
// any-hit rays traced one thread per ray 3 % (2^22 through 195 nodes 352 -> 363). Not for closest hits,
// where a claim of long traversals among quick ones keeps camera images alive: 2^20 rays over 2M triangles
// 332 -> 379.
// With `perm` (sorted rays), position j of the order is ray perm[j]. kRefillOnly: every warp goes
// the second way.
constexpr int kPersistBlock = kTraceBlock;
constexpr int kTraceBlocksPerSm = 8;
constexpr uint32_t kPersistChunk = 4;  // first runs in a block's own chunk, at most
constexpr uint32_t kClaimRays = 32;
constexpr uint32_t kQuickSteps = 3;       // a run of rays that took fewer steps, or by one thread per
constexpr uint32_t kQuickTicks = 5000;    // ray no more clock ticks, was quick
constexpr uint32_t kSmallTree = 64;       // nodes
constexpr uint32_t kAdaptiveRefill = 6;   // idle lanes before a refill (4 to 8 measured within 2 %)

// Origins within 1/16 of the tree's extent of the warp's first ray's and directions within 11
// degrees of its: half of a 32-ray run of camera rays spans a degree, rays after a bounce the
// sphere. The choice changes no answer.
__device__ __forceinline__ bool coherent_rays(const DeviceScene& s, bool valid, float4 a, float4 b) {
    const float ox = __shfl_sync(0xFFFFFFFFu, a.x, 0), oy = __shfl_sync(0xFFFFFFFFu, a.y, 0), oz = __shfl_sync(0xFFFFFFFFu, a.z, 0);
    const float dx = __shfl_sync(0xFFFFFFFFu, b.x, 0), dy = __shfl_sync(0xFFFFFFFFu, b.y, 0), dz = __shfl_sync(0xFFFFFFFFu, b.z, 0);
    const float off = fabsf(a.x - ox) + fabsf(a.y - oy) + fabsf(a.z - oz);
    const float c = b.x * dx + b.y * dy + b.z * dz;
    const float l2 = (b.x * b.x + b.y * b.y + b.z * b.z) * (dx * dx + dy * dy + dz * dz);
    const bool near = off <= 0.125f * s.tree_reach && c > 0.0f && c * c >= 0.9635f * l2;
    return __all_sync(0xFFFFFFFFu, !valid || near);
}

// Whether one thread per ray pays for coherent rays: where most of a launch is throughput, not the
// latency of its longest traversals. Camera rays, one thread per ray against warp traversal (us):
// 20 K triangles 2^20 121 / 123, 2^21 174 / 198; 405 K 2^20 222 / 191, 2^21 275 / 270, 2^22 390 / 428;
// 2 M 2^21 437 / 370, 2^22 589 / 540. Below 2^20 rays only through small trees, whose longest traversals
// are short: 109 nodes 2^18 34 / 47, 2^19 59 / 76; 195 nodes 2^18 47 / 63, 2^19 79 / 102; 369 nodes 2^19
// 117 / 148.
__device__ __forceinline__ bool coherent_pays(const DeviceScene& s, uint32_t n) {
    return n / 32u >= s.num_nodes && (n >= (1u << 20) || n / 1024u >= s.num_nodes);
}

// Trees through which any rays are traced one thread per ray, in blocks for all of them without claims:
// traversals of a few nodes are not worth refilling a lane for, nor 32 of them a claim (those on one cursor
// are served 0.85 ns apart, 107 us for 2^22 rays). Uniform rays before the persistent warps / by them / so
// (us): Cornell box (1 node) 2^18 27.7 / 29.7 / 21.6, 2^22 311 / 308 / 234, any hit 219 / 281 / 165;
// 8 nodes 2^18 23.9 / 25.7 / 17.3, 2^22 250 / 203 / 177; 61 nodes 2^18 58 / 46 / 36, 2^20 191 / 122 / 119,
// 2^21 363 / 217 / 223: a launch gains by refills from about 2^26 rays times nodes on. Few rays, whose
// latency counts: 1,001 over 61 nodes 15.1 us, 17.6 by warp traversal.
__host__ __device__ __forceinline__ bool thread_per_ray(uint32_t num_nodes, uint32_t n) {
    return num_nodes <= 8u || (num_nodes <= kSmallTree && n <= (1u << 26) / num_nodes);
}

// The rays a block works on: all n of them, claimed from a cursor that the grid shares, or where there is
// none (and kOwn) `chunk` consecutive ones, claimed from a cursor of the block's own. The warps' first
// runs go by their index in the grid or the block. Without a cursor and with chunks of one first run, the
// rays past the grid's first runs are a second run for the warps by index.
template <uint32_t kBlockRays, bool kOwn>
struct BlockRays {
    uint32_t n, chunk;
    uint32_t *cursor, *own;

    __device__ __forceinline__ uint32_t begin() const { return blockIdx.x * (kOwn && !cursor ? chunk : kBlockRays); }
    __device__ __forceinline__ void start() const {
        if (!kOwn || cursor || chunk == kBlockRays) return;
        if (threadIdx.x == 0) *own = 0;
        __syncthreads();
    }
    // Whether the grid's warps have four more runs each to come.
    __device__ __forceinline__ bool plenty(uint32_t end) const { return cursor && (n - end) / 4u > gridDim.x * kBlockRays; }
    // The next `count` rays for a warp (run to end); false when there are none. Out of line in kernels with
    // every way of claiming: their code in the traversal loop cost it 1 % (2^22 uniform rays 1,071 -> 1,061 us).
    __device__ __forceinline__ bool claim(uint32_t count, uint32_t& run, uint32_t& end) const {
        if (!kOwn) return take(n, chunk, cursor, own, count, run, end);
        const uint2 r = taken(n, chunk, cursor, own, count, end);
        run = r.x;
        end = r.y;
        return r.x != r.y;
    }
    static __device__ __noinline__ uint2 taken(uint32_t n, uint32_t chunk, uint32_t* cursor, uint32_t* own, uint32_t count,
                                               uint32_t end) {
        uint32_t run = 0;
        return take(n, chunk, cursor, own, count, run, end) ? make_uint2(run, end) : make_uint2(0u, 0u);
    }
    static __device__ __forceinline__ bool take(uint32_t n, uint32_t chunk, uint32_t* cursor, uint32_t* own, uint32_t count,
                                                uint32_t& run, uint32_t& end) {
        uint32_t b = 0, limit = n, first = gridDim.x * kBlockRays;
        if (!kOwn && !cursor) return false;
        if (!kOwn || cursor) {
            if ((threadIdx.x & 31u) == 0) b = atomicAdd(cursor, count);
        } else if (chunk == kBlockRays) {
            if (end > first || n - end <= first - count) return false;  // a second run, or none behind it
            run = end + (first - count);
            end = run + min(count, n - run);
            return true;
        } else {
            const uint32_t from = blockIdx.x * chunk, rays = min(chunk, n - from);
            if (rays <= kBlockRays) return false;
            first = from + kBlockRays;
            limit = from + rays;
            if ((threadIdx.x & 31u) == 0) b = atomicAdd(own, count);
        }
        run = first + __shfl_sync(0xFFFFFFFFu, b, 0);
        if (run < first || run >= limit) return false;  // past the end (run < first: past 2^32)
        end = run + min(count, limit - run);
        return true;
    }
};

// The SM's clock, read no earlier than x is known.
__device__ __forceinline__ uint32_t clock_after(float x) {
    uint32_t t;
    asm volatile("{ .reg .pred p; setp.eq.f32 p, %1, %1; @p mov.u32 %0, %%clock; @!p mov.u32 %0, %%clock; }" : "=r"(t) : "f"(x));
    return t;
}

template <bool kAny, bool kStream, bool kRefillOnly>
__global__ void __launch_bounds__(kPersistBlock, kTraceBlocksPerSm)
    k_trace(DeviceScene s, const float4* __restrict__ rays, uint32_t n, const uint32_t* __restrict__ perm,
            uint2* __restrict__ hits, uint8_t* __restrict__ occ, int* err, uint32_t* cursor, uint32_t chunk,
            uint32_t refill_min) {
    __shared__ WarpRays shared[kPersistBlock / 32];
    __shared__ uint32_t own;
    WarpRays& w = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const BlockRays<kPersistBlock, true> mine{n, chunk, cursor, &own};
    mine.start();
    uint32_t run = mine.begin() + (threadIdx.x & ~31u);  // warp-uniform
    if (run < mine.begin() || run >= n) return;
    uint32_t end = run + min(kClaimRays, n - run);  // warp-uniform
    auto claim = [&](bool quick = false) {
        return mine.claim(kAny && quick && mine.plenty(end) ? 2 * kClaimRays : kClaimRays, run, end);
    };
    if (!kRefillOnly && (coherent_pays(s, n) || thread_per_ray(s.num_nodes, n))) {
        uint32_t i = run + lane;
        bool valid = i < end;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
        if (valid) {
            a = ray_word<kStream>(rays + 2 * static_cast<size_t>(i));
            b = ray_word<kStream>(rays + 2 * static_cast<size_t>(i) + 1);
        }
        if (thread_per_ray(s.num_nodes, n) || coherent_rays(s, valid, a, b)) {
            while (true) {
                uint32_t ticks = 0;
                if (valid) {
                    float t = 0.0f;
                    if (kAny && cursor) ticks = clock_after(b.x);
                    const uint32_t r = traverse<kAny>(s, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, t, err);
                    if (kAny && cursor) ticks = clock_after(__uint_as_float(r)) - ticks;
                    if (kAny) occ[i] = static_cast<uint8_t>(r);
                    else put_hit<kStream>(hits + i, make_uint2(r, r == 0xFFFFFFFFu ? 0u : __float_as_uint(t)));
                }
                if (kAny && run + kClaimRays < end) run += kClaimRays;
                else if (!claim(kAny && !__any_sync(0xFFFFFFFFu, ticks > kQuickTicks))) return;
                i = run + lane;
                valid = i < end;
                if (valid) {
                    a = ray_word<kStream>(rays + 2 * static_cast<size_t>(i));
                    b = ray_word<kStream>(rays + 2 * static_cast<size_t>(i) + 1);
                }
            }
        }
    }
    bool exhausted = false;      // warp-uniform
    uint32_t steps = 0;          // since the last refill, warp-uniform
    uint32_t idx = 0xFFFFFFFFu;  // this lane's ray
    LaneRay lr;
    uint2 stack[kStackSize];
    auto answer = [&]() {
        const unsigned long long b = w.best[lane];
        if (kAny) {
            occ[idx] = b != 0;
        } else {
            const uint32_t prim = hit_prim(b);
            put_hit<kStream>(hits + idx, make_uint2(prim, prim == 0xFFFFFFFFu ? 0u : hit_tbits(b)));
        }
        idx = 0xFFFFFFFFu;
    };
    while (true) {
        uint32_t need = __ballot_sync(0xFFFFFFFFu, idx == 0xFFFFFFFFu);
        // refill once at least refill_min lanes are idle (or all of them): a refill costs the
        // whole warp a few ballots and a ray load, so lanes may idle for a few steps first
        while (need != 0 && !exhausted && (static_cast<uint32_t>(__popc(need)) >= refill_min || need == 0xFFFFFFFFu)) {
            if (run >= end && !claim(steps < kQuickSteps && __popc(need) >= 24)) {
                exhausted = true;
                break;
            }
            const uint32_t j = run + __popc(need & lane_mask_lt());
            if (((need >> lane) & 1u) && j < end) {
                idx = perm ? __ldg(perm + j) : j;
                const float4 a = ray_word<kStream>(rays + 2 * static_cast<size_t>(idx));
                const float4 b = ray_word<kStream>(rays + 2 * static_cast<size_t>(idx) + 1);
                // finished at once: takes another ray in the same pass
                if (lane_begin<kAny>(s, w, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, lr)) answer();
            }
            run = min(end, run + __popc(need));  // each round consumes at least one ray
            steps = 0;
            need = __ballot_sync(0xFFFFFFFFu, idx == 0xFFFFFFFFu);
        }
        const bool active = idx != 0xFFFFFFFFu;
        if (__ballot_sync(0xFFFFFFFFu, active) == 0) break;  // only when the rays are exhausted
        ++steps;
        if (warp_step<kAny>(s, w, active, lr, stack, err)) answer();
    }
}

// ------------------------------------------------------------------------------------------
// Warp-cooperative traversal: a group of 8 lanes traces one ray (4 rays per warp; group_step in
// rbr_device.cuh) and takes the next ray of the warp's chunk when its own is done. Rays and hits go
// without streaming hints: a small batch's are too few to drive the BVH out of the L2, and with the hints
// the closest-hit kernel spills.
// ------------------------------------------------------------------------------------------
constexpr int kCoopBlock = kTraceBlock;
constexpr uint32_t kCoopChunk = 16;

template <bool kAny, bool kOwn>
__device__ __forceinline__ void trace_coop_body(const DeviceScene& s, const float4* __restrict__ rays, uint32_t n,
                                                uint2* __restrict__ hits, uint8_t* __restrict__ occ, int* err,
                                                uint32_t* cursor, uint32_t chunk) {
    __shared__ uint32_t own;
    const GroupLanes g = group_lanes();
    // A warp's first run is four rays, one per group, by its index; then an equal share of the rest
    // for every warp by claims (four at a time of a block's own chunk).
    const BlockRays<kCoopBlock / 8, kOwn> mine{n, chunk, cursor, &own};
    mine.start();
    uint32_t run = mine.begin() + 4u * (threadIdx.x >> 5);  // warp-uniform
    if (run < mine.begin() || run >= n) return;
    uint32_t end = run + min(4u, n - run);    // warp-uniform
    bool exhausted = false;                   // warp-uniform
    auto claim = [&]() {
        return mine.claim(kOwn ? 4u : min(32u, max(4u, n / (gridDim.x * (kCoopBlock / 32)))), run, end);
    };
    uint32_t idx = 0xFFFFFFFFu;               // group-uniform
    uint32_t anyhit = 0;
    GroupRay st{};
    uint2 stack[kStackSize];
    auto answer = [&]() {
        if (g.j == 0) {
            if (kAny) occ[idx] = static_cast<uint8_t>(anyhit);
            else hits[idx] = make_uint2(st.best < 0 ? 0xFFFFFFFFu : static_cast<uint32_t>(st.best),
                                        st.best < 0 ? 0u : __float_as_uint(st.tbest));
        }
        idx = 0xFFFFFFFFu;
    };
    while (true) {
        // give idle groups new rays from the warp's chunk
        uint32_t need = __ballot_sync(0xFFFFFFFFu, g.j == 0 && idx == 0xFFFFFFFFu);
        while (need != 0 && !exhausted) {
            if (run >= end && !claim()) {
                exhausted = true;
                break;
            }
            const uint32_t j = run + __popc(need & ((1u << g.shift) - 1u));
            if (((need >> g.shift) & 1u) && j < end) {
                idx = j;
                const float4 a = __ldg(rays + 2 * static_cast<size_t>(idx));
                const float4 b = __ldg(rays + 2 * static_cast<size_t>(idx) + 1);
                // finished at once: takes another ray in the same pass
                if (group_begin<kAny>(s, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, st, anyhit)) answer();
            }
            run = min(end, run + __popc(need));
            need = __ballot_sync(0xFFFFFFFFu, g.j == 0 && idx == 0xFFFFFFFFu);
        }
        if (__ballot_sync(0xFFFFFFFFu, idx != 0xFFFFFFFFu) == 0) break;  // rays exhausted
        if (idx != 0xFFFFFFFFu && group_step<kAny>(s, g, st, stack, err, anyhit)) answer();
    }
}

template <bool kAny>
__global__ void __launch_bounds__(kCoopBlock) k_trace_coop(DeviceScene s, const float4* __restrict__ rays, uint32_t n,
                                                           uint2* __restrict__ hits, uint8_t* __restrict__ occ,
                                                           int* err, uint32_t* cursor, uint32_t chunk) {
    trace_coop_body<kAny, false>(s, rays, n, hits, occ, err, cursor, chunk);
}

// Blocks with chunks of their own: another kernel, since the shared cursor's has no registers to spare
// (with both in one, 8,192 rays through 1.3M triangles 50 -> 54 us).
template <bool kAny>
__global__ void __launch_bounds__(kCoopBlock, 8)
    k_trace_coop_own(DeviceScene s, const float4* __restrict__ rays, uint32_t n, uint2* __restrict__ hits,
                     uint8_t* __restrict__ occ, int* err, uint32_t* cursor, uint32_t chunk) {
    trace_coop_body<kAny, true>(s, rays, n, hits, occ, err, cursor, chunk);
}

}  // namespace

// Whether the cursor of `slot` is free for a launch on `stream`: the launch that used it last was on the
// same stream (the wait for it then costs nothing; should the handle be a destroyed stream's, come back
// for another one, it orders the two) or is done. The query is allowed while another thread captures in
// the global mode: the events are never recorded in a capture.
static cudaError_t cursor_free(rbr_ctx::CursorSlot& slot, cudaStream_t stream, bool* free) {
    *free = true;
    if (!slot.done) return cudaEventCreateWithFlags(&slot.done, cudaEventDisableTiming);
    if (slot.stream == stream) return cudaStreamWaitEvent(stream, slot.done, 0);
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return e;
    const cudaError_t q = cudaEventQuery(slot.done);
    e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (q != cudaErrorNotReady) return q != cudaSuccess ? q : e;
    cudaGetLastError();
    *free = false;
    return e;
}

// How a launch of up to *grid resident blocks with first runs of `block_rays` rays a block hands out n
// rays: nothing to claim where the first runs are all of them, or for warps of 32 rays (kPersistBlock)
// where a second run for one to three quarters of the warps is (clearing a cursor and every warp's last,
// vain claim cost 4 us, more than they even out: 2^18 rays that hit the first primitive they meet 14.8
// -> 12.4 us, uniform ones through 195 nodes 79 -> 73, through 1.3M triangles 133 -> 130, camera rays
// 145 -> 142; with fewer second runs claims by whichever warps are done first gained up to a fifth,
// 170,000 camera rays 120 / 142, with more up to 7 %, 300,000 114 / 122). Else a cursor of zero, the next of the ring.
// That one may still be in use by a launch on another stream (64 short launches beside one long one), which
// this call must not wait for, and a launch captured into a graph can run beside any later one: these two
// get no cursor. *grid becomes blocks for all rays, each with a chunk of up to `most` first runs of its
// own, so that lanes are refilled within a block and the hardware hands out the blocks. 2^22 uniform rays
// through 330 K triangles, kernel 0: 1,099 us (951 by a cursor, 1,485 with first runs only, 1,082 with the
// resident blocks taking runs in turn, which lost a quarter on camera rays: 691 -> 897); kernel 2: 3,560
// (3,240; 4,444).
// The events cost nothing that shows: 2^22 uniform rays 1,048 us before, 1,032 with them (another run).
static cudaError_t take_cursor(rbr_ctx* ctx, uint32_t n, uint32_t block_rays, uint32_t most, uint32_t* grid,
                               uint32_t* chunk, uint32_t** cursor, cudaEvent_t* done, cudaStream_t stream) {
    *cursor = nullptr;
    *chunk = block_rays;
    const uint32_t first = *grid * block_rays;
    if (n <= first || (block_rays == kPersistBlock && n >= first + first / 4u && n <= first + first / 4u * 3u)) return cudaSuccess;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(stream, &capture);
    if (e != cudaSuccess) return e;
    const uint32_t at = ctx->cursor_next % kCursorRing;
    rbr_ctx::CursorSlot& slot = ctx->cursors[at];
    bool free = capture == cudaStreamCaptureStatusNone;
    if (free) {
        ++ctx->cursor_next;
        if ((e = cursor_free(slot, stream, &free)) != cudaSuccess) return e;
    }
    if (!free) {
        *chunk *= std::min(n / first, most);
        *grid = static_cast<uint32_t>((uint64_t(n) + *chunk - 1) / *chunk);
        return cudaSuccess;
    }
    slot.stream = stream;
    *done = slot.done;
    *cursor = ctx->d_cursors + at;
    return cudaMemsetAsync(*cursor, 0, sizeof(uint32_t), stream);
}

// Kernel 2, and kernel 0 on small batches (which ignores the context's grid parameter).
static cudaError_t launch_trace_coop(rbr_ctx* ctx, const rbr_ray* rays, uint32_t n, int any_hit, void* out, int per_sm,
                                     cudaStream_t stream) {
    auto k = any_hit ? k_trace_coop<true> : k_trace_coop<false>;
    if (per_sm == 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kCoopBlock, 0);
        if (e != cudaSuccess) return e;
        per_sm = std::max(1, per_sm);
    }
    // no more warps than there are groups of 8 lanes to fill
    constexpr uint32_t kBlockRays = kCoopBlock / 8;
    uint32_t grid = static_cast<uint32_t>(std::max<uint64_t>(
        1, std::min<uint64_t>(uint64_t(ctx->num_sms) * per_sm, (uint64_t(n) + kBlockRays - 1) / kBlockRays)));
    uint32_t *cursor = nullptr, chunk = 0;
    cudaEvent_t done = nullptr;
    cudaError_t e = take_cursor(ctx, n, kBlockRays, kCoopChunk, &grid, &chunk, &cursor, &done, stream);
    if (e != cudaSuccess) return e;
    if (chunk != kBlockRays) k = any_hit ? k_trace_coop_own<true> : k_trace_coop_own<false>;
    e = launch_query(ctx, k, grid, stream, ctx->scene, reinterpret_cast<const float4*>(rays), n,
                     any_hit ? nullptr : static_cast<uint2*>(out), any_hit ? static_cast<uint8_t*>(out) : nullptr,
                     ctx->d_error, cursor, chunk);
    return e != cudaSuccess || !cursor ? e : cudaEventRecord(done, stream);
}

// Whether the batch is one that never refills a lane in kernel 1 (every ray is in a resident warp's first
// run). It goes kernel 0's ways, so that a context tuned on large batches traces small ones as well: 33 to
// 32,768 rays through 61 nodes 19.4 to 21.6 us by kernel 1, 15.3 to 16.6 so; 1,024 through 1.3M triangles 53
// and 44. Not where the grid or an order is asked for.
static bool first_runs_only(const rbr_ctx* ctx, uint32_t n) {
    return ctx->trace_kernel == 1 && ctx->trace_order == 0 && ctx->trace_blocks_per_sm == 0 &&
           n <= static_cast<uint32_t>(ctx->num_sms) * (kTraceBlocksPerSm * kPersistBlock);
}

// Kernels 0 (in the given order) and 1: k_trace with the context's parameters.
static cudaError_t launch_trace_warps(rbr_ctx* ctx, const rbr_ray* rays, uint32_t n, int any_hit, void* out,
                                      const uint32_t* perm, cudaStream_t stream) {
    const bool refill_only = ctx->trace_kernel == 1 && !first_runs_only(ctx, n);
    const bool st = ctx->trace_stream_io != 0;
    auto k = any_hit ? (refill_only ? (st ? k_trace<true, true, true> : k_trace<true, false, true>)
                                    : (st ? k_trace<true, true, false> : k_trace<true, false, false>))
                     : (refill_only ? (st ? k_trace<false, true, true> : k_trace<false, false, true>)
                                    : (st ? k_trace<false, true, false> : k_trace<false, false, false>));
    int per_sm = refill_only ? ctx->trace_blocks_per_sm : 0;
    if (per_sm == 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kPersistBlock, 0);
        if (e != cudaSuccess) return e;
        per_sm = std::max(1, per_sm);
    }
    // no more warps than there are runs of rays
    const uint64_t all = (uint64_t(n) + kPersistBlock - 1) / kPersistBlock;
    uint32_t grid = static_cast<uint32_t>(
        !refill_only && thread_per_ray(ctx->scene.num_nodes, n) ? all : std::min<uint64_t>(uint64_t(ctx->num_sms) * per_sm, all));
    uint32_t *cursor = nullptr, chunk = 0;
    cudaEvent_t done = nullptr;
    cudaError_t e = take_cursor(ctx, n, kPersistBlock, kPersistChunk, &grid, &chunk, &cursor, &done, stream);
    if (e != cudaSuccess) return e;
    e = launch_query(ctx, k, grid, stream, ctx->scene, reinterpret_cast<const float4*>(rays), n, perm,
                     any_hit ? nullptr : static_cast<uint2*>(out), any_hit ? static_cast<uint8_t*>(out) : nullptr,
                     ctx->d_error, cursor, chunk, refill_only ? static_cast<uint32_t>(ctx->trace_refill_min) : kAdaptiveRefill);
    return e != cudaSuccess || !cursor ? e : cudaEventRecord(done, stream);
}

// The sort buffers of the streams of a chunked rbr_trace_host (slot 0: the context's stream).
static DevBuf& sort_slot(rbr_ctx* ctx, int slot) {
    return slot <= 0 ? ctx->sort_buf : slot == 1 ? ctx->sort_buf2 : ctx->sort_more[slot == 2 ? 0 : 1];
}

// Sorts the rays by their key of order ctx->trace_order on `stream` and returns the permutation:
// orders 4 and 5 by the counting sort above, orders 1-3 (21- and 30-bit keys) by CUB's radix sort.
static cudaError_t sort_rays(rbr_ctx* ctx, DevBuf& sort_buf, const rbr_ray* rays, uint32_t n, const uint32_t** perm,
                             cudaStream_t stream) {
    const int order = ctx->trace_order;
    float3 lo = make_float3(0.0f, 0.0f, 0.0f), sc = make_float3(0.0f, 0.0f, 0.0f);
    const float* blo = ctx->bounds_lo;
    const float* bhi = ctx->bounds_hi;
    float* so[3] = {&sc.x, &sc.y, &sc.z};
    float* lo3[3] = {&lo.x, &lo.y, &lo.z};
    for (int a = 0; a < 3; ++a) {
        const float ext = bhi[a] - blo[a];
        if (std::isfinite(blo[a]) && std::isfinite(ext) && ext > 0.0f) {
            *lo3[a] = blo[a];
            *so[a] = 512.0f / ext;
        }
    }
    const int grid = std::min<int>((n + 255) / 256, ctx->num_sms * 8);
    if (order >= 4) {  // 16-bit keys: the counting sort above
        const size_t perm_bytes = (size_t(n) * 4 + 255) & ~size_t(255);
        const size_t key_bytes = (size_t(n) * 2 + 255) & ~size_t(255);
        if (ensure(ctx, sort_buf, perm_bytes + key_bytes + (kKeyValues + kScanChunks) * 4, "ray sort") != RBR_OK)
            return cudaErrorMemoryAllocation;
        char* base = static_cast<char*>(sort_buf.ptr);
        auto* pm = reinterpret_cast<uint32_t*>(base);
        auto* keys = reinterpret_cast<uint16_t*>(base + perm_bytes);
        auto* counts = reinterpret_cast<uint32_t*>(base + perm_bytes + key_bytes);
        uint32_t* chunk_sum = counts + kKeyValues;
        cudaError_t e = cudaMemsetAsync(counts, 0, kKeyValues * 4, stream);
        if (e != cudaSuccess) return e;
        k_ray_keys16<<<grid, 256, 0, stream>>>(reinterpret_cast<const float4*>(rays), n, lo, sc, order, keys, counts);
        k_key_offsets<<<kScanChunks, kScanThreads, 0, stream>>>(counts, chunk_sum);
        k_ray_scatter16<<<grid, 256, 0, stream>>>(keys, n, counts, chunk_sum, pm);
        *perm = pm;
        return cudaGetLastError();
    }
    const int key_bits = order == 1 ? 30 : 21;
    size_t temp = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, temp, static_cast<const uint32_t*>(nullptr),
                                                    static_cast<uint32_t*>(nullptr), static_cast<const uint32_t*>(nullptr),
                                                    static_cast<uint32_t*>(nullptr), static_cast<int>(n), 0, key_bits, stream);
    if (e != cudaSuccess) return e;
    if (ensure(ctx, sort_buf, size_t(n) * 16 + temp + 256, "ray sort") != RBR_OK) return cudaErrorMemoryAllocation;
    uint32_t* base = static_cast<uint32_t*>(sort_buf.ptr);
    uint32_t *keys = base, *keys2 = base + n, *idx = base + 2 * size_t(n), *idx2 = base + 3 * size_t(n);
    void* tmp = reinterpret_cast<char*>(base + 4 * size_t(n)) + (256 - (reinterpret_cast<uintptr_t>(base + 4 * size_t(n)) & 255));
    k_ray_keys<<<grid, 256, 0, stream>>>(reinterpret_cast<const float4*>(rays), n, lo, sc, order, keys, idx);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cub::DeviceRadixSort::SortPairs(tmp, temp, keys, keys2, idx, idx2, static_cast<int>(n), 0, key_bits, stream);
    *perm = idx2;
    return e;
}

cudaError_t launch_trace(rbr_ctx* ctx, const rbr_ray* rays, uint32_t n, int any_hit, void* out, cudaStream_t stream,
                         int slot) {
    if (ctx->trace_kernel == 0 && ctx->trace_order != 0 && n > 0) {
        const uint32_t* perm = nullptr;
        cudaError_t e = sort_rays(ctx, sort_slot(ctx, slot), rays, n, &perm, stream);
        if (e != cudaSuccess) return e;
        const uint32_t blocks = (n + kTraceBlock - 1) / kTraceBlock;
        const auto* r = reinterpret_cast<const float4*>(rays);
        if (any_hit) {
            k_trace_any_perm<<<blocks, kTraceBlock, 0, stream>>>(ctx->scene, r, n, perm, static_cast<uint8_t*>(out),
                                                                ctx->d_error);
        } else {
            auto* h = static_cast<uint2*>(out);
            const bool st = ctx->trace_stream_io != 0;
            const int mb = ctx->trace_min_blocks;
            auto k = mb >= 12 ? (st ? k_trace_closest_perm<12, true> : k_trace_closest_perm<12, false>)
                     : mb >= 10 ? (st ? k_trace_closest_perm<10, true> : k_trace_closest_perm<10, false>)
                                : (st ? k_trace_closest_perm<8, true> : k_trace_closest_perm<8, false>);
            return launch_query(ctx, k, blocks, stream, ctx->scene, r, n, perm, h, ctx->d_error);
        }
        return cudaGetLastError();
    }
    if (n == 0) return cudaSuccess;
    if (ctx->trace_kernel == 2) return launch_trace_coop(ctx, rays, n, any_hit, out, ctx->trace_blocks_per_sm, stream);
    // Few rays through a large tree take as long as their longest traversals, whose steps are shorter
    // by groups of 8 lanes: up to 112 rays per SM (16,576) 9 to 25 % faster than by warps of 32 rays
    // on three scenes of 1.3M and 2M triangles (1,024 uniform rays 76 -> 70 us, 8,192 91 -> 78,
    // 8,192 shadow segments 48 -> 40, 16,384 camera rays 185 -> 165).
    if ((ctx->trace_kernel == 0 || first_runs_only(ctx, n)) && ctx->scene.num_nodes > kSmallTree &&
        n <= static_cast<uint32_t>(ctx->num_sms) * 112u)
        return launch_trace_coop(ctx, rays, n, any_hit, out, 0, stream);
    const uint32_t* perm = nullptr;  // kernel 1 refills its lanes in sorted order when trace.order is set
    if (ctx->trace_order != 0) {
        cudaError_t e = sort_rays(ctx, sort_slot(ctx, slot), rays, n, &perm, stream);
        if (e != cudaSuccess) return e;
    }
    return launch_trace_warps(ctx, rays, n, any_hit, out, perm, stream);
}

// Times every traversal variant on the caller's rays (device pointer) and keeps the fastest.
rbr_status autotune_trace(rbr_ctx* ctx, const rbr_ray* rays, uint32_t n, int any_hit, int64_t* chosen_ms_x1000) {
    struct Cand {
        int kernel, min_blocks, per_sm, order, refill;
    };
    // Rays in the given order (kernel 0 chooses between one thread per ray and warp traversal by
    // the rays' coherence; kernel 1 always refills), and sorted ones with the 16-bit keys of orders
    // 4 and 5 (the counting sort of this file). Not candidates: orders 1-3 (CUB's radix sort,
    // slower than orders 4 and 5) and kernel 2 (slower on batches large enough to tune on); both
    // stay selectable by parameter.
    const int refill = ctx->trace_refill_min;
    const Cand cands[] = {{0, 10, 0, 0, refill}, {1, 10, 0, 0, refill}, {1, 10, 0, 0, 4}, {1, 10, 0, 0, 8},
                          {0, 8, 0, 4, refill},  {0, 10, 0, 4, refill}, {0, 8, 0, 5, refill}, {0, 10, 0, 5, refill},
                          {0, 12, 0, 5, refill}, {1, 10, 0, 5, 4}};
    rbr_status st = ensure(ctx, ctx->stage_out, size_t(n) * (any_hit ? 1 : sizeof(rbr_hit)), "autotune output");
    if (st != RBR_OK) return st;
    const Cand saved{ctx->trace_kernel, ctx->trace_min_blocks, ctx->trace_blocks_per_sm, ctx->trace_order, refill};
    float best_ms = 1e30f;
    Cand best = saved;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    for (const Cand& c : cands) {
        ctx->trace_kernel = c.kernel;
        ctx->trace_min_blocks = c.min_blocks;
        ctx->trace_blocks_per_sm = c.per_sm;
        ctx->trace_order = c.order;
        ctx->trace_refill_min = c.refill;
        cudaError_t e = launch_trace(ctx, rays, n, any_hit, ctx->stage_out.ptr, ctx->stream);  // warm-up
        float ms = 0.0f, total = 0.0f;
        for (int k = 0; k < 3 && e == cudaSuccess; ++k) {
            cudaEventRecord(a, ctx->stream);
            e = launch_trace(ctx, rays, n, any_hit, ctx->stage_out.ptr, ctx->stream);
            cudaEventRecord(b, ctx->stream);
            cudaEventSynchronize(b);
            cudaEventElapsedTime(&ms, a, b);
            total += ms;
        }
        if (e != cudaSuccess) {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
            ctx->trace_kernel = saved.kernel;
            ctx->trace_min_blocks = saved.min_blocks;
            ctx->trace_blocks_per_sm = saved.per_sm;
            ctx->trace_order = saved.order;
            ctx->trace_refill_min = saved.refill;
            return cuda_fail(ctx, e, "autotune launch");
        }
        if (total < best_ms) {
            best_ms = total;
            best = c;
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    ctx->trace_kernel = best.kernel;
    ctx->trace_min_blocks = best.min_blocks;
    ctx->trace_blocks_per_sm = best.per_sm;
    ctx->trace_order = best.order;
    ctx->trace_refill_min = best.refill;
    if (chosen_ms_x1000) *chosen_ms_x1000 = static_cast<int64_t>(best_ms / 3.0f * 1000.0f);
    return check_device_error(ctx, ctx->stream);
}

cudaError_t launch_trace_counts(const DeviceScene& s, const rbr_ray* rays, uint32_t n, int any_hit,
                                unsigned long long* totals, int* err, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const uint32_t blocks = (n + kTraceBlock - 1) / kTraceBlock;
    if (any_hit)
        k_trace_count<true><<<blocks, kTraceBlock, 0, stream>>>(s, reinterpret_cast<const float4*>(rays), n, totals, err);
    else
        k_trace_count<false><<<blocks, kTraceBlock, 0, stream>>>(s, reinterpret_cast<const float4*>(rays), n, totals, err);
    return cudaGetLastError();
}

}  // namespace rbr
