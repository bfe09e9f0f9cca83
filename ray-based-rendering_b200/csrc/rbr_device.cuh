// Device-side scene view, exact float helpers and the 8-wide BVH traversal.
//
// Primitive tests restate the reference operation for operation with explicitly rounded
// intrinsics (__fmul_rn/__fadd_rn/__fsub_rn/__fdiv_rn/__fsqrt_rn never fuse into an FMA), so
// a GPU hit distance equals the reference's bit for bit:
//   Triangle::intersect  src/geometry/triangle.cpp:6-24   (Moller-Trumbore, |a| < EPSILON cull)
//   Sphere::intersect    src/geometry/sphere.cpp:6-19
//   Quad::intersect      src/geometry/quad.cpp:12-28
//   Plane::intersect     src/geometry/plane.cpp:12-20
// Closest hit keeps the smallest t and, at equal t, the highest primitive id: exactly what a
// loop over Scene::primitives() in order returns (a later primitive at t == tMax replaces an
// earlier one because only t > tMax is rejected).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rbr_layout.h"
#include "rbr_scene_dev.h"

namespace rbr {

// ----------------------------------------------------------------------------------------
// Exactly rounded float3 arithmetic (the reference's Vec3, include/render/core/vector.h)
// ----------------------------------------------------------------------------------------
struct f3 {
    float x, y, z;
};

__device__ __forceinline__ f3 mk(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 xsub(f3 a, f3 b) { return mk(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
__device__ __forceinline__ f3 xadd(f3 a, f3 b) { return mk(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)); }
__device__ __forceinline__ f3 xmuls(f3 a, float s) { return mk(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s)); }
__device__ __forceinline__ f3 xmul(f3 a, f3 b) { return mk(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z)); }
__device__ __forceinline__ f3 xneg(f3 a) { return mk(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float xdot(f3 a, f3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ f3 xcross(f3 a, f3 b) {
    return mk(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
              __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}
// Vec3::operator/(float): multiply by the rounded reciprocal
__device__ __forceinline__ f3 xdivs(f3 a, float s) { return xmuls(a, __fdiv_rn(1.0f, s)); }
__device__ __forceinline__ float xlen(f3 a) { return __fsqrt_rn(xdot(a, a)); }
__device__ __forceinline__ f3 xnorm(f3 a) {
    const float l = xlen(a);
    return l > 0.0f ? xdivs(a, l) : mk(0.0f, 0.0f, 0.0f);
}
__device__ __forceinline__ f3 ld3(const float* p) { return mk(p[0], p[1], p[2]); }

// ----------------------------------------------------------------------------------------
// Primitive tests. `tbest`/`best` hold the current closest hit (best = -1: none yet).
// Each returns the candidate t (or a negative value for no hit); acceptance with the tie rule
// happens in accept().
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ bool accept(float t, uint32_t id, float tbest, int best) {
    return t < tbest || (t == tbest && static_cast<int>(id) > best);
}

// Triangle::intersect (triangle.cpp:6-24). v0, e1 = v1 - v0, e2 = v2 - v0.
__device__ __forceinline__ float hit_triangle(f3 o, f3 d, f3 v0, f3 e1, f3 e2, float tmax, float* pu = nullptr,
                                              float* pv = nullptr) {
    const f3 h = xcross(d, e2);
    const float a = xdot(e1, h);
    if (fabsf(a) < kEpsilon) return -1.0f;
    const float f = __fdiv_rn(1.0f, a);
    const f3 s = xsub(o, v0);
    const float u = __fmul_rn(f, xdot(s, h));
    if (u < 0.0f || u > 1.0f) return -1.0f;
    const f3 q = xcross(s, e1);
    const float v = __fmul_rn(f, xdot(d, q));
    if (v < 0.0f || __fadd_rn(u, v) > 1.0f) return -1.0f;
    const float t = __fmul_rn(f, xdot(e2, q));
    if (t < kEpsilon || t > tmax) return -1.0f;
    if (pu) {
        *pu = u;
        *pv = v;
    }
    return t;
}

// Sphere::intersect (sphere.cpp:6-19): near root, else far root, both within [EPSILON, tmax].
__device__ __forceinline__ float hit_sphere(f3 o, f3 d, f3 c, float r2, float tmax) {
    const f3 oc = xsub(o, c);
    const float a = xdot(d, d);
    const float halfB = xdot(oc, d);
    const float cc = __fsub_rn(xdot(oc, oc), r2);
    const float disc = __fsub_rn(__fmul_rn(halfB, halfB), __fmul_rn(a, cc));
    if (disc < 0.0f) return -1.0f;
    const float sq = __fsqrt_rn(disc);
    float t = __fdiv_rn(__fsub_rn(-halfB, sq), a);
    if (t < kEpsilon || t > tmax) {
        t = __fdiv_rn(__fadd_rn(-halfB, sq), a);
        if (t < kEpsilon || t > tmax) return -1.0f;
    }
    return t;
}

// fd(x, y) < 0 or > 1 for y >= 0, without the division (the same answer for every x, zero, infinite and
// NaN operands included): the rounded quotient exceeds 1 exactly if x > y, since then x >= y + ulp(y) and
// ulp(y) > 2^-24 y; it is below 0 if x is and the quotient does not round to -0 (|x| <= 2^-150 y).
__device__ __forceinline__ bool outside01(float x, float y) {
    return x > y || (x < 0.0f && -x * 1.267650600e30f > y * 8.881784197e-16f);  // 2^100, 2^-50
}

// Quad::intersect (quad.cpp:12-28); n is the normal as the constructor computes it. The record
// tests of a Cornell box bound its rays, and the normal's root and quotient and the two quotients of
// the edge coordinates were half of this test's instructions: without them the Cornell box went from
// 822 to 746 us, the foggy one from 1,499 to 1,279.
__device__ __forceinline__ float hit_quad(f3 o, f3 d, f3 org, f3 u, f3 v, f3 n, float ulen2, float vlen2, float tmax) {
    const float denom = xdot(n, d);
    if (fabsf(denom) < kEpsilon) return -1.0f;
    const float t = __fdiv_rn(xdot(xsub(org, o), n), denom);
    if (t < kEpsilon || t > tmax) return -1.0f;
    const f3 hp = xadd(o, xmuls(d, t));
    const f3 lp = xsub(hp, org);
    if (outside01(xdot(lp, u), ulen2) || outside01(xdot(lp, v), vlen2)) return -1.0f;
    return t;
}

// Plane::intersect (plane.cpp:12-20).
__device__ __forceinline__ float hit_plane(f3 o, f3 d, f3 n, float pd, float tmax) {
    const float denom = xdot(n, d);
    if (fabsf(denom) < kEpsilon) return -1.0f;
    const float t = __fdiv_rn(-__fadd_rn(xdot(n, o), pd), denom);
    if (t < kEpsilon || t > tmax) return -1.0f;
    return t;
}

// Tests leaf record `rec`; returns t or negative. `tag` receives the record's tag word.
__device__ __forceinline__ float hit_record(const DeviceScene& s, uint32_t rec, f3 o, f3 d, float tmax, uint32_t& tag) {
    const float4 a = __ldg(s.records + 3 * rec);
    const float4 b = __ldg(s.records + 3 * rec + 1);
    const float4 c = __ldg(s.records + 3 * rec + 2);
    tag = __float_as_uint(c.y);
    const uint32_t type = tag >> kTypeShift;
    if (type == kPrimTriangle) {
        return hit_triangle(o, d, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, c.x), tmax);
    } else if (type == kPrimSphere) {
        return hit_sphere(o, d, mk(a.x, a.y, a.z), b.x, tmax);
    } else {
        const float4 q = __ldg(s.quads + __float_as_uint(c.z));  // normal, |u|^2
        return hit_quad(o, d, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, c.x), mk(q.x, q.y, q.z), q.w, c.w, tmax);
    }
}

// ----------------------------------------------------------------------------------------
// 8-wide node test
//
// The traversal is bound by instruction issue and by the ALU pipe (byte permutes, min / max,
// compares, mask logic), not by memory, so the test is arranged to issue few of those:
//   - Slab distances are taken in units of the ray's current limit T, so one saturating FMA per
//     far plane and one saturating product for the near ones clamp them to [0, 1]: a box is hit if near < far, with no separate comparison
//     against 0 and T (a box behind the origin or past the limit has near = far = 0 or 1).
//   - near - far is one FADD whose sign bit a funnel shift appends to the hit mask: no compare,
//     no predicated OR.
//   - The byte selectors carry the ray's octant (its low two bits) and the two words of a plane
//     row its high bit, so the mask comes out in visiting order without a permutation; the node
//     stores its mask of internal slots permuted for every octant.
//   - Leaf records are looked up when a leaf slot is visited, not for every slot.
// 17 instructions per slot (9 on the ALU pipe) where a test with separate clamps that builds the
// record mask slot by slot takes 23 (15). Measured against that test: 2^22 uniform rays through
// 1.3M triangles 1,827 -> 1,430 us, 2M camera rays 607 -> 450 us, 1.5M shadow segments 340 -> 282
// us, the 1080p GGX render at 64 spp 128.6 -> 106.9 ms, Cornell box 908 -> 884 us (bound by the
// latency of its record tests). Not kept: leaf slots walked inside the record loop (see
// leaf_records).
// ----------------------------------------------------------------------------------------
struct RayCtx {
    float ix, iy, iz;  // 1 / (d T)
    float qx, qy, qz;  // o / (d T)
    uint32_t oct;      // bit k set: d_k negative (visiting order)
};

// Near distances are lowered by 2^-16 of themselves: covers the rounding of a plane's distance that
// grows with the distance (2^-22 of it) and that of the primitive tests near a box face. What grows
// with the node instead (2^-9 grid steps in each rounding of the biased offset and factor) lies within
// kQuantMargin. The widening must not grow with T: 2^-16 of the limit, which for a ray without one is
// the reach of the whole tree, is more than the leaves of a small mesh in a large scene (330 K triangles
// of radius 1 over a ground of half size 20,000: 405 nodes and 6,263 records a ray from the mesh where
// this takes 21 nodes and 125 records; 2^20 rays 84 ms against 2.3). One product per slot with the largest
// near distance: scaled factors and offsets of the planes take six registers more, and the path tracer's
// kernels spill (256x256 Cornell box, 16 spp, 722 us, 719 so; 64x48 preview 154 both; 2^22 uniform rays
// 1,039 and 1,044).
constexpr float kNearScale = 1.0f - 1.0f / 65536.0f;

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 1 / (d T) with |d T| raised to at least 2^-64 (sign kept). With an exact zero component the
// slab distances of that axis would be q*inf + (-inf) = NaN: every box the ray crosses in the
// other two axes would pass, a traversal of much of the tree. With 2^64 the distances stay
// finite and the axis is tested by containment, as the reference's BoundingBox::intersect does
// for a zero component (include/render/acceleration/bbox.h:92-120). Boxes stay conservative: the
// ray moves by less than 2^-64 over [0, T], far below the boxes' padding.
__device__ __forceinline__ float safe_inv(float d, float T) {
    return rcp_approx(copysignf(fmaxf(fabsf(d * T), 5.421010862e-20f), d));
}

// Scales the slab arithmetic to the limit T: every box that starts before T may be hit.
__device__ __forceinline__ void set_limit(RayCtx& r, f3 o, f3 d, float T) {
    r.ix = safe_inv(d.x, T);
    r.iy = safe_inv(d.y, T);
    r.iz = safe_inv(d.z, T);
    r.qx = o.x * r.ix;
    r.qy = o.y * r.iy;
    r.qz = o.z * r.iz;
}

// `tmax` (infinite, NaN and huge values included) is lowered to a finite limit no hit can lie
// beyond: the distance from the origin to the centre of the tree's box plus the box's half
// extents, in the 1-norm, over the largest direction component. Limits below the tests'
// EPSILON cull are raised to 1e-5 (no hit either way).
__device__ __forceinline__ RayCtx make_ctx(const DeviceScene& s, f3 o, f3 d, float tmax) {
    RayCtx r;
    r.oct = (signbit(d.x) ? 1u : 0u) | (signbit(d.y) ? 2u : 0u) | (signbit(d.z) ? 4u : 0u);
    const float reach = fabsf(o.x - s.tree_centre[0]) + fabsf(o.y - s.tree_centre[1]) + fabsf(o.z - s.tree_centre[2]) +
                        s.tree_reach;
    const float far = 1.01f * reach * rcp_approx(fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fmaxf(fabsf(d.z), 1e-30f)));
    set_limit(r, o, d, fmaxf(fminf(fminf(tmax, far), 1e30f), 1e-5f));
    return r;
}

// kGridBias + (byte of `word` the selector names), exactly: one byte permute of the byte into
// bits 8-15 of the mantissa of 32768.0f (bits 0x47000000). Selector 0x7404 | (byte << 4).
__device__ __forceinline__ float qplane(uint32_t word, uint32_t sel) {
    return __uint_as_float(__byte_perm(word, kGridBiasBits, sel));
}

// a * b + c clamped to [0, 1] (NaN to 0).
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float mul_sat(float a, float b) {
    float d;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// Three-input minimum / maximum (sm_100).
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// One 32-byte sector of a node in one load (sm_100: 256-bit loads).
struct Words8 {
    uint32_t w[8];
};
__device__ __forceinline__ Words8 ld_sector(const uint4* p) {
    Words8 v;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7])
        : "l"(p));
    return v;
}

// What a traversal keeps of a node: its children, its leaves, and the slots the ray hits, all
// masks of 8 bits in visiting order (bit j is slot j ^ octant, visited from bit 7 down).
struct NodeHits {
    uint32_t child_base, prim_base;
    uint32_t meta0, meta1;  // per slot byte of a leaf: (records << 5) | first record offset
    uint32_t imask;         // internal slots, by slot
    uint32_t inner, leaf;   // slots hit
};

// Per node and ray: the slab arithmetic of the node's grid. Plane byte q of axis k is hit at
// (kGridBias + q) a_k + b_k (in units of T) with a_k = step_k / (d_k T), b_k = (p_k - o_k) / (d_k T).
// b comes from one FMA of p with the ray's o / (d T): its rounding error, 2^-24 o / d, stays below
// the 2^-20 of the scene's largest coordinate every box is padded with, plus the widening in t.
struct NodeView {
    float ax, ay, az, bx, by, bz;                       // factors, offsets
    uint32_t px[2], Px[2], py[2], Py[2], pz[2], Pz[2];  // near (p) and far (P) plane bytes, 8 slots
};

__device__ __forceinline__ NodeView node_view(const uint4* __restrict__ nodes, uint32_t idx, const RayCtx& r,
                                              NodeHits& h, uint32_t& perm_inner) {
    const uint4* np = nodes + (kDevNodeWords / 4) * static_cast<size_t>(idx);
    const Words8 A = ld_sector(np), B = ld_sector(np + 2), C = ld_sector(np + 4);
    NodeView v;
    v.ax = __uint_as_float(C.w[6] << 16) * r.ix;
    v.ay = __uint_as_float(C.w[6] & 0xFFFF0000u) * r.iy;
    v.az = __uint_as_float(C.w[7]) * r.iz;
    v.bx = fmaf(__uint_as_float(A.w[0]), r.ix, -r.qx);
    v.by = fmaf(__uint_as_float(A.w[1]), r.iy, -r.qy);
    v.bz = fmaf(__uint_as_float(A.w[2]), r.iz, -r.qz);
    const bool sx = r.oct & 1u, sy = r.oct & 2u, sz = r.oct & 4u;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        v.px[w] = sx ? B.w[2 + w] : B.w[w];
        v.Px[w] = sx ? B.w[w] : B.w[2 + w];
        v.py[w] = sy ? B.w[6 + w] : B.w[4 + w];
        v.Py[w] = sy ? B.w[4 + w] : B.w[6 + w];
        v.pz[w] = sz ? C.w[2 + w] : C.w[w];
        v.Pz[w] = sz ? C.w[w] : C.w[2 + w];
    }
    h.imask = A.w[3];
    h.child_base = A.w[4];
    h.prim_base = A.w[5];
    h.meta0 = A.w[6];
    h.meta1 = A.w[7];
    perm_inner = __byte_perm(C.w[4], C.w[5], r.oct);  // low byte: internal slots in visiting order
    return v;
}

// near - far of the slot whose plane bytes lie in word w at selector sel: negative if hit.
__device__ __forceinline__ float slot_gap(const NodeView& v, int w, uint32_t sel) {
    const float n = fmax3(fmaf(qplane(v.px[w], sel), v.ax, v.bx), fmaf(qplane(v.py[w], sel), v.ay, v.by),
                          fmaf(qplane(v.pz[w], sel), v.az, v.bz));
    const float f = fmin3(fma_sat(qplane(v.Px[w], sel), v.ax, v.bx), fma_sat(qplane(v.Py[w], sel), v.ay, v.by),
                          fma_sat(qplane(v.Pz[w], sel), v.az, v.bz));
    return mul_sat(n, kNearScale) - f;
}

// Tests the 8 children of node `idx`.
__device__ __forceinline__ NodeHits intersect_node(const uint4* __restrict__ nodes, uint32_t idx, const RayCtx& r) {
    NodeHits h;
    uint32_t pin;
    const NodeView v = node_view(nodes, idx, r, h, pin);
    const uint32_t sel0 = 0x7404u | ((r.oct & 3u) << 4);
    uint32_t m0 = 0, m1 = 0;  // slots 0-3 and 4-7
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        const uint32_t sel = sel0 ^ (static_cast<uint32_t>(k) << 4);
        m0 = __funnelshift_l(__float_as_uint(slot_gap(v, 0, sel)), m0, 1);
        m1 = __funnelshift_l(__float_as_uint(slot_gap(v, 1, sel)), m1, 1);
    }
    const uint32_t m = (r.oct & 4u) ? (m0 << 4) | m1 : (m1 << 4) | m0;
    h.inner = m & pin;
    h.leaf = m & ~pin;
    return h;
}

// Internal slots still to visit, packed with the internal mask: (mask << 8) | imask.
__device__ __forceinline__ uint2 node_group(const NodeHits& h) { return make_uint2(h.child_base, (h.inner << 8) | h.imask); }

// Takes the next child (nearest first) out of a non-empty group.
__device__ __forceinline__ uint32_t next_child(uint2& g, uint32_t oct) {
    const uint32_t b = 31u - static_cast<uint32_t>(__clz(static_cast<int>(g.y)));
    g.y ^= 1u << b;
    const uint32_t slot = (b - 8u) ^ oct;
    return g.x + __popc(g.y & ((1u << slot) - 1u));
}

// Mask of (width mod 32) bits starting at bit (pos mod 32). PTX's bmsk.wrap uses the low five
// bits of both operands, so a byte of a leaf's meta word can be passed as it is.
__device__ __forceinline__ uint32_t bitmask_at(uint32_t pos, uint32_t width) {
    uint32_t d;
    asm("bmsk.wrap.b32 %0, %1, %2;" : "=r"(d) : "r"(pos), "r"(width));
    return d;
}

// The records (bit r: record prim_base + r) of the leaf slots hit; none for an empty slot that the
// widening alone let through. One mask of records keeps the lanes of a warp together in the record
// loop that follows: walking the slots inside that loop splits the warp by the sizes of the lanes'
// leaves (Cornell box 909 -> 1,143 us).
__device__ __forceinline__ uint32_t leaf_records(const NodeHits& h, uint32_t oct) {
    uint32_t leaf = h.leaf, recs = 0;
    while (leaf != 0) {
        const uint32_t b = 31u - static_cast<uint32_t>(__clz(static_cast<int>(leaf)));
        leaf ^= 1u << b;
        const uint32_t meta = __byte_perm(h.meta0, h.meta1, b ^ oct) & 0xFFu;
        recs |= bitmask_at(meta, meta >> 5);
    }
    return recs;
}

// ----------------------------------------------------------------------------------------
// Traversal. Closest hit: returns the primitive id (or RBR_MISS) and its t.
// Any hit: returns 1 as soon as a primitive lies in [EPSILON, tmax].
// ----------------------------------------------------------------------------------------
// With kCount, `counts` receives the number of wide nodes fetched (x) and leaf records
// tested (y) by this ray: the traversal is deterministic per ray, so these are the ray's
// algorithmic node and record traffic.
template <bool kAny, bool kCount = false>
__device__ __forceinline__ uint32_t traverse(const DeviceScene& s, f3 o, f3 d, float tmax, float& thit, int* err,
                                             uint2* counts = nullptr) {
    float tbest = tmax;
    int best = -1;
    for (uint32_t i = 0; i < s.num_planes; ++i) {
        const float4 pl = __ldg(s.planes + i);
        const float t = hit_plane(o, d, mk(pl.x, pl.y, pl.z), pl.w, tbest);
        if (t >= 0.0f) {
            const uint32_t id = __ldg(s.plane_tags + i) & kIdMask;
            if (kAny) return 1u;
            if (accept(t, id, tbest, best)) {
                tbest = t;
                best = static_cast<int>(id);
            }
        }
    }
    if (s.num_nodes != 0) {
        RayCtx r = make_ctx(s, o, d, tbest);
        uint2 stack[kStackSize];
        int sp = 0;
        uint32_t node = 0;
        while (true) {
            const NodeHits h = intersect_node(s.nodes, node, r);
            if (kCount) counts->x += 1;
            uint2 ng = node_group(h);
            uint32_t recs = leaf_records(h, r.oct);
            bool closer = false;
            while (recs != 0) {
                const uint32_t rec = h.prim_base + static_cast<uint32_t>(__ffs(static_cast<int>(recs)) - 1);
                recs &= recs - 1;
                if (kCount) counts->y += 1;
                uint32_t tag;
                const float t = hit_record(s, rec, o, d, tbest, tag);
                if (t >= 0.0f) {
                    if (kAny) return 1u;
                    const uint32_t id = tag & kIdMask;
                    if (accept(t, id, tbest, best)) {
                        tbest = t;
                        best = static_cast<int>(id);
                        closer = true;
                    }
                }
            }
            if (!kAny && closer) set_limit(r, o, d, tbest);
            if (ng.y < 256u) {
                if (sp == 0) break;
                ng = stack[--sp];
            }
            node = next_child(ng, r.oct);
            if (ng.y >= 256u) {
                if (sp < kStackSize) {
                    stack[sp++] = ng;
                } else {
                    atomicOr(err, kErrStackOverflow);
                    break;
                }
            }
        }
    }
    if (kAny) return 0u;
    thit = tbest;
    return best < 0 ? 0xFFFFFFFFu : static_cast<uint32_t>(best);
}

// ----------------------------------------------------------------------------------------
// Warp traversal: 32 rays advance together, one node each per step, and the leaf records that the
// lanes found in a step go through a queue in shared memory to all 32 lanes of the warp. A ray
// finds a record in every third node or so; tested by the lanes that found them, the records took
// 2.5 rounds of some 140 instructions a step with 3 of 32 lanes active, 60 % of the instructions
// of incoherent closest-hit queries. Through the queue a step takes one round (10 records on
// average). A lane whose ray is done can be given another one between steps, so the warp does not
// idle behind its longest ray: 2^22 uniform rays through 1.3M triangles 1,305 us with refilled lanes
// alone, 1,135 with the queue filled by ballots a record at a time, 1,065 by a prefix sum of counts.
// Every lane of the warp takes part in every call.
// ----------------------------------------------------------------------------------------
constexpr uint32_t kNoHit = 0xFFFFFFFFu;

struct WarpRays {
    float4 o[32];                  // origin, t of the closest hit so far (or tmax)
    float4 d[32];                  // direction
    unsigned long long best[32];   // closest: (t bits << 32) | (kIdMask - id), low word kNoHit before a hit;
                                   // any hit: nonzero once a primitive is hit
    uint2 item[64];                // (record, lane) waiting for their tests
};

struct LaneRay {
    RayCtx r;
    uint32_t node;  // the next node to test
    int sp;
};

__device__ __forceinline__ uint32_t hit_prim(unsigned long long best) {
    const uint32_t low = static_cast<uint32_t>(best);
    return low == kNoHit ? 0xFFFFFFFFu : kIdMask - low;
}
__device__ __forceinline__ uint32_t hit_tbits(unsigned long long best) { return static_cast<uint32_t>(best >> 32); }

// Gives this lane a ray (called by the lanes that take one). Returns true if it is already
// complete: an any-hit ray that hits a plane, no BVH, or a closest-hit limit that is NaN (which
// no distance is below).
template <bool kAny>
__device__ __forceinline__ bool lane_begin(const DeviceScene& s, WarpRays& w, f3 o, f3 d, float tmax, LaneRay& lr) {
    const uint32_t lane = threadIdx.x & 31u;
    float tbest = tmax;
    int best = -1;
    for (uint32_t i = 0; i < s.num_planes; ++i) {
        const float4 pl = __ldg(s.planes + i);
        const float t = hit_plane(o, d, mk(pl.x, pl.y, pl.z), pl.w, tbest);
        if (t >= 0.0f) {
            const uint32_t id = __ldg(s.plane_tags + i) & kIdMask;
            if (kAny) {
                w.best[lane] = 1u;
                return true;
            }
            if (accept(t, id, tbest, best)) {
                tbest = t;
                best = static_cast<int>(id);
            }
        }
    }
    w.best[lane] = kAny ? 0u
                        : (static_cast<unsigned long long>(__float_as_uint(tbest)) << 32) |
                              (best < 0 ? kNoHit : kIdMask - static_cast<uint32_t>(best));
    if (s.num_nodes == 0 || (!kAny && !(tbest == tbest))) return true;
    w.o[lane] = make_float4(o.x, o.y, o.z, tbest);
    w.d[lane] = make_float4(d.x, d.y, d.z, 0.0f);
    lr.r = make_ctx(s, o, d, tbest);
    lr.sp = 0;
    lr.node = 0;
    return false;
}

// Tests leaf record `rec` against the ray of lane `owner`; true for a hit.
template <bool kAny>
__device__ __forceinline__ bool test_record(const DeviceScene& s, WarpRays& w, uint32_t rec, uint32_t owner) {
    const float4 o = w.o[owner], d = w.d[owner];
    uint32_t tag;
    const float t = hit_record(s, rec, mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), o.w, tag);
    if (!(t >= 0.0f)) return false;
    if (kAny)
        w.best[owner] = 1u;
    else
        atomicMin(&w.best[owner],
                  (static_cast<unsigned long long>(__float_as_uint(t)) << 32) | (kIdMask - (tag & kIdMask)));
    return true;
}

// One step of the warp: every lane with `active` tests its node, then the warp tests the records
// found. Returns true for a lane whose ray is complete.
template <bool kAny>
__device__ __forceinline__ bool warp_step(const DeviceScene& s, WarpRays& w, bool active, LaneRay& lr, uint2* stack,
                                          int* err) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    uint32_t recs = 0, prim_base = 0;
    bool done = false;
    if (active) {
        const NodeHits h = intersect_node(s.nodes, lr.node, lr.r);
        uint2 ng = node_group(h);
        recs = leaf_records(h, lr.r.oct);
        prim_base = h.prim_base;
        if (ng.y < 256u) {
            if (lr.sp == 0) done = true;
            else ng = stack[--lr.sp];  // only non-empty groups are pushed
        }
        if (!done) {
            lr.node = next_child(ng, lr.r.oct);
            if (ng.y >= 256u) {
                if (lr.sp < kStackSize) {
                    stack[lr.sp++] = ng;
                } else {
                    atomicOr(err, kErrStackOverflow);
                    done = true;
                }
            }
        }
    }
    bool any = false;
    const bool with = __any_sync(0xFFFFFFFFu, recs != 0);
    // 64 records at a time
    if (with) {
        const uint32_t mine = __popc(recs);
        uint32_t first = 0, total = 0;  // exclusive prefix of the lanes' counts, and their sum
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, (mine >> k) & 1u);
            first += __popc(m & lt) << k;
            total += __popc(m) << k;
        }
        if (__any_sync(0xFFFFFFFFu, mine > 7u)) {
#pragma unroll
            for (int k = 3; k < 6; ++k) {
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, (mine >> k) & 1u);
                first += __popc(m & lt) << k;
                total += __popc(m) << k;
            }
        }
        for (uint32_t base = 0; base < total; base += 64u) {
            while (recs != 0 && first < base + 64u) {
                const uint32_t b = 31u - static_cast<uint32_t>(__clz(static_cast<int>(recs)));
                recs ^= 1u << b;
                w.item[first - base] = make_uint2(prim_base + b, lane);
                ++first;
            }
            __syncwarp();
            const uint32_t n = min(64u, total - base);
            for (uint32_t k = 0; k < n; k += 32u) {
                bool hit = false;
                if (k + lane < n) {
                    const uint2 it = w.item[k + lane];
                    hit = test_record<kAny>(s, w, it.x, it.y);
                }
                any |= __any_sync(0xFFFFFFFFu, hit);
            }
            __syncwarp();
        }
    }
    if (any) {
        __syncwarp();
        const unsigned long long b = w.best[lane];
        if (kAny) {
            if (active && b != 0) done = true;
        } else if (active && !done) {
            const float t = __uint_as_float(hit_tbits(b));
            const float4 o = w.o[lane];
            if (t < o.w) {
                const float4 d = w.d[lane];
                w.o[lane].w = t;
                set_limit(lr.r, mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), t);
            }
        }
    }
    return done;
}

// ----------------------------------------------------------------------------------------
// Group traversal: 8 lanes trace one ray. In a node step lane j tests the slot visited j-th from
// last (slot j ^ octant) and a ballot gives the hit mask; then each lane whose slot is a leaf the
// ray hits tests that leaf's records, and a shuffle minimum (key = t bits, then the highest id)
// keeps the closest. State is replicated in the 8 lanes, so the group never diverges internally.
// A step's dependent chain is one slot and one leaf long instead of eight slots and all leaves,
// and a warp waits for the longest of 4 rays instead of 32: the shorter latency for few rays.
// ----------------------------------------------------------------------------------------
struct GroupLanes {
    uint32_t j;     // lane within the group
    uint32_t shift; // first lane of the group
    uint32_t mask;  // the group's lanes
};
__device__ __forceinline__ GroupLanes group_lanes() {
    const uint32_t lane = threadIdx.x & 31u;
    return GroupLanes{lane & 7u, lane & 24u, 0xFFu << (lane & 24u)};
}

struct GroupRay {
    RayCtx r;
    f3 o, d;
    float tbest;
    int best;
    uint32_t node;  // the next node to test
    int sp;
};

// Starts a ray: planes, then the root node is next. Returns true if the ray is already complete
// (any hit on a plane, or no BVH).
template <bool kAny>
__device__ __forceinline__ bool group_begin(const DeviceScene& s, f3 o, f3 d, float tmax, GroupRay& st,
                                            uint32_t& anyhit) {
    st.o = o;
    st.d = d;
    st.tbest = tmax;
    st.best = -1;
    anyhit = 0;
    for (uint32_t i = 0; i < s.num_planes; ++i) {
        const float4 pl = __ldg(s.planes + i);
        const float t = hit_plane(o, d, mk(pl.x, pl.y, pl.z), pl.w, st.tbest);
        if (t >= 0.0f) {
            const uint32_t id = __ldg(s.plane_tags + i) & kIdMask;
            if (kAny) {
                anyhit = 1;
                return true;
            }
            if (accept(t, id, st.tbest, st.best)) {
                st.tbest = t;
                st.best = static_cast<int>(id);
            }
        }
    }
    if (s.num_nodes == 0) return true;
    st.r = make_ctx(s, o, d, st.tbest);
    st.sp = 0;
    st.node = 0;
    return false;
}

// One step of the group's ray; returns true when it is complete (anyhit: a primitive was hit).
template <bool kAny>
__device__ __forceinline__ bool group_step(const DeviceScene& s, const GroupLanes& g, GroupRay& st, uint2* stack,
                                           int* err, uint32_t& anyhit) {
    NodeHits h;
    uint32_t pin;
    const NodeView v = node_view(s.nodes, st.node, st.r, h, pin);
    const uint32_t slot = g.j ^ st.r.oct;
    const uint32_t sel = 0x7404u | ((slot & 3u) << 4);
    const float gap = (slot & 4u) ? slot_gap(v, 1, sel) : slot_gap(v, 0, sel);
    const uint32_t m = (__ballot_sync(g.mask, gap < 0.0f) >> g.shift) & 0xFFu;
    h.inner = m & pin;
    h.leaf = m & ~pin;
    uint2 ng = node_group(h);
    if (h.leaf != 0) {
        unsigned long long key = ~0ull;
        if ((h.leaf >> g.j) & 1u) {
            const uint32_t meta = __byte_perm(h.meta0, h.meta1, slot) & 0xFFu;
            const uint32_t first = h.prim_base + (meta & 31u);
            for (uint32_t k = 0; k < (meta >> 5); ++k) {
                uint32_t tag;
                const float t = hit_record(s, first + k, st.o, st.d, st.tbest, tag);
                if (t >= 0.0f) {
                    const unsigned long long c =
                        (static_cast<unsigned long long>(__float_as_uint(t)) << 32) | (~(tag & kIdMask));
                    key = c < key ? c : key;
                }
            }
        }
        if (kAny) {
            if (__ballot_sync(g.mask, key != ~0ull) != 0) {
                anyhit = 1;
                return true;
            }
        } else {
            for (int off = 1; off < 8; off <<= 1) {
                const unsigned long long o2 = __shfl_xor_sync(g.mask, key, off, 8);
                key = o2 < key ? o2 : key;
            }
            if (key != ~0ull) {
                const float t = __uint_as_float(static_cast<uint32_t>(key >> 32));
                const uint32_t id = ~static_cast<uint32_t>(key) & kIdMask;
                if (accept(t, id, st.tbest, st.best)) {
                    st.tbest = t;
                    st.best = static_cast<int>(id);
                    set_limit(st.r, st.o, st.d, t);
                }
            }
        }
    }
    if (ng.y < 256u) {
        if (st.sp == 0) return true;
        ng = stack[--st.sp];
    }
    st.node = next_child(ng, st.r.oct);
    if (ng.y >= 256u) {
        if (st.sp < kStackSize) {
            stack[st.sp++] = ng;
        } else {
            atomicOr(err, kErrStackOverflow);
            return true;
        }
    }
    return false;
}

}  // namespace rbr
