// Memory layout of a scene (shared by the host builder and the kernels).
//
// Wide BVH node in device memory (96 B, three 32 B sectors, each read by one 256-bit load):
//   w0-w2    px, py, pz (f32): biased origin of the node's quantisation grid (as below)
//   w3       imask (bits 0-7): slots that hold an internal node
//   w4, w5   child_base, prim_base
//   w6, w7   per slot byte of a leaf: (records << 5) | offset of its first record from prim_base
//   w8-w19   per axis qlo[8], qhi[8]: child boxes in 8-bit grid coordinates
//   w20, w21 byte o: imask in the visiting order of octant o (bit j set if slot j ^ o is internal)
//   w22      grid steps of x (low half) and y (high half) as BF16 (powers of two, so exact)
//   w23      grid step of z as f32
// device_node() makes it from the builder's node:
//
// Wide BVH node of the builder (80 B, five 16 B words):
//   word0  px, py, pz (f32)      biased origin of the node's quantisation grid: plane byte q of
//                                axis k lies at p_k + (kGridBias + q) * 2^(e_k - 127), so one
//                                byte permute of q into the mantissa of 32768.0f gives the
//                                factor (kGridBias + q) as an exact float
//          ex|ey|ez|imask (u8)   biased exponents of the per-axis grid step 2^(e-127),
//                                imask bit s = slot s holds an internal node
//   word1  child_base (u32)      index of the first internal child (children are stored
//                                consecutively in slot order)
//          prim_base (u32)       index of the first leaf record of this node's leaves
//          meta[8] (u8)          per slot: (width << 5) | position of the slot's bits in the
//                                node's 32-bit hit mask -- leaf: width = record count (1..4),
//                                position = first record offset from prim_base; internal:
//                                width 1, position 24 + slot; empty: 0
//   word2  qlo_x[8], qlo_y[8]    child boxes, 8-bit grid coordinates, rounded outwards with a
//   word3  qlo_z[8], qhi_x[8]    margin of at least kQuantMargin grid steps
//   word4  qhi_y[8], qhi_z[8]
// Slot s holds the child whose centre lies furthest towards the octant whose axis k is
// negative when bit k of s is set, so a ray with direction-sign bits D visits children in
// decreasing order of (s ^ D): roughly front to back, without sorting. A ray XORs the
// position of an internal slot with D, so bits 24-31 of its hit mask are in visiting order.
// A node with internal children keeps its leaf records at offsets below 24 (bits 24-31 are
// the internal slots'); a node without internal children may use all 32 record bits.
//
// Leaf record (48 B, three 16 B words) in leaf order:
//   triangle  v0.xyz, e1.xyz, e2.xyz, tag      (e1 = v1 - v0, e2 = v2 - v0, rounded as
//                                               Triangle::intersect computes them)
//   sphere    centre.xyz, radius, r*r, -, -, -, -, -, tag
//   quad      origin.xyz, u.xyz, v.xyz, tag, index of its normal and dot(u,u), dot(v,v)
//   tag = primitive id | (type << 30)
// Planes (unbounded) live outside the tree: float4 (unit normal, d) + id.
#pragma once

#include <stdint.h>

namespace rbr {

constexpr uint32_t kPrimTriangle = 0;
constexpr uint32_t kPrimSphere = 1;
constexpr uint32_t kPrimQuad = 2;
constexpr uint32_t kPrimPlane = 3;
constexpr uint32_t kTypeShift = 30;
constexpr uint32_t kIdMask = (1u << kTypeShift) - 1;

constexpr int kNodeWords = 20;     // u32 words per wide node of the builder
constexpr int kDevNodeWords = 24;  // u32 words per wide node in device memory
constexpr int kRecordWords = 12; // u32 words per leaf record
constexpr int kMaxLeafPrims = 4;
constexpr int kStackSize = 64;   // traversal stack entries; the builder keeps the tree shallower
constexpr int kMaxTreeDepth = 62;
constexpr double kGridBias = 32768.0;        // plane byte q sits at grid coordinate kGridBias + q
constexpr uint32_t kGridBiasBits = 0x47000000u;  // 32768.0f
constexpr double kQuantMargin = 1.0 / 64.0;  // least outward rounding of a child plane, in grid steps
constexpr uint32_t kInnerRecordLimit = 24;   // records of a node that also has internal children

// Geometry constant of the reference (include/render/core/common.h:22).
constexpr float kEpsilon = 1e-4f;

// Device-side error bits (rbr_ctx::d_error).
constexpr int kErrStackOverflow = 1;
constexpr int kErrQueueOverflow = 2;
constexpr int kErrDeviceTimeout = 4;  // a bounded wait (tensor-core completion) ran out

// The device form of a builder node.
inline void device_node(const uint32_t* w, uint32_t* out) {
    const uint32_t imask = w[3] >> 24;
    uint32_t step[3], perm[8];
    for (int a = 0; a < 3; ++a) step[a] = ((w[3] >> (8 * a)) & 0xFFu) << 23;  // 2^(e - 127) as f32 bits
    for (uint32_t o = 0; o < 8; ++o) {
        perm[o] = 0;
        for (uint32_t j = 0; j < 8; ++j) perm[o] |= ((imask >> (j ^ o)) & 1u) << j;
    }
    for (int a = 0; a < 3; ++a) out[a] = w[a];
    out[3] = imask;
    for (int k = 4; k < 8; ++k) out[k] = w[k];
    for (int a = 0; a < 3; ++a)
        for (int k = 0; k < 2; ++k) {
            out[8 + 4 * a + k] = w[8 + 2 * a + k];
            out[10 + 4 * a + k] = w[14 + 2 * a + k];
        }
    out[20] = perm[0] | perm[1] << 8 | perm[2] << 16 | perm[3] << 24;
    out[21] = perm[4] | perm[5] << 8 | perm[6] << 16 | perm[7] << 24;
    out[22] = (step[0] >> 16) | (step[1] & 0xFFFF0000u);
    out[23] = step[2];
}

}  // namespace rbr
