// aur_wide.cuh — the NMH traversed two levels at a time.
//
// A wide node (a treelet) is an NMH node with its two children: their six
// triangles and the four grandchild subtrees, each as an axis-aligned box
// quantised outward to 8 bits per plane on a grid over the treelet. A ray
// tests ten boxes per 96-byte record, then runs Moller-Trumbore only on the
// triangles whose own box it meets; the walk of intersect() instead tests a
// slab, two triangles and two boxes per NMH node, at a 128-byte record each.
//
// Results are those of intersect() / intersectAny() (kernels/lib/
// intersect.cuh:36-152) bit for bit. What the boxes decide is only which
// triangles are tested, and they are conservative (padding below), so every
// triangle that walk can accept is tested here with the same arithmetic. That
// walk also leaves out triangles whose node its slab ranges miss; those
// decisions are checked after the fact, for the one triangle a ray reports
// (finish_closest / finish_any below).
//
// One kind of closest hit no box can vouch for: a triangle met edge-on, within
// about 1e-6 rad of its plane, where the t that Moller-Trumbore computes is
// rounding noise and can lie far from the triangle. intersect() takes such a t
// when it is the smallest; here the triangle is left out when its box lies
// behind the nearest other hit. (Rays made to graze so, det 1e-7 to 1e-6 with
// edges of 1 and origins up to 30 away: 0.5 to 0.9 % of 20,000 closest hits;
// 0.2 to 0.3 % in the node-by-node walk with its boxes. No any hit.)
//
// Small boxes on a grid of their node, a byte a plane, are those of compressed
// wide BVHs (Ylitie, Karras, Laine, "Efficient incoherent ray traversal on GPUs
// through compressed wide BVHs", HPG'17); tree, record and walk are the NMH's.
//
// Record of treelet i on its level (24 words; 16-byte aligned, read as
// 32-byte sectors):
//   0..2   o       3..5  cell size s   (plane of byte q: o + (1024 + q) * s)
//   6..11  planes (x lo, x hi, y lo, y hi, z lo, z hi) of triangles 0..3,
//          one byte each: the node's pair, then the first child's pair
//   12..14 per axis: lo, lo, hi, hi bytes of triangles 4, 5 (second child)
//   15     bits 0-5: triangle exists; bits 8-11: grandchild subtree exists
//   16..21 planes as words 6..11 of the four grandchild subtrees
// Treelets at the bottom have no grandchildren: their words 16..23 are not
// written, and nothing read from them counts.
//
// Treelet roots sit on every other heap level, chosen so that the bottom
// level is always the second level of a treelet: with an odd number of levels
// the top treelet's own node is a virtual one above the root, whose first
// child is the root. A level's treelets are numbered left to right (i), its
// place in the heap is given by lvlbit = 2^(level of the treelet's children).
#pragma once

#include <cmath>
#include <cstring>

#include "aur_internal.h"
#include "aur_math.cuh"
#include "aur_traverse.cuh"

namespace aur {

constexpr uint32_t kWideStride = 6;   // uint4 per record

__host__ __device__ __forceinline__ uint32_t float_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t b;
    memcpy(&b, &f, sizeof(b));
    return b;
#endif
}

struct WideView {
    const float4* recs;       // NMH records: the triangles (and the slabs, for the checks)
    const uint4* wide;        // treelet records
    const uint32_t* perm;
    const float* verts;       // NMH order, 9 floats per triangle
    uint32_t nodes;           // NMH nodes
    uint32_t levels;          // NMH levels
    // No triangle's det (intersect_tri) exceeds this times the largest
    // component of the direction: the six products of two edge components and
    // one of the direction, edges no longer than the soup's extent.
    float reach = INFINITY;

    // the tree that a lane's ray runs in (WideQueue): the same for all
    __device__ __forceinline__ const float4* recs_of(uint32_t) const { return recs; }
    __device__ __forceinline__ const uint32_t* perm_of(uint32_t) const { return perm; }
};

// WideView::reach of an NMH (infinite where the extent is unknown, and where
// its square overflows).
inline float wide_reach(const aur_nmh* nmh) {
    return nmh->extent > 0.0f ? 6.01f * nmh->extent * nmh->extent : INFINITY;
}

inline WideView wide_view(const aur_nmh* nmh) {
    return WideView{nmh->node_recs, nmh->wide, nmh->perm, nmh->verts, nmh->nodes, nmh->levels, wide_reach(nmh)};
}

// Largest origin spread of a warp packet: 1/64 of the soup's extent. Rays
// that start further apart visit mostly different nodes near their origins,
// and one ray per lane is faster for them.
inline float packet_span(const aur_nmh* nmh) { return nmh->extent * (1.0f / 64.0f); }

// Largest spread of a packet's directions (per component): about two and a
// half times the angle that one of the soup's count^(1/3) cells along a side
// takes at the distance of its extent. Wider packets meet many more treelets
// than each of their rays does. 1M triangles (0.025): a 2.8k-pixel-wide pinhole's
// rows (spread 0.011) 4.3 ms as packets against 7.0 ms one ray per lane, a
// 1k-wide one's (0.032) 1.32 against 1.36, a 512-wide one's (0.06) 0.91 against
// 0.62, a 200-wide one's (0.16) 1.1 against 0.21. 30k triangles (0.08): 0.60
// against 0.83 (0.032) and 0.40 against 0.45 (0.06).
inline float dir_span(const aur_nmh* nmh) { return 2.5f / cbrtf((float)(nmh->count ? nmh->count : 1u)); }

// Index of the first treelet with this lvlbit among all records.
__host__ __device__ __forceinline__ uint32_t wide_base(uint32_t lvlbit, uint32_t levels) {
    return ((lvlbit >> 1) + ((levels & 1u) ? 1u : 0xFFFFFFFFu)) / 3u;
}
__host__ __device__ __forceinline__ uint32_t wide_top(uint32_t levels) { return (levels & 1u) ? 1u : 2u; }
__host__ __device__ __forceinline__ uint32_t wide_leafbit(uint32_t levels) { return 1u << (levels - 1u); }
// Records of an NMH of `levels` levels (all treelets of all levels).
__host__ __device__ __forceinline__ uint64_t wide_count(uint32_t levels) {
    if (levels == 0) return 0;
    return (((uint64_t)wide_leafbit(levels) << 1) + (levels & 1u ? 1 : -1)) / 3;
}

// ------------------------------------------------------------ build
// Writes the record of treelet t of an NMH of n nodes: verts are the
// NMH-ordered vertices, box[6k..] the subtree box (lo.xyz, hi.xyz) of node k.
// Each box is padded on every axis by 1e-5 of that axis' coordinates plus
// 1e-6 of the largest axis' (the triangle test's rounding scales with the
// distance, not with one axis), the grid spans the padded boxes in 253 cells,
// and the bytes are rounded outward with 1/16 cell to spare for the rounding
// of the box test's plane distances. Both are far above that rounding.
__host__ __device__ __forceinline__ void wide_record(const float* __restrict__ verts, const float* __restrict__ box,
                                                     uint32_t n, uint32_t levels, uint32_t t, uint4* __restrict__ rec) {
    uint32_t lvlbit = wide_top(levels);
    while (lvlbit != wide_leafbit(levels) && t >= wide_base(lvlbit << 2, levels)) lvlbit <<= 2;
    const uint32_t i = t - wide_base(lvlbit, levels);
    const bool leaf = lvlbit == wide_leafbit(levels), virt = lvlbit == 1u;
    const uint32_t cb = lvlbit - 1u + 2u * i;
    float lo[10][3], hi[10][3];
    uint32_t valid = 0;
#pragma unroll
    for (int b = 0; b < 10; ++b) {
        bool have;
        if (b < 6) {
            const uint32_t node = b < 2 ? (cb - 1u) >> 1 : cb + (uint32_t)((b - 2) >> 1);
            have = !(virt && (b < 2 || b >= 4)) && node < n;
            if (have) {
                const float* v = verts + ((size_t)2 * node + (b & 1)) * 9;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[b][a] = fminf(fminf(v[3 * a], v[3 * a + 1]), v[3 * a + 2]);
                    hi[b][a] = fmaxf(fmaxf(v[3 * a], v[3 * a + 1]), v[3 * a + 2]);
                }
                valid |= 1u << b;
            }
        } else {
            const uint32_t g = 2u * cb + 1u + (uint32_t)(b - 6);
            have = !leaf && !(virt && b >= 8);
            if (have) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[b][a] = box[6 * (size_t)g + a];
                    hi[b][a] = box[6 * (size_t)g + 3 + a];
                }
                valid |= 1u << (b + 2);
            }
        }
        if (have) {
            float m = 0.0f;
#pragma unroll
            for (int a = 0; a < 3; ++a) m = fmaxf(m, fabsf(lo[b][a]) + fabsf(hi[b][a]));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float pad = 1e-5f * (fabsf(lo[b][a]) + fabsf(hi[b][a])) + 1e-6f * m + 1e-30f;
                lo[b][a] -= pad;
                hi[b][a] += pad;
            }
        } else {
#pragma unroll
            for (int a = 0; a < 3; ++a) { lo[b][a] = INFINITY; hi[b][a] = -INFINITY; }
        }
    }
    float o[3], s[3];
    uint32_t plane[6][3];      // [axis * 2 + side]: bytes of triangles 0-3, of triangles 4-5, of the subtrees
    bool finite = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float l = INFINITY, h = -INFINITY;
#pragma unroll
        for (int b = 0; b < 10; ++b) { l = fminf(l, lo[b][a]); h = fmaxf(h, hi[b][a]); }
        s[a] = (h - l) * (1.0f / 253.0f);
        o[a] = l - 1024.5f * s[a];
        finite = finite && fabsf(s[a]) <= 3.0e35f && fabsf(o[a]) <= 3.0e38f;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            uint32_t w[3] = {0u, 0u, 0u};
#pragma unroll
            for (int b = 0; b < 10; ++b) {
                const float x = ((side ? hi[b][a] : lo[b][a]) - o[a]) / s[a] - 1024.0f;
                const float q = side ? ceilf(x + 0.0625f) : floorf(x - 0.0625f);
                const uint32_t byte = (uint32_t)fminf(fmaxf(q, 0.0f), 255.0f);
                if (b < 4) w[0] |= byte << (8 * b);
                else if (b < 6) w[1] |= byte << (8 * (b - 4));
                else w[2] |= byte << (8 * (b - 6));
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) plane[2 * a + side][q] = w[q];
        }
    }
    uint32_t ow[3], sw[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {   // beyond the float range: NaN planes, which prune nothing
        ow[a] = finite ? float_bits(o[a]) : 0x7FC00000u;
        sw[a] = finite ? float_bits(s[a]) : 0x7FC00000u;
    }
    rec[0] = make_uint4(ow[0], ow[1], ow[2], sw[0]);
    rec[1] = make_uint4(sw[1], sw[2], plane[0][0], plane[1][0]);
    rec[2] = make_uint4(plane[2][0], plane[3][0], plane[4][0], plane[5][0]);
    rec[3] = make_uint4(plane[0][1] | (plane[1][1] << 16), plane[2][1] | (plane[3][1] << 16),
                        plane[4][1] | (plane[5][1] << 16), valid);
    if (!leaf) {
        rec[4] = make_uint4(plane[0][2], plane[1][2], plane[2][2], plane[3][2]);
        rec[5] = make_uint4(plane[4][2], plane[5][2], 0u, 0u);
    }
}

// ------------------------------------------------------------ box test
// Distances to a plane: t = (1024 + q) * A + B with A = s / d and
// B = (o - pos) / d. Two bytes become the halves 1024 + q by one byte permute
// (q is the low byte of a half of value 1024) and the floats by a conversion
// each, and one packed multiply-add gives both distances: the integer pipe,
// where permutes and min / max run, is the busiest of the traversal. (Closest
// hit, 8M random rays: 8.9 ms; a permute per byte into the mantissa of 1.0 and
// single multiply-adds 9.3 ms; either change alone 9.1 to 9.2 ms.) Near the
// treelet the distances' rounding is below 2^-12 of a cell, and the boxes are
// widened by 1/16 of a cell (wide_record). From further away it grows with the
// distance, as t does, and stays below 2^-21 of t: there it is the 2e-4 between
// kBoxNear and kBoxFar that keeps the test conservative.
struct WidePlanes {
    f3 A, B;
};

__device__ __forceinline__ float max3f(float a, float b, float c) {
#ifdef __CUDACC__
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
#ifdef __CUDACC__
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fminf(fminf(a, b), c);
#endif
}

// Distances to the planes of bytes kB0 and kB1 of a word.
template <int kB0, int kB1>
__device__ __forceinline__ void plane_pair(uint32_t word, float A, float B, float& t0, float& t1) {
#ifdef __CUDACC__
    const uint32_t halves = __byte_perm(word, 0x64646464u, 0x4040u | (kB1 << 8) | kB0);
    asm("{\n\t"
        ".reg .f16 h0, h1;\n\t"
        ".reg .f32 f0, f1;\n\t"
        ".reg .b64 v, a, b;\n\t"
        "mov.b32 {h0, h1}, %2;\n\t"
        "cvt.f32.f16 f0, h0;\n\t"
        "cvt.f32.f16 f1, h1;\n\t"
        "mov.b64 v, {f0, f1};\n\t"
        "mov.b64 a, {%3, %3};\n\t"
        "mov.b64 b, {%4, %4};\n\t"
        "fma.rn.f32x2 v, v, a, b;\n\t"
        "mov.b64 {%0, %1}, v;\n\t"
        "}"
        : "=f"(t0), "=f"(t1)
        : "r"(halves), "f"(A), "f"(B));
#else
    t0 = __fmaf_rn(1024.0f + (float)((word >> (8 * kB0)) & 255u), A, B);
    t1 = __fmaf_rn(1024.0f + (float)((word >> (8 * kB1)) & 255u), A, B);
#endif
}

// Two box tests: near planes in bytes kN0 and kN1, far planes in kF0 and kF1
// of the plane words (near and far by the sign of the ray's reciprocal). A NaN
// distance (a grid or ray beyond the float range) drops its axis from the
// test: it never prunes. The verdicts are the signs of tf - tn, shifted into
// acc from below, the first box first (0: hit).
template <int kN0, int kF0, int kN1, int kF1>
__device__ __forceinline__ uint32_t wide_boxes(uint32_t acc, uint32_t xn, uint32_t xf, uint32_t yn, uint32_t yf,
                                               uint32_t zn, uint32_t zf, const WidePlanes& p, float tlimit) {
    float n0[3], n1[3], f0[3], f1[3];
    plane_pair<kN0, kN1>(xn, p.A.x, p.B.x, n0[0], n1[0]);
    plane_pair<kN0, kN1>(yn, p.A.y, p.B.y, n0[1], n1[1]);
    plane_pair<kN0, kN1>(zn, p.A.z, p.B.z, n0[2], n1[2]);
    plane_pair<kF0, kF1>(xf, p.A.x, p.B.x, f0[0], f1[0]);
    plane_pair<kF0, kF1>(yf, p.A.y, p.B.y, f0[1], f1[1]);
    plane_pair<kF0, kF1>(zf, p.A.z, p.B.z, f0[2], f1[2]);
    const float tn0 = fmaxf(max3f(n0[0], n0[1], n0[2]), 0.0f), tf0 = fminf(min3f(f0[0], f0[1], f0[2]), tlimit);
    const float tn1 = fmaxf(max3f(n1[0], n1[1], n1[2]), 0.0f), tf1 = fminf(min3f(f1[0], f1[1], f1[2]), tlimit);
    acc = __funnelshift_l(__float_as_uint(__fmaf_rn(tn0, -kBoxNear / kBoxFar, tf0)), acc, 1);
    return __funnelshift_l(__float_as_uint(__fmaf_rn(tn1, -kBoxNear / kBoxFar, tf1)), acc, 1);
}

// ------------------------------------------------------------ ray and state
struct WideRay {
    f3 pos, dir, inv;     // inv: reciprocal direction, clamped (wide_ray)
    uint32_t order;       // bit 31 - b: the ray visits the second child first on level b (0 < b < 31)
};

__device__ __forceinline__ float wide_recip(float d, float least) {
    return 1.0f / copysignf(fmaxf(fabsf(d), least), d);
}

__device__ __forceinline__ uint32_t wide_order(bool nx, bool ny, bool nz) {
    return (nx ? 0x12492492u : 0u) | (ny ? 0x49249249u : 0u) | (nz ? 0x24924924u : 0u);
}

// Components below 1e-20, and below 1e-12 of the largest, are taken as that
// for the box tests. Over the distance to a hit the ray is moved sideways by at
// most 1e-12 of that distance, far below the boxes' padding, and the
// reciprocals of axis-parallel rays stay finite.
__device__ __forceinline__ void wide_ray(WideRay& r, const f3& pos, const f3& dir) {
    r.pos = pos;
    r.dir = dir;
    const float least = fminf(1e-20f, 1e-12f * fmaxf(largest(dir), kShortDir));
    r.inv = mk3(wide_recip(dir.x, least), wide_recip(dir.y, least), wide_recip(dir.z, least));
    r.order = wide_order(dir.x < 0.0f, dir.y < 0.0f, dir.z < 0.0f);
}

// What a ray has found: best is the NMH position of the triangle (kNoPrim:
// none; kWalkRay: the ray is too short for box tests, the checks walk it), t2
// the smallest t of any other triangle it meets (tmax at the start).
constexpr uint32_t kWalkRay = 0xFFFFFFFEu;

struct WideHit {
    float t, t2;
    uint32_t best;
};

// Pending subtrees: a nibble per treelet level, the current level's lowest
// (bits in visit order), pushed by a shift of 4 on every descent. kOrdered
// walks also keep one bit per level in `pair`: the second child's pair is
// still to be tested, after the first child's subtrees.
struct WideState {
    uint32_t i, lvlbit;
    unsigned long long trail;
    uint32_t pair;
    bool at_pair;
};

enum WideMode { kWideClosest, kWideAny, kWideFirst };

__device__ __forceinline__ void wide_init(WideState& s, uint32_t levels) {
    s.i = 0;
    s.lvlbit = wide_top(levels);
    s.trail = 0;
    s.pair = 0;
    s.at_pair = false;
}

// Starts a ray. Returns false when there is nothing to traverse: it can hit
// nothing (no t in (Epsilon, tmax), no direction, or a component that is NaN or
// infinite: every t test of such a ray fails), or its direction is short. The
// exact walk takes short ones (h.best is kWalkRay) where some triangle's det
// can reach Epsilon.
__device__ __forceinline__ bool wide_begin(WideRay& r, WideState& s, WideHit& h, const WideView& w, const f3& pos,
                                           const f3& dir, float tmax) {
    wide_ray(r, pos, dir);
    wide_init(s, w.levels);
    h.t = h.t2 = tmax;
    h.best = kNoPrim;
    const float len = largest(dir);
    if (!(w.nodes != 0u && tmax > kEpsilon && largest(pos) < INFINITY && len < INFINITY)) return false;
    if (len >= kShortDir) return true;
    if (len * w.reach >= kEpsilon) h.best = kWalkRay;
    return false;
}

// Tests the ten boxes of the current treelet against (0, lim]: its pending
// subtrees go on the trail, the triangles to test are returned (bits in slot
// order; kWideFirst: in the order intersectAny() tests them).
template <WideMode kMode>
__device__ __forceinline__ uint32_t wide_visit(const WideView& w, const WideRay& r, WideState& s, float lim) {
    if (kMode == kWideFirst && s.at_pair) return 0x30u;
    const bool leaf = s.lvlbit == wide_leafbit(w.levels);
    const uint32_t ord = (r.order >> (__clz(s.lvlbit) - 1)) & 3u;
    uint32_t tris, kids = 0;
    const uint4* rec = w.wide + (size_t)(wide_base(s.lvlbit, w.levels) + s.i) * kWideStride;
    const Sector a = ld_sector(reinterpret_cast<const float4*>(rec));
    const Sector b = ld_sector(reinterpret_cast<const float4*>(rec + 2));
    Sector c;
    if (!leaf) c = ld_sector(reinterpret_cast<const float4*>(rec + 4));
    WidePlanes p;
    p.A = mk3(a.a.w * r.inv.x, a.b.x * r.inv.y, a.b.y * r.inv.z);
    p.B = mk3((a.a.x - r.pos.x) * r.inv.x, (a.a.y - r.pos.y) * r.inv.y, (a.a.z - r.pos.z) * r.inv.z);
    // byte selectors of the near planes: the hi words (bytes 4-7 of a pair) where the ray runs down the axis
    const uint32_t sx = r.inv.x < 0.0f ? 0x4444u : 0u, sy = r.inv.y < 0.0f ? 0x4444u : 0u,
                   sz = r.inv.z < 0.0f ? 0x4444u : 0u;
    uint32_t miss = 0;
    {
        // triangles 4, 5: bytes (lo, lo, hi, hi) of one word per axis, turned by two bytes
        const uint32_t x = __byte_perm(__float_as_uint(b.b.x), 0, 0x3210u ^ (sx >> 1)),
                       y = __byte_perm(__float_as_uint(b.b.y), 0, 0x3210u ^ (sy >> 1)),
                       z = __byte_perm(__float_as_uint(b.b.z), 0, 0x3210u ^ (sz >> 1));
        miss = wide_boxes<1, 3, 0, 2>(miss, x, x, y, y, z, z, p, lim);
    }
    {
        const uint32_t x0 = __float_as_uint(a.b.z), x1 = __float_as_uint(a.b.w), y0 = __float_as_uint(b.a.x),
                       y1 = __float_as_uint(b.a.y), z0 = __float_as_uint(b.a.z), z1 = __float_as_uint(b.a.w);
        const uint32_t xn = sx ? x1 : x0, xf = sx ? x0 : x1, yn = sy ? y1 : y0, yf = sy ? y0 : y1,
                       zn = sz ? z1 : z0, zf = sz ? z0 : z1;
        miss = wide_boxes<3, 3, 2, 2>(miss, xn, xf, yn, yf, zn, zf, p, lim);
        miss = wide_boxes<1, 1, 0, 0>(miss, xn, xf, yn, yf, zn, zf, p, lim);
    }
    const uint32_t valid = __float_as_uint(b.b.w);
    tris = ~miss & valid & 63u;
    if (!leaf) {
        // bytes into visit order: rank k is grandchild k ^ ord
        const uint32_t sel = ord * 0x1111u, nx = sel ^ sx, ny = sel ^ sy, nz = sel ^ sz;
        const uint32_t x0 = __float_as_uint(c.a.x), x1 = __float_as_uint(c.a.y), y0 = __float_as_uint(c.a.z),
                       y1 = __float_as_uint(c.a.w), z0 = __float_as_uint(c.b.x), z1 = __float_as_uint(c.b.y);
        const uint32_t xn = __byte_perm(x0, x1, 0x3210u ^ nx), xf = __byte_perm(x0, x1, 0x7654u ^ nx),
                       yn = __byte_perm(y0, y1, 0x3210u ^ ny), yf = __byte_perm(y0, y1, 0x7654u ^ ny),
                       zn = __byte_perm(z0, z1, 0x3210u ^ nz), zf = __byte_perm(z0, z1, 0x7654u ^ nz);
        miss = wide_boxes<3, 3, 2, 2>(0u, xn, xf, yn, yf, zn, zf, p, lim);
        miss = wide_boxes<1, 1, 0, 0>(miss, xn, xf, yn, yf, zn, zf, p, lim);
        kids = ~miss & (valid >> 8);   // only the virtual top lacks any, and its order bit keeps its two in ranks 0, 1
    }
    s.trail = (s.trail << 4) | kids;
    if (kMode == kWideFirst) {
        // pairs into visit order; the far child's comes after the near child's subtrees
        if (ord & 2u) tris = (tris & 3u) | ((tris & 0x0Cu) << 2) | ((tris & 0x30u) >> 2);
        const bool later = (tris & 0x30u) != 0u && (kids & 3u) != 0u;
        s.pair = (s.pair << 1) | (later ? 1u : 0u);
        if (later) tris &= 0x0Fu;
    }
    return tris;
}

// NMH position of the triangle of bit `slot` of wide_visit's result.
template <WideMode kMode>
__device__ __forceinline__ uint32_t wide_tri_index(const WideRay& r, const WideState& s, uint32_t slot) {
    if (kMode == kWideFirst && slot >= 2u && ((r.order >> (__clz(s.lvlbit) - 1)) & 2u)) slot ^= 6u;
    const uint32_t cb = s.lvlbit - 1u + 2u * s.i;   // the first child
    return slot < 2u ? cb - 1u + slot : 2u * cb + slot - 2u;
}

// Moller-Trumbore (intersect_tri) on the triangle at NMH position idx.
__device__ __forceinline__ bool wide_tri(const float4* __restrict__ recs, uint32_t idx, const f3& pos, const f3& dir,
                                         float& t) {
    const bool second = idx & 1u;
    const float4* rec = recs + (size_t)(idx >> 1) * kRecStride + (second ? 2 : 0);
    const Sector a = ld_sector(rec), b = ld_sector(rec + 2);
    const f3 v1 = second ? mk3(a.a.w, a.b.x, a.b.y) : mk3(a.a.z, a.a.w, a.b.x);
    const f3 e1 = second ? mk3(a.b.z, a.b.w, b.a.x) : mk3(a.b.y, a.b.z, a.b.w);
    const f3 e2 = second ? mk3(b.a.y, b.a.z, b.a.w) : mk3(b.a.x, b.a.y, b.a.z);
    float u, v;
    return intersect_tri(pos, dir, v1, e1, e2, u, v, t) && t > kEpsilon;
}

// On to the next pending treelet (or, kWideFirst, pair): the lowest level
// with one. Returns false when none is left.
template <WideMode kMode>
__device__ __forceinline__ bool wide_next(const WideRay& r, WideState& s) {
    if (kMode == kWideFirst) {
        const uint32_t zt = s.trail ? (uint32_t)(__ffsll((long long)s.trail) - 1) >> 2 : 32u;
        const uint32_t zp = s.pair ? (uint32_t)__ffs(s.pair) - 1u : 32u;
        const uint32_t z = min(zt, zp);
        if (z == 32u) return false;
        s.trail >>= 4 * z;
        s.pair >>= z;
        s.i >>= 2 * z;
        s.lvlbit >>= 2 * z;
        s.at_pair = (s.pair & 1u) && !(s.trail & 3ull);
        if (s.at_pair) {
            s.pair &= ~1u;
            return true;
        }
    } else {
        if (s.trail == 0) return false;
        const uint32_t z = (uint32_t)(__ffsll((long long)s.trail) - 1) >> 2;
        s.trail >>= 4 * z;
        s.i >>= 2 * z;
        s.lvlbit >>= 2 * z;
    }
    const uint32_t m = (uint32_t)s.trail & 15u;
    const uint32_t q = ((uint32_t)__ffs(m) - 1u) ^ ((r.order >> (__clz(s.lvlbit) - 1)) & 3u);
    s.trail &= s.trail - 1ull;
    s.i = 4u * s.i + q;
    s.lvlbit <<= 2;
    return true;
}

// One treelet: box tests, triangle tests, and on to the next pending
// treelet. Returns false when the traversal has ended (any hit: a triangle
// was found). kWideFirst visits nodes in the order of intersectAny().
template <WideMode kMode>
__device__ __forceinline__ bool wide_step(const WideView& w, const WideRay& r, WideState& s, WideHit& h) {
    uint32_t tris = wide_visit<kMode>(w, r, s, h.t);
    while (tris) {
        const uint32_t idx = wide_tri_index<kMode>(r, s, __ffs(tris) - 1);
        tris &= tris - 1u;
        float t;
        if (wide_tri(w.recs, idx, r.pos, r.dir, t)) {
            if (kMode != kWideClosest) {
                if (t < h.t) {
                    h.best = idx;
                    return false;
                }
            } else if (t < h.t) {
                h.t2 = h.t;
                h.t = t;
                h.best = idx;
            } else {
                if (t == h.t && h.best != kNoPrim && w.perm[idx] < w.perm[h.best]) h.best = idx;
                h.t2 = fminf(h.t2, t);
            }
        }
    }
    return wide_next<kMode>(r, s);
}

// ------------------------------------------------------------ triangle queue
// Few lanes of a warp meet a triangle's box in the same step (a ray meets
// about 0.4 a treelet), so the warp collects (ray, triangle) pairs and tests
// 32 of them at once, one per lane, whichever lane's ray they belong to. A
// ray's result lives in shared memory meanwhile: the smallest key
//   closest hit: t, prim id   (ties in t go to the lower prim id)
//   first occluder: position in the ray's own test order
// found so far. Rays go on to further treelets while their pairs wait, so a
// box is now and then tested against a t that is about to shrink; what is
// found is the same. (AUR_HOST_WARP: host builds that bring the warp
// intrinsics along.)
#if defined(__CUDACC__) || defined(AUR_HOST_WARP)
struct WideQueue {
    float4 pd[32];                // pos.xyz, dir.x of each lane's ray
    float2 d[32];                 // dir.yz
    unsigned long long key[32];
    uint32_t best[32];            // NMH position of key's triangle
    uint32_t t2[32];              // closest hit: WideHit::t2, as bits (t is positive); any hit: tmax
    uint32_t idx[64];             // waiting pairs: NMH position,
    uint32_t seq[64];             //   position in the ray's test order (first occluder),
    uint8_t lane[64];             //   and the ray's lane
};

constexpr unsigned long long kNoKey = ~0ull;

// best: WideHit::best as wide_begin left it.
template <WideMode kMode>
__device__ __forceinline__ void queue_ray(WideQueue& q, uint32_t lane, const f3& pos, const f3& dir, float tmax,
                                          uint32_t best) {
    q.pd[lane] = make_float4(pos.x, pos.y, pos.z, dir.x);
    q.d[lane] = make_float2(dir.y, dir.z);
    // a triangle at exactly tmax is not a hit: no (tmax, prim id) is below (tmax, 0)
    q.key[lane] = kMode == kWideClosest ? (unsigned long long)__float_as_uint(tmax) << 32 : kNoKey;
    q.best[lane] = best;
    q.t2[lane] = __float_as_uint(tmax);
}

// Tests the last m (<= 32) waiting pairs; `w` tells each lane's tree (WideView,
// or one tree per lane). Call with all lanes.
template <WideMode kMode, typename Trees>
__device__ __forceinline__ void queue_test(WideQueue& q, uint32_t lane, uint32_t count, uint32_t m, const Trees& w) {
    __syncwarp();
    uint32_t own = 0, idx = 0;
    unsigned long long mine = kNoKey;
    if (lane < m) {
        const uint32_t e = count - m + lane;
        own = q.lane[e];
        idx = q.idx[e];
        const float4 a = q.pd[own];
        const float2 b = q.d[own];
        float t;
        if (wide_tri(w.recs_of(own), idx, mk3(a.x, a.y, a.z), mk3(a.w, b.x, b.y), t)) {
            if (kMode == kWideClosest) {
                if (t <= __uint_as_float(q.t2[own])) {
                    const unsigned long long k = ((unsigned long long)__float_as_uint(t) << 32) | w.perm_of(own)[idx];
                    const unsigned long long old = atomicMin(&q.key[own], k);
                    if (k < old) mine = k;
                    atomicMin(&q.t2[own], (uint32_t)((k < old ? old : k) >> 32));
                }
            } else if (t < __uint_as_float(q.t2[own])) {
                mine = kMode == kWideFirst ? q.seq[e] : 0ull;
                atomicMin(&q.key[own], mine);
            }
        }
    }
    __syncwarp();
    if (mine != kNoKey && q.key[own] == mine) q.best[own] = idx;
    __syncwarp();
}

// Adds the triangles of each lane's `tris` (wide_visit) to the queue, testing
// 32 pairs whenever that many wait. count and seq as left by the last call.
template <WideMode kMode, typename Trees>
__device__ __forceinline__ void queue_add(WideQueue& q, uint32_t lane, uint32_t& count, uint32_t& seq, uint32_t tris,
                                          const WideRay& r, const WideState& s, const Trees& w) {
    for (;;) {
        const uint32_t have = __ballot_sync(0xffffffffu, tris != 0u);
        if (have == 0u) break;
        if (tris) {
            uint32_t lt;
#ifdef __CUDACC__
            asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
#else
            lt = (1u << lane) - 1u;
#endif
            const uint32_t e = count + __popc(have & lt);
            q.idx[e] = wide_tri_index<kMode>(r, s, __ffs(tris) - 1);
            q.lane[e] = (uint8_t)lane;
            if (kMode == kWideFirst) q.seq[e] = seq++;
            tris &= tris - 1u;
        }
        count += __popc(have);
        if (count >= 32u) {
            queue_test<kMode>(q, lane, count, 32u, w);
            count -= 32u;
        }
    }
}

// The warp's 32 rays (`valid`: the lane has one), one per lane, to their end.
// Call with all 32 lanes.
template <WideMode kMode>
__device__ __forceinline__ void wide_warp(const WideView& w, WideQueue& q, bool valid, const f3& pos, const f3& dir,
                                          float tmax, WideHit& h) {
    const uint32_t lane = threadIdx.x & 31;
    WideRay r;
    WideState s;
    bool running = wide_begin(r, s, h, w, pos, dir, tmax) && valid;
    __syncwarp();
    queue_ray<kMode>(q, lane, pos, dir, tmax, h.best);
    __syncwarp();
    float lim = tmax;
    uint32_t count = 0, seq = 0;
    while (__any_sync(0xffffffffu, running)) {
        uint32_t tris = 0;
        if (running) tris = wide_visit<kMode>(w, r, s, lim);
        queue_add<kMode>(q, lane, count, seq, tris, r, s, w);
        if (running) {
            if (kMode == kWideClosest) lim = __uint_as_float((uint32_t)(q.key[lane] >> 32));
            running = (kMode == kWideClosest || q.key[lane] == kNoKey) && wide_next<kMode>(r, s);
        }
    }
    queue_test<kMode>(q, lane, count, count, w);
    if (kMode == kWideClosest) h.t = __uint_as_float((uint32_t)(q.key[lane] >> 32));
    h.t2 = __uint_as_float(q.t2[lane]);
    h.best = q.best[lane];
}
#endif  // __CUDACC__ || AUR_HOST_WARP

// ------------------------------------------------------------ a few triangles
// An NMH of at most kTinyTris triangles has no use for a tree: every lane
// tests every triangle, staged in shared memory and read by the whole warp at
// one address, so no lane waits for another's path and no load waits for a
// node. (1M rays, 100 triangles: 0.20 ms so, 0.20 ms over the treelets; 34:
// 0.10 ms against 0.19 ms.)
//
// A filter goes first, two triangles at a time in packed multiply-adds. With
// m = pos x dir, the three signs Moller-Trumbore decides by are
//   det     = dir . (e2 x e1)
//   u * det = e2 . m + dir . (v1 x e2)
//   v * det = -e1 . m - dir . (v1 x e1)
// and the constants are staged. Their rounding, and that of intersect_tri's
// own terms, is below 1.3e-6 (|pos| + R) |dir| times the longer edge (R: the
// vertices' largest distance from the origin; at most a dozen roundings of
// 2^-24 each on terms no larger); a triangle is dropped when a sign is wrong
// by more than three times that, so every triangle intersect_tri accepts is
// kept. The few kept ones are then tested exactly. (256x256 box frame, 16
// samples: 0.96 ms without the filter, 0.86 with it; 1M rays, 34 triangles:
// 0.10 and 0.08 ms.)
constexpr uint32_t kTinyTris = 64;

struct TinyStage {
    float4 tri[3 * kTinyTris];          // (v1, prim id), e1, e2
    float2 pre[kTinyTris / 2][16];      // of two triangles: e2 x e1, e2, v1 x e2, -e1, -(v1 x e1), longer edge
    uint32_t radius;                    // R, as bits
};

// Stages the `count` (even) triangles. The whole block calls it; ends with a
// block barrier.
__device__ __forceinline__ void stage_tiny(TinyStage& s, const float* __restrict__ verts,
                                           const uint32_t* __restrict__ perm, uint32_t count) {
    if (threadIdx.x == 0) s.radius = 0u;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < count; j += blockDim.x) {
        const float* q = verts + (size_t)j * 9;
        const f3 v1 = mk3(q[0], q[3], q[6]), v2 = mk3(q[1], q[4], q[7]), v3 = mk3(q[2], q[5], q[8]);
        const f3 e1 = v2 - v1, e2 = v3 - v1;
        s.tri[3 * j] = make_float4(v1.x, v1.y, v1.z, __uint_as_float(perm[j]));
        s.tri[3 * j + 1] = make_float4(e1.x, e1.y, e1.z, 0.0f);
        s.tri[3 * j + 2] = make_float4(e2.x, e2.y, e2.z, 0.0f);
        const float r = sqrtf(fmaxf(fmaxf(dot(v1, v1), dot(v2, v2)), dot(v3, v3)));
        float c[16];
        const f3 n = cross(e2, e1), c2 = cross(v1, e2), c1 = -cross(v1, e1);
        c[0] = n.x; c[1] = n.y; c[2] = n.z;
        c[3] = e2.x; c[4] = e2.y; c[5] = e2.z;
        c[6] = c2.x; c[7] = c2.y; c[8] = c2.z;
        c[9] = -e1.x; c[10] = -e1.y; c[11] = -e1.z;
        c[12] = c1.x; c[13] = c1.y; c[14] = c1.z;
        c[15] = sqrtf(fmaxf(dot(e1, e1), dot(e2, e2)));
        const bool usable = r < 1.0e12f;       // far from overflow; otherwise the triangle is always kept
#pragma unroll
        for (int k = 0; k < 16; ++k)
            reinterpret_cast<float*>(&s.pre[j >> 1][k])[j & 1u] = usable ? c[k] : (k == 15 ? 1.0f : 0.0f);
        if (usable) atomicMax(&s.radius, __float_as_uint(r));
    }
    __syncthreads();
}

#ifdef __CUDACC__
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
#else
static inline unsigned long long pack2(float a, float b) {
    return (unsigned long long)float_bits(a) | ((unsigned long long)float_bits(b) << 32);
}
static inline float2 unpack2(unsigned long long v) {
    return make_float2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
}
static inline unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    const float2 x = unpack2(a), y = unpack2(b), z = unpack2(c);
    return pack2(__fmaf_rn(x.x, y.x, z.x), __fmaf_rn(x.y, y.y, z.y));
}
#endif

// Bit j: triangle j is kept.
__device__ __forceinline__ uint64_t tiny_filter(const TinyStage& s, uint32_t count, const f3& pos, const f3& dir) {
    const uint64_t all = count >= 64u ? ~0ull : (1ull << count) - 1ull;
    const float dd = dot(dir, dir);
    const float scale = 4.0e-6f * (sqrtf(dot(pos, pos)) + __uint_as_float(s.radius)) * sqrtf(dd);
    // products beyond the float range, or a length that its square's underflow makes too small
    if (!(scale < 1.0e24f && dd > 1.0e-30f)) return all;
    const f3 m = cross(pos, dir);
    const unsigned long long dx = pack2(dir.x, dir.x), dy = pack2(dir.y, dir.y), dz = pack2(dir.z, dir.z);
    const unsigned long long mx = pack2(m.x, m.x), my = pack2(m.y, m.y), mz = pack2(m.z, m.z);
    const unsigned long long sc = pack2(scale, scale), one = pack2(-1.0f, -1.0f), zero = pack2(0.0f, 0.0f);
    uint32_t lo = 0, hi = 0;      // verdicts of the even and the odd triangles, the last pair in bit 0 (0: kept)
#pragma unroll 1
    for (uint32_t p = 0; p < count / 2u; ++p) {
        const ulonglong2* c = reinterpret_cast<const ulonglong2*>(s.pre[p]);
        const ulonglong2 q0 = c[0], q1 = c[1], q2 = c[2], q3 = c[3], q4 = c[4], q5 = c[5], q6 = c[6], q7 = c[7];
        const unsigned long long g = fma2(q7.y, sc, zero);
        const unsigned long long det = fma2(q0.x, dx, fma2(q0.y, dy, fma2(q1.x, dz, fma2(q7.y, sc, g))));
        const unsigned long long du =
            fma2(q1.y, mx, fma2(q2.x, my, fma2(q2.y, mz, fma2(q3.x, dx, fma2(q3.y, dy, fma2(q4.x, dz, g))))));
        const unsigned long long dv =
            fma2(q4.y, mx, fma2(q5.x, my, fma2(q5.y, mz, fma2(q6.x, dx, fma2(q6.y, dy, fma2(q7.x, dz, g))))));
        // det - du - dv with a margin of 3 (the terms carry 2, 1 and 1)
        const unsigned long long w = fma2(dv, one, fma2(du, one, fma2(g, pack2(3.0f, 3.0f), det)));
        const float2 a = unpack2(det), b = unpack2(du), d = unpack2(dv), e = unpack2(w);
        lo = __funnelshift_l(__float_as_uint(fminf(min3f(a.x, b.x, d.x), e.x)), lo, 1);
        hi = __funnelshift_l(__float_as_uint(fminf(min3f(a.y, b.y, d.y), e.y)), hi, 1);
    }
    // pair p's verdicts are bit count / 2 - 1 - p: reversed, then interleaved
    const uint32_t even = __brev(~lo) >> (32u - count / 2u), odd = __brev(~hi) >> (32u - count / 2u);
    uint64_t mask = 0;
    auto spread = [](uint32_t x) {
        uint64_t v = x;
        v = (v | (v << 16)) & 0x0000FFFF0000FFFFull;
        v = (v | (v << 8)) & 0x00FF00FF00FF00FFull;
        v = (v | (v << 4)) & 0x0F0F0F0F0F0F0F0Full;
        v = (v | (v << 2)) & 0x3333333333333333ull;
        return (v | (v << 1)) & 0x5555555555555555ull;
    };
    mask = spread(even) | (spread(odd) << 1);
    return mask & all;
}

__device__ __forceinline__ bool tiny_tri(const TinyStage& s, uint32_t j, const f3& pos, const f3& dir, float& t,
                                         uint32_t& id) {
    const float4 a = s.tri[3 * j], b = s.tri[3 * j + 1], c = s.tri[3 * j + 2];
    float u, v;
    id = __float_as_uint(a.w);
    return intersect_tri(pos, dir, mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), mk3(c.x, c.y, c.z), u, v, t) && t > kEpsilon;
}

__device__ __forceinline__ void tiny_closest(const TinyStage& s, uint32_t count, const f3& pos, const f3& dir,
                                             float tmax, WideHit& h) {
    h.t = h.t2 = tmax;
    h.best = kNoPrim;
    uint32_t best_id = 0;
    for (uint64_t kept = tiny_filter(s, count, pos, dir); kept; kept &= kept - 1ull) {
        const uint32_t j = (uint32_t)__ffsll((long long)kept) - 1u;
        float t;
        uint32_t id;
        if (!tiny_tri(s, j, pos, dir, t, id)) continue;
        if (t < h.t) {
            h.t2 = h.t;
            h.t = t;
            h.best = j;
            best_id = id;
        } else {
            if (t == h.t && h.best != kNoPrim && id < best_id) {
                h.best = j;
                best_id = id;
            }
            h.t2 = fminf(h.t2, t);
        }
    }
}

__device__ __forceinline__ uint32_t tiny_any(const TinyStage& s, uint32_t count, const f3& pos, const f3& dir,
                                             float tmax) {
    for (uint64_t kept = tiny_filter(s, count, pos, dir); kept; kept &= kept - 1ull) {
        const uint32_t j = (uint32_t)__ffsll((long long)kept) - 1u;
        float t;
        uint32_t id;
        if (tiny_tri(s, j, pos, dir, t, id) && t < tmax) return j;
    }
    return kNoPrim;
}
// ------------------------------------------------------------ the checks
// intersect() visits a triangle's node when the ray's range, clipped by the
// slab of every node from the root down to it (ray.cuh:225-237), is not empty
// and starts no later than the best t so far. Each of those slabs contains
// the triangle, and (plane - pos) / dir rounds monotonically, so on each axis
// the slabs' entries are at most, and their exits at least, those of the
// triangle's own bounds: if the range of the three own slabs [E, X] is not
// empty and E is no later than the best t, the node was visited.

// The exact range of node tri / 2's visit: every slab on its path.
static __device__ __noinline__ float2 path_range(const float4* recs, uint32_t tri, float px, float py, float pz, float dx,
                                          float dy, float dz) {
    float lo = kEpsilon, hi = kInfinity;
    for (uint32_t k = tri >> 1;; k = (k - 1u) >> 1) {
        const uint32_t ax = (31u - (uint32_t)__clz(k + 1u)) % 3u;
        const float p = sel3(ax, px, py, pz), d = sel3(ax, dx, dy, dz);
        const float4 q = recs[(size_t)k * kRecStride];
        const float d0 = (q.x - p) / d, d1 = (q.y - p) / d;
        lo = fmaxf(fminf(d0, d1), lo);
        hi = fminf(fmaxf(d0, d1), hi);
        if (k == 0) break;
    }
    return make_float2(lo, hi);
}

// The walk of intersect() itself, for a ray whose triangle fails the check
// (its slab ranges exclude the triangle by rounding), or whose direction is
// short: (t, u, v, NMH position).
template <bool kAny>
static __device__ __forceinline__ float4 exact_walk(const float4* recs, uint32_t nodes, const uint32_t* perm, float px, float py,
                                          float pz, float dx, float dy, float dz, float tmax) {
    float lo[kStackDepth], hi[kStackDepth];
    StackRef stk;
    stk.lo = lo;
    stk.hi = hi;
    stk.stride = 1;
    stk.cap = kStackDepth;
    float t = tmax, u = 0.0f, v = 0.0f;
    uint32_t visits = 0;
    const uint32_t best = traverse<kAny>(recs, nodes, perm, mk3(px, py, pz), mk3(dx, dy, dz), t, u, v, stk, visits);
    return make_float4(t, u, v, __uint_as_float(best));
}

__device__ __forceinline__ void own_range(const float* __restrict__ v, const f3& pos, const f3& dir, float& E, float& X) {
    E = kEpsilon;
    X = kInfinity;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float p = a == 0 ? pos.x : (a == 1 ? pos.y : pos.z), d = a == 0 ? dir.x : (a == 1 ? dir.y : dir.z);
        const float d0 = (fminf(fminf(v[3 * a], v[3 * a + 1]), v[3 * a + 2]) - p) / d;
        const float d1 = (fmaxf(fmaxf(v[3 * a], v[3 * a + 1]), v[3 * a + 2]) - p) / d;
        E = fmaxf(E, fminf(d0, d1));
        X = fminf(X, fmaxf(d0, d1));
    }
}

// True when a visit whose range starts at `lo` was made whatever had been
// found before it: no later than the hit itself, or than every other triangle
// the ray meets (all those up to 1.0001 t have been tested).
__device__ __forceinline__ bool visited_before(float lo, const WideHit& h) {
    return lo <= h.t || (lo <= h.t2 && lo <= h.t * 1.0001f);
}

// The closest hit as intersect() reports it: h.best becomes the NMH position
// (kNoPrim: none) and t, u, v its values.
__device__ __forceinline__ void finish_closest(const WideView& w, const WideRay& r, WideHit& h, float tmax, float& u,
                                               float& v) {
    u = v = 0.0f;
    if (h.best == kNoPrim) return;
    if (h.best != kWalkRay) {
        float q[9];
        const float* src = w.verts + (size_t)h.best * 9;
#pragma unroll
        for (int j = 0; j < 9; ++j) q[j] = __ldg(src + j);
        float t, E, X;
        intersect_tri(r.pos, r.dir, mk3(q[0], q[3], q[6]), mk3(q[1] - q[0], q[4] - q[3], q[7] - q[6]),
                      mk3(q[2] - q[0], q[5] - q[3], q[8] - q[6]), u, v, t);
        own_range(q, r.pos, r.dir, E, X);
        // a zero direction component has 0/0 distances: only the path's own slabs tell
        const bool quick = r.dir.x != 0.0f && r.dir.y != 0.0f && r.dir.z != 0.0f && E <= X && visited_before(E, h);
        if (quick) return;
        const float2 range = path_range(w.recs, h.best, r.pos.x, r.pos.y, r.pos.z, r.dir.x, r.dir.y, r.dir.z);
        if (range.x <= range.y && visited_before(range.x, h)) return;
    }
    const float4 e = exact_walk<false>(w.recs, w.nodes, w.perm, r.pos.x, r.pos.y, r.pos.z, r.dir.x, r.dir.y, r.dir.z, tmax);
    h.t = e.x;
    u = e.y;
    v = e.z;
    h.best = __float_as_uint(e.w);
}

// The occluder of a ray that found triangle h.best: that triangle when its
// node was visited (best t is tmax throughout), else whatever the walk of
// intersectAny() finds.
__device__ __forceinline__ uint32_t finish_any(const WideView& w, const WideRay& r, uint32_t best, float tmax) {
    if (best == kNoPrim) return best;
    if (best != kWalkRay) {
        float q[9];
        const float* src = w.verts + (size_t)best * 9;
#pragma unroll
        for (int j = 0; j < 9; ++j) q[j] = __ldg(src + j);
        float E, X;
        own_range(q, r.pos, r.dir, E, X);
        if (r.dir.x != 0.0f && r.dir.y != 0.0f && r.dir.z != 0.0f && E <= X && E <= tmax) return best;
        const float2 range = path_range(w.recs, best, r.pos.x, r.pos.y, r.pos.z, r.dir.x, r.dir.y, r.dir.z);
        if (range.x <= range.y && range.x <= tmax) return best;
    }
    const float4 e = exact_walk<true>(w.recs, w.nodes, w.perm, r.pos.x, r.pos.y, r.pos.z, r.dir.x, r.dir.y, r.dir.z, tmax);
    return __float_as_uint(e.w);
}

// ------------------------------------------------------------ warp packets
// 32 rays of one direction octant that start close together walk the
// treelets as one: a box is tested once for the warp, by one lane, against
// the interval of all origins and reciprocal directions, so a treelet costs
// the warp one box test per lane instead of ten. Each lane then tests every
// triangle whose box the interval meets. One octant means one visit order, so
// each lane meets its triangles in its own order and its result is its own
// walk's (in any hit, the first accepted triangle). Call with all 32 lanes;
// `valid`: the lane has a ray; oct: the octant (dir_octant of any of them).
#if defined(__CUDACC__) || defined(AUR_HOST_WARP)
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <WideMode kMode>
__device__ __forceinline__ void wide_packet(const WideView& w, bool valid, uint32_t oct, const f3& pos, const f3& dir,
                                            float tmax, WideRay& r, WideHit& h) {
    const uint32_t lane = threadIdx.x & 31;
    WideState s;
    bool live = wide_begin(r, s, h, w, pos, dir, tmax) && valid;
    // The walk (s, and the order it follows) must be the same in every lane,
    // also in those without a ray.
    r.order = wide_order(oct & 1u, oct & 2u, oct & 4u);
    // Per axis, mirrored so that the packet runs up it: origins in
    // [plo, phi], reciprocals in [ilo, ihi].
    float plo[3], phi[3], ilo[3], ihi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float p = a == 0 ? pos.x : (a == 1 ? pos.y : pos.z), iv = fabsf(a == 0 ? r.inv.x : (a == 1 ? r.inv.y : r.inv.z));
        const float m = (oct >> a) & 1u ? -p : p;
        plo[a] = warp_min(live ? m : INFINITY);
        phi[a] = warp_max(live ? m : -INFINITY);
        ilo[a] = warp_min(live ? iv : INFINITY);
        ihi[a] = warp_max(live ? iv : 0.0f);
    }
    // Where this lane's box (0-5 triangles, 6-9 subtrees) has its bytes.
    const uint32_t word = lane < 4u ? 6u : (lane < 6u ? 12u : 16u), step = lane >= 4u && lane < 6u ? 1u : 2u;
    const uint32_t hi_word = step - 1u, sh_lo = 8u * (lane < 4u ? lane : (lane < 6u ? lane - 4u : (lane - 6u) & 3u));
    const uint32_t sh_hi = sh_lo + (step == 1u ? 16u : 0u);
    if (!__any_sync(0xffffffffu, live)) return;
    float lim = __uint_as_float(__reduce_max_sync(0xffffffffu, live ? __float_as_uint(h.t) : 0u));
    for (;;) {
        uint32_t tris;
        if (kMode == kWideFirst && s.at_pair) {
            tris = 0x30u;
        } else {
            const uint4* rec = w.wide + (size_t)(wide_base(s.lvlbit, w.levels) + s.i) * kWideStride;
            const uint32_t* rw = reinterpret_cast<const uint32_t*>(rec);
            const uint4 h0 = __ldg(rec);
            const uint2 h1 = __ldg(reinterpret_cast<const uint2*>(rec + 1));
            const uint32_t valid_bits = __ldg(rw + 15);
            float tn = 0.0f, tf = lim;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float o = __uint_as_float(a == 0 ? h0.x : (a == 1 ? h0.y : h0.z));
                const float sc = __uint_as_float(a == 0 ? h0.w : (a == 1 ? h1.x : h1.y));
                const uint32_t wl = __ldg(rw + word + a * step), wh = __ldg(rw + word + a * step + hi_word);
                const float lo = __fmaf_rn((float)(((wl >> sh_lo) & 255u) + 1024u), sc, o),
                            hi = __fmaf_rn((float)(((wh >> sh_hi) & 255u) + 1024u), sc, o);
                const bool neg = (oct >> a) & 1u;
                const float xn = (neg ? -hi : lo) - phi[a], xf = (neg ? -lo : hi) - plo[a];
                tn = fmaxf(tn, xn * (xn >= 0.0f ? ilo[a] : ihi[a]));
                tf = fminf(tf, xf * (xf >= 0.0f ? ihi[a] : ilo[a]));
            }
            const uint32_t met = __ballot_sync(0xffffffffu, tn * (kBoxNear / kBoxFar) <= tf);
            tris = met & valid_bits & 63u;
            uint32_t kids = (met >> 6) & (valid_bits >> 8) & 15u;
            const uint32_t ord = (r.order >> (__clz(s.lvlbit) - 1)) & 3u;
            if (ord & 1u) kids = ((kids & 5u) << 1) | ((kids >> 1) & 5u);
            if (ord & 2u) kids = ((kids & 3u) << 2) | (kids >> 2);
            s.trail = (s.trail << 4) | kids;
            if (kMode == kWideFirst) {
                if (ord & 2u) tris = (tris & 3u) | ((tris & 0x0Cu) << 2) | ((tris & 0x30u) >> 2);
                const bool later = (tris & 0x30u) != 0u && (kids & 3u) != 0u;
                s.pair = (s.pair << 1) | (later ? 1u : 0u);
                if (later) tris &= 0x0Fu;
            }
        }
        bool found = false;
        while (tris) {
            const uint32_t idx = wide_tri_index<kMode>(r, s, __ffs(tris) - 1);
            tris &= tris - 1u;
            float t;
            if (live && wide_tri(w.recs, idx, r.pos, r.dir, t)) {
                if (kMode != kWideClosest) {
                    if (t < h.t) {
                        h.best = idx;
                        live = false;
                        found = true;
                    }
                } else if (t < h.t) {
                    h.t2 = h.t;
                    h.t = t;
                    h.best = idx;
                    found = true;
                } else {
                    if (t == h.t && h.best != kNoPrim && w.perm[idx] < w.perm[h.best]) h.best = idx;
                    h.t2 = fminf(h.t2, t);
                }
            }
        }
        if (__any_sync(0xffffffffu, found)) {
            lim = __uint_as_float(__reduce_max_sync(0xffffffffu, live ? __float_as_uint(h.t) : 0u));
            if (lim == 0.0f) break;
        }
        if (!wide_next<kMode>(r, s)) break;
    }
}
#endif  // __CUDACC__ || AUR_HOST_WARP

}  // namespace aur
