/* Host build of the traversals that a whole warp runs together (wide_packet,
 * wide_warp and its triangle queue: aurora_gb300/csrc/aur_wide.cuh, the source
 * the CUDA kernels compile), for tests/test_warp_model.py. Each of the 32 lanes
 * is a fiber; a warp intrinsic stops its lane until all 32 have come to the
 * same one. Lanes that meet different intrinsics, or of which some have ended,
 * are reported: on the GPU that warp would hang. Between two intrinsics the
 * lanes run one after the other, in either order, so that a missing
 * __syncwarp shows as a difference. */
#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <vector>

using std::max;
using std::min;
#ifndef __forceinline__
#define __forceinline__ inline
#endif
#undef __noinline__
#define __noinline__
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static inline float __uint_as_float(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
static inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
static inline int __ffsll(long long x) { return __builtin_ffsll(x); }
static inline int __popc(uint32_t x) { return __builtin_popcount(x); }
template <typename T> static inline T __ldg(const T* p) { return *p; }
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s) {
    const uint64_t v = ((uint64_t)y << 32) | x;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= (uint32_t)((v >> (8 * ((s >> (4 * i)) & 7u))) & 255u) << (8 * i);
    return r;
}
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) { return s ? (hi << s) | (lo >> (32 - s)) : hi; }
static inline uint32_t __brev(uint32_t x) { uint32_t r = 0; for (int i = 0; i < 32; ++i) r |= ((x >> i) & 1u) << (31 - i); return r; }

/* ---- 32 fibers */
namespace {
uint32_t g_lane;
struct Warp {
    ucontext_t main, lane[32];
    std::vector<char> stack[32];
    int op[32];               // the intrinsic a lane waits at, 0: it runs, -1: it has ended
    uint32_t in[32], out[32];
    std::function<void(uint32_t)> body;
} *g_warp;

uint32_t collective(int op, uint32_t v) {
    Warp& w = *g_warp;
    const uint32_t l = g_lane;
    w.op[l] = op;
    w.in[l] = v;
    swapcontext(&w.lane[l], &w.main);
    return w.out[l];
}
void lane_main() {
    g_warp->body(g_lane);
    g_warp->op[g_lane] = -1;
}
enum { kBallot = 1, kSync, kMax, kShfl = 64, kXor = 128 };   // kShfl + source lane, kXor + lane mask

/* Runs body(lane) on 32 lanes; false: they did not stay together. */
bool run_warp(Warp& w, bool backwards, std::function<void(uint32_t)> body) {
    g_warp = &w;
    w.body = std::move(body);
    for (int l = 0; l < 32; ++l) {
        w.stack[l].resize(128 << 10);
        getcontext(&w.lane[l]);
        w.lane[l].uc_stack.ss_sp = w.stack[l].data();
        w.lane[l].uc_stack.ss_size = w.stack[l].size();
        w.lane[l].uc_link = &w.main;
        makecontext(&w.lane[l], lane_main, 0);
    }
    for (;;) {
        for (int k = 0; k < 32; ++k) {
            g_lane = backwards ? 31 - k : k;
            w.op[g_lane] = 0;
            swapcontext(&w.main, &w.lane[g_lane]);
        }
        for (int l = 1; l < 32; ++l)
            if (w.op[l] != w.op[0]) return false;
        const int op = w.op[0];
        if (op < 0) return true;
        uint32_t all = 0, top = 0;
        for (int l = 0; l < 32; ++l) {
            all |= (w.in[l] ? 1u : 0u) << l;
            top = max(top, w.in[l]);
        }
        for (int l = 0; l < 32; ++l)
            w.out[l] = op >= kXor ? w.in[l ^ (op - kXor)] : op >= kShfl ? w.in[op - kShfl] : op == kMax ? top : all;
    }
}
}  // namespace

static inline uint32_t __ballot_sync(uint32_t, bool p) { return collective(kBallot, p); }
static inline bool __any_sync(uint32_t, bool p) { return collective(kBallot, p) != 0u; }
static inline bool __all_sync(uint32_t, bool p) { return collective(kBallot, p) == 0xffffffffu; }
static inline void __syncwarp() { collective(kSync, 0); }
static inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { return collective(kMax, v); }
static inline float __shfl_xor_sync(uint32_t, float v, int o) { return __uint_as_float(collective(kXor + o, __float_as_uint(v))); }
template <typename T> static inline T atomicMin(T* p, T v) { const T old = *p; if (v < old) *p = v; return old; }
static inline void atomicMax(uint32_t* p, uint32_t v) { if (v > *p) *p = v; }
struct LaneIdx { struct { operator uint32_t() const { return g_lane; } } x; };
static const LaneIdx threadIdx;
static const struct { uint32_t x; } blockDim = {32};
#define __syncthreads() __syncwarp()

#define AUR_HOST_WARP
#include "../aurora_gb300/csrc/aur_wide.cuh"

using namespace aur;

namespace {
struct Model {   // as tests/wide_model.cpp makes it
    uint32_t n, levels;
    std::vector<float> verts, box;
    std::vector<uint32_t> perm;
    std::vector<float4> recs;
    std::vector<uint4> wide;
};

template <WideMode kMode>
long trace(const WideView& w, const float* rays, uint32_t n, bool packets, bool backwards, float* tuv, uint32_t* prim) {
    Warp warp;
    WideQueue queue;
    for (uint32_t c = 0; c < n; c += 32) {
        const bool together = run_warp(warp, backwards, [&](uint32_t lane) {
            const uint32_t i = c + lane;
            const bool valid = i < n;
            const float* q = rays + 8 * (size_t)i;
            const f3 pos = valid ? mk3(q[0], q[1], q[2]) : mk3(0.0f), dir = valid ? mk3(q[4], q[5], q[6]) : mk3(0.0f);
            const float tmax = valid ? q[3] : 0.0f;
            const float* q0 = rays + 8 * (size_t)c;
            WideRay r;
            WideHit h;
            if (packets) {
                wide_packet<kMode>(w, valid, dir_octant(mk3(q0[4], q0[5], q0[6])), pos, dir, tmax, r, h);
            } else {
                wide_warp<kMode>(w, queue, valid, pos, dir, tmax, h);
                r.pos = pos;
                r.dir = dir;
            }
            if (!valid) return;
            if (kMode == kWideClosest) {
                float u, v;
                finish_closest(w, r, h, tmax, u, v);
                const bool hit = h.best != kNoPrim;
                tuv[3 * (size_t)i] = hit ? h.t : tmax;
                tuv[3 * (size_t)i + 1] = hit ? u : 0.0f;
                tuv[3 * (size_t)i + 2] = hit ? v : 0.0f;
            } else {
                h.best = finish_any(w, r, h.best, tmax);
            }
            prim[i] = h.best == kNoPrim ? 0xFFFFFFFFu : w.perm[h.best];
        });
        if (!together) return (long)c;
    }
    return -1;
}
}  // namespace

/* Traces rays in chunks of 32 (the last one may be partial) over a model of
 * wide_model_create(). packets: wide_packet (the rays of a chunk share their
 * octant), else wide_warp; mode 0: closest hit, 1: any hit (prim: any
 * occluder), 2: the occluder intersectAny() reports. Returns -1, or the first
 * ray of a chunk whose lanes did not stay together. */
extern "C" long warp_model_trace(const void* p, const float* rays, uint32_t n, int packets, int mode, int backwards,
                                 float* tuv, uint32_t* prim) {
    const Model* m = (const Model*)p;
    const WideView w{m->recs.data(), m->wide.data(), m->perm.data(), m->verts.data(), m->n, m->levels};
    if (mode == 0) return trace<kWideClosest>(w, rays, n, packets, backwards, tuv, prim);
    if (mode == 1) return trace<kWideAny>(w, rays, n, packets, backwards, tuv, prim);
    return trace<kWideFirst>(w, rays, n, packets, backwards, tuv, prim);
}
