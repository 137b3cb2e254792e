/* Host build of the treelet traversal (aurora_gb300/csrc/aur_wide.cuh, the
 * same source the CUDA kernels compile) for tests/test_wide_model.py. The
 * device intrinsics it uses are restated below; g++ -ffp-contract=off gives
 * the same float arithmetic. */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
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
/* one thread that plays a whole block */
static const struct { uint32_t x; } threadIdx = {0}, blockDim = {1};
#define __syncthreads()
static inline void atomicMax(uint32_t* p, uint32_t v) { if (v > *p) *p = v; }
#define __shfl_xor_sync(m, v, o) (v)
#define __any_sync(m, p) (p)
#define __reduce_or_sync(m, v) (v)

#include "../aurora_gb300/csrc/aur_wide.cuh"

using namespace aur;

namespace {
struct Model {
    uint32_t n, levels;
    std::vector<float> verts, box;
    std::vector<uint32_t> perm;
    std::vector<float4> recs;
    std::vector<uint4> wide;
};
}  // namespace

extern "C" {

/* NMH of `count` (even) triangles in NMH order. */
void* wide_model_create(const float* verts, const uint32_t* perm, uint32_t count) {
    Model* m = new Model;
    const uint32_t n = m->n = count / 2;
    m->levels = 0;
    while (n >> m->levels) ++m->levels;
    m->verts.assign(verts, verts + (size_t)count * 9);
    m->perm.assign(perm, perm + count);
    m->box.resize((size_t)n * 6);
    m->recs.assign((size_t)n * kRecStride, make_float4(0, 0, 0, 0));
    for (uint32_t k = n; k-- > 0;) {
        float lo[3], hi[3], r[20];
        const float* c = &m->verts[(size_t)18 * k];
        for (int a = 0; a < 3; ++a) {
            lo[a] = INFINITY; hi[a] = -INFINITY;
            for (int t = 0; t < 2; ++t)
                for (int q = 0; q < 3; ++q) { lo[a] = fminf(lo[a], c[9 * t + 3 * a + q]); hi[a] = fmaxf(hi[a], c[9 * t + 3 * a + q]); }
        }
        const int ax = (31 - __clz(k + 1)) % 3;
        r[0] = lo[ax]; r[1] = hi[ax];
        for (int t = 0; t < 2; ++t)
            for (int a = 0; a < 3; ++a) {
                const float* v = c + 9 * t + 3 * a;
                r[2 + 9 * t + a] = v[0]; r[5 + 9 * t + a] = v[1] - v[0]; r[8 + 9 * t + a] = v[2] - v[0];
            }
        for (uint32_t j = 2 * k + 1; j <= 2 * k + 2 && j < n; ++j)
            for (int a = 0; a < 3; ++a) { lo[a] = fminf(lo[a], m->box[6 * (size_t)j + a]); hi[a] = fmaxf(hi[a], m->box[6 * (size_t)j + 3 + a]); }
        for (int a = 0; a < 3; ++a) { m->box[6 * (size_t)k + a] = lo[a]; m->box[6 * (size_t)k + 3 + a] = hi[a]; }
        float4* rec = &m->recs[(size_t)k * kRecStride];
        memcpy(rec, r, sizeof(r));
        float cb[12];
        for (int j = 0; j < 2; ++j)
            for (int a = 0; a < 3; ++a) {
                const uint32_t g = 2 * k + 1 + j;
                const float l = g < n ? m->box[6 * (size_t)g + a] : 1.0f, h = g < n ? m->box[6 * (size_t)g + 3 + a] : -1.0f;
                const float p = g < n ? 1e-5f * (fabsf(l) + fabsf(h)) + 1e-30f : 0.0f;
                cb[6 * j + a] = l - p; cb[6 * j + 3 + a] = h + p;
            }
        memcpy((float*)rec + 20, cb, sizeof(cb));
    }
    const uint32_t T = (uint32_t)wide_count(m->levels);
    m->wide.assign((size_t)T * kWideStride, make_uint4(0, 0, 0, 0));
    for (uint32_t t = 0; t < T; ++t) wide_record(m->verts.data(), m->box.data(), n, m->levels, t, &m->wide[(size_t)t * kWideStride]);
    return m;
}

void wide_model_destroy(void* p) { delete (Model*)p; }

/* mode 0: closest hit (t, u, v, prim id) per ray; 1: any hit, 1 or 0 in
 * prim; 2: the occluder intersectAny() reports; 3, 4: modes 0 and 1 without
 * the tree (at most kTinyTris triangles). Rays are 8 floats (origin,
 * tmax, direction, pad). steps[i] (optional): treelet steps of ray i.
 * Returns the number of rays that left the treelets for the exact walk's
 * checks to reject, or -1 when a ray took more steps than there are items. */
long wide_model_trace(void* p, const float* rays, uint32_t n, int mode, float* tuv, uint32_t* prim, uint32_t* steps) {
    Model* m = (Model*)p;
    const WideView w{m->recs.data(), m->wide.data(), m->perm.data(), m->verts.data(), m->n, m->levels};
    long changed = 0;
    TinyStage* tiny = nullptr;
    if (mode >= 3) {
        if (2 * m->n > kTinyTris) return -1;
        tiny = new TinyStage;
        stage_tiny(*tiny, m->verts.data(), m->perm.data(), 2 * m->n);
    }
    for (uint32_t i = 0; i < n; ++i) {
        const float* q = rays + 8 * (size_t)i;
        WideRay r;
        WideState s;
        WideHit h;
        uint64_t c = 1;
        const f3 pos = mk3(q[0], q[1], q[2]), dir = mk3(q[4], q[5], q[6]);
        const bool begun = wide_begin(r, s, h, w, pos, dir, q[3]);
        if (mode == 3) tiny_closest(*tiny, 2 * m->n, pos, dir, q[3], h);
        else if (mode == 4) h.best = tiny_any(*tiny, 2 * m->n, pos, dir, q[3]);
        else if (begun) while (mode == 0 ? wide_step<kWideClosest>(w, r, s, h) : mode == 1 ? wide_step<kWideAny>(w, r, s, h) : wide_step<kWideFirst>(w, r, s, h))
            if (++c > 3ull * m->n + 8) return -1;
        if (steps) steps[i] = (uint32_t)c;
        const uint32_t found = h.best;
        float u = 0, v = 0;
        if (mode == 0 || mode == 3) {
            finish_closest(w, r, h, q[3], u, v);
            tuv[3 * (size_t)i] = h.best == kNoPrim ? q[3] : h.t;
            tuv[3 * (size_t)i + 1] = h.best == kNoPrim ? 0.0f : u;
            tuv[3 * (size_t)i + 2] = h.best == kNoPrim ? 0.0f : v;
        } else {
            h.best = finish_any(w, r, h.best, q[3]);
        }
        changed += found != h.best;
        prim[i] = mode == 1 || mode == 4 ? (h.best != kNoPrim) : h.best == kNoPrim ? 0xFFFFFFFFu : m->perm[h.best];
    }
    delete tiny;
    return changed;
}

}  // extern "C"
