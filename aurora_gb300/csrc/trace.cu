// trace.cu — closest-hit and any-hit traversal of the NMH pair-heap.
//
// Results of intersect() / intersectAny() (kernels/lib/intersect.cuh:36-152)
// bit for bit, ties in t to the lower original prim id. A trace runs over the
// treelet records of aur_wide.cuh in three launches. k_trace_packets takes the
// rays in chunks of 32 consecutive rays and traverses each chunk whose rays
// share a direction octant and start close together, as one warp packet when
// their directions are close too, else one ray per lane; the other chunks go
// to k_trace_wide, one ray per lane with finished lanes refilled;
// k_trace_finish checks and stores what both found. A launch that fits the
// GPU at once does without the second, an NMH of a few triangles without all
// three (k_trace_tiny). k_trace walks node by node and is what the counting
// entry points run.
#include <algorithm>

#include "aur_internal.h"
#include "aur_math.cuh"
#include "aur_traverse.cuh"
#include "aur_wide.cuh"

namespace aur {
namespace {

constexpr int kTraceThreads = 128;
constexpr uint32_t kNoRay = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Stores a ray's result (hits: t, u, v, original prim id; occ: the
// occluder's original prim id) as intersect()/intersectAny() report it.
template <bool kAny>
__device__ __forceinline__ void store_result(uint32_t i, uint32_t best, float tmax, float best_t, float bu, float bv,
                                             const uint32_t* __restrict__ perm, float4* __restrict__ hits,
                                             uint32_t* __restrict__ occ) {
    if (kAny) {
        occ[i] = best == kNoPrim ? AUR_NO_HIT : perm[best];
    } else {
        float4 h;
        h.x = best == kNoPrim ? tmax : best_t;
        h.y = best == kNoPrim ? 0.0f : bu;
        h.z = best == kNoPrim ? 0.0f : bv;
        h.w = __uint_as_float(best == kNoPrim ? AUR_NO_HIT : perm[best]);
        hits[i] = h;
    }
}

// First pass of a trace: persistent warps take the rays in chunks of 32
// consecutive rays (one atomic per warp). A chunk whose rays share their
// direction octant and start within `packet_span` of each other stays here:
// as a warp packet (wide_packet: coherent rays, such as a camera's, share the
// treelets they meet) when its directions lie within `dir_span`, else one ray
// per lane (wide_warp). Any other chunk goes to the deferred list for
// k_trace_wide, or is traversed here too when `small`. Compiled for 6 blocks
// per SM (80 registers): at 8 the closest-hit form spills (4.9 ms per 8M
// pinhole rays against 4.3 ms; one node at a time per warp took 7.0 ms).
template <bool kAny>
__global__ void __launch_bounds__(kTraceThreads, 6) k_trace_packets(WideView w, const float4* __restrict__ rays,
                                                                 uint32_t n, float4* __restrict__ hits,
                                                                 uint32_t* __restrict__ occ,
                                                                 uint32_t* __restrict__ ctr,
                                                                 uint32_t* __restrict__ defer, float packet_span,
                                                                 float dir_span, bool small) {
    constexpr WideMode kMode = kAny ? kWideFirst : kWideClosest;
    __shared__ WideQueue s_queue[kTraceThreads / 32];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t chunks = (uint32_t)(((uint64_t)n + 31) >> 5);
    for (;;) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(ctr + 1, 1u);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= chunks) break;
        const uint32_t i = c * 32u + lane;
        const bool valid = i < n;       // lane 0 always has a ray
        f3 pos = mk3(0.0f), dir = mk3(0.0f);
        float tmax = 0.0f;
        if (valid) {
            const float4 r0 = rays[2 * (size_t)i];
            const float4 r1 = rays[2 * (size_t)i + 1];
            pos = mk3(r0.x, r0.y, r0.z);
            dir = mk3(r1.x, r1.y, r1.z);
            tmax = r0.w;
        }
        const uint32_t oct = dir_octant(dir);
        const uint32_t oct0 = __shfl_sync(0xffffffffu, oct, 0);
        const bool mixed = !__all_sync(0xffffffffu, !valid || oct == oct0) || !(warp_span(pos, valid) <= packet_span);
        if (mixed) {
            uint32_t e = 0;
            if (lane == 0) e = atomicAdd(ctr + 2, 1u);
            if (!small) {
                if (lane == 0) defer[e] = c;
                continue;
            }
        }
        WideHit h;
        if (!mixed && warp_span(dir, valid) <= dir_span) {
            WideRay r;
            wide_packet<kMode>(w, valid, oct0, pos, dir, tmax, r, h);
        } else {
            wide_warp<kMode>(w, s_queue[threadIdx.x >> 5], valid, pos, dir, tmax, h);
        }
        if (valid) {
            if (kAny) occ[i] = h.best;
            else hits[i] = make_float4(h.t, h.t2, 0.0f, __uint_as_float(h.best));
        }
    }
}

// The counting kernel (roofline accounting): every ray one per lane, node by
// node. Persistent lanes with dynamic ray fetch: a lane whose ray is done
// takes the next unprocessed ray at once (one atomic per warp for all lanes
// asking together; Aila & Laine, "Understanding the efficiency of ray
// traversal on GPUs", HPG'09). Every ray is traversed as intersect() /
// intersectAny(); kBoxes adds the subtree-box pruning (off to count the
// reference's own node visits). Adds up node fetches, slab crossings
// (triangle tests) and crossings of nodes with children (box loads) into
// counters[0..2]. ctr[0] is the ray fetch counter.
template <bool kAny, bool kBoxes>
__global__ void __launch_bounds__(kTraceThreads, 9) k_trace(const float4* __restrict__ recs, uint32_t nodes,
                                                         const uint32_t* __restrict__ perm,
                                                         const float4* __restrict__ rays, uint32_t n,
                                                         float4* __restrict__ hits, uint32_t* __restrict__ occ,
                                                         unsigned long long* __restrict__ counters,
                                                         uint32_t* __restrict__ ctr, int cap) {
    extern __shared__ uint32_t smem[];
    const int tid = threadIdx.x;
    StackRef stk;
    stk.lo = reinterpret_cast<float*>(smem) + tid;
    stk.hi = reinterpret_cast<float*>(smem + cap * kTraceThreads) + tid;
    stk.stride = kTraceThreads;
    stk.cap = cap;
    uint32_t visits = 0, crossings = 0, inner = 0;
    uint32_t i = kNoRay;
    f3 pos = mk3(0.0f), dir = mk3(0.0f), inv = mk3(0.0f);
    float tmax = 0.0f, best_t = 0.0f, bu = 0.0f, bv = 0.0f;
    uint32_t best = kNoPrim;
    TravState s;
    trav_init(s);
    for (;;) {
        if (i == kNoRay) {
            const uint32_t am = __activemask();
            const int leader = __ffs(am) - 1;
            uint32_t base = 0;
            if ((tid & 31) == leader) base = atomicAdd(ctr, (uint32_t)__popc(am));
            base = __shfl_sync(am, base, leader);
            i = base + __popc(am & lanemask_lt());
            if (i >= n) break;
            const float4 r0 = rays[2 * (size_t)i];
            const float4 r1 = rays[2 * (size_t)i + 1];
            pos = mk3(r0.x, r0.y, r0.z);
            dir = mk3(r1.x, r1.y, r1.z);
            inv = box_inv(dir);
            tmax = best_t = r0.w;
            bu = bv = 0.0f;
            best = kNoPrim;
            trav_init(s);
        }
        Sector s0;
        float4 q5;
        float nlo, nhi;
        bool done;
        if (trav_next(s, recs, nodes, pos, dir, inv, best_t, stk, s0, nlo, nhi, visits)) {
            ++crossings;
            inner += 2 * s.k + 1 < nodes;
            done = node_triangles<kAny>(recs, s.k, s0, perm, pos, dir, best_t, bu, bv, best, q5);
            if (!done) trav_descend<kBoxes>(s, recs, q5, pos, dir, inv, best_t, nodes, stk, nlo, nhi);
        } else {
            done = true;
        }
        if (done) {
            store_result<kAny>(i, best, tmax, best_t, bu, bv, perm, hits, occ);
            i = kNoRay;
        }
    }
    atomicAdd(counters, (unsigned long long)visits);
    atomicAdd(counters + 1, (unsigned long long)crossings);
    atomicAdd(counters + 2, (unsigned long long)inner);
}

// The deferred chunks, one ray per lane over the treelets: a lane takes one
// treelet a step (wide_visit), the warp tests the triangles its lanes met 32
// at a time (WideQueue). Lanes whose ray is done store the raw result (closest
// hit: t, t2, NMH position; any hit: NMH position) and are refilled once
// kRefill of them wait. Compiled for 8 blocks per SM (64 registers, none
// spilled): what bounds it is latency and the issue slots (the box tests'
// integer pipe), not memory. Per 8M random rays over 1M triangles, closest
// hit, before the packed box tests (wide_step) took 0.5 ms off: 8, 9 and 10
// blocks per SM 9.3, 9.7 and 10.0 ms (refilled at 8 lanes, 5, 6, 7 and 8
// blocks: 10.3, 10.5, 10.0 and 9.5); refilled at 1, 2, 4, 6 and 8 waiting
// lanes 10.1, 9.6, 9.3, 9.4 and 9.5 ms; triangles tested by the lane that met
// them instead of the queue 12.2 ms. Now 8.8 ms; the node-by-node kernel it
// replaces took 18.3 ms. Any hit, 4M rays toward a light: 7.2 ms before, 3.7
// ms now.
constexpr int kRefill = 4;

template <bool kAny>
__global__ void __launch_bounds__(kTraceThreads, 8) k_trace_wide(WideView w, const float4* __restrict__ rays, uint32_t n,
                                                                 float4* __restrict__ hits, uint32_t* __restrict__ occ,
                                                                 uint32_t* __restrict__ ctr,
                                                                 const uint32_t* __restrict__ defer) {
    constexpr WideMode kMode = kAny ? kWideFirst : kWideClosest;
    __shared__ WideQueue s_queue[kTraceThreads / 32];
    WideQueue& q = s_queue[threadIdx.x >> 5];
    const uint32_t m = (uint32_t)min((unsigned long long)ctr[2] * 32ull, 0xFFFFFFFFull);
    const uint32_t lane = threadIdx.x & 31;
    uint32_t i = kNoRay, count = 0, seq = 0;
    bool running = false, pool = true;
    WideRay r;
    WideState s;
    float lim = 0.0f;
    wide_ray(r, mk3(0.0f), mk3(0.0f));
    wide_init(s, w.levels);
    for (;;) {
        const uint32_t run = __ballot_sync(0xffffffffu, running);
        if (run == 0u || (pool && __popc(run) <= 32 - kRefill)) {
            queue_test<kMode>(q, lane, count, count, w);
            count = 0;
            if (!running && i != kNoRay) {
                if (kAny) occ[i] = q.best[lane];
                else hits[i] = make_float4(__uint_as_float((uint32_t)(q.key[lane] >> 32)), __uint_as_float(q.t2[lane]),
                                           0.0f, __uint_as_float(q.best[lane]));
                i = kNoRay;
            }
            if (pool) {
                const uint32_t want = ~run;
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(ctr, (uint32_t)__popc(want));
                base = __shfl_sync(0xffffffffu, base, 0);
                pool = base < m && m - base > (uint32_t)__popc(want);
                const uint32_t j = base + __popc(want & lanemask_lt());
                if (!running && j >= base && j < m) {
                    // a chunk's positions past the last ray trace the last ray again (the same result, stored twice)
                    i = min(defer[j >> 5] * 32u + (j & 31u), n - 1u);
                    const float4 r0 = rays[2 * (size_t)i];
                    const float4 r1 = rays[2 * (size_t)i + 1];
                    WideHit h;
                    running = wide_begin(r, s, h, w, mk3(r0.x, r0.y, r0.z), mk3(r1.x, r1.y, r1.z), r0.w);
                    queue_ray<kMode>(q, lane, r.pos, r.dir, r0.w, h.best);
                    lim = r0.w;
                    seq = 0;
                }
            }
            if (!__any_sync(0xffffffffu, running || i != kNoRay)) break;
        }
        uint32_t tris = 0;
        if (running) tris = wide_visit<kMode>(w, r, s, lim);
        queue_add<kMode>(q, lane, count, seq, tris, r, s, w);
        if (running) {
            if (kAny) running = q.key[lane] == kNoKey && wide_next<kMode>(r, s);
            else {
                lim = __uint_as_float((uint32_t)(q.key[lane] >> 32));
                running = wide_next<kMode>(r, s);
            }
        }
    }
}

// Turns what the traversals left in the result buffers (closest hit: t, t2,
// NMH position; any hit: NMH position) into results, checked against the walk
// of intersect() (finish_closest, finish_any) and stored as store_result
// does. Kept apart from the traversals: there the checks would run for a few
// lanes at a time and cost the loop registers (a spill in every step and up
// to twice k_trace_wide's time).
template <bool kAny>
__global__ void __launch_bounds__(kTraceThreads) k_trace_finish(WideView w, const float4* __restrict__ rays, uint32_t n,
                                                                float4* __restrict__ hits,
                                                                uint32_t* __restrict__ occ) {
    const uint32_t step = gridDim.x * kTraceThreads;
    for (uint64_t k = blockIdx.x * kTraceThreads + threadIdx.x; k < n; k += step) {
        const uint32_t i = (uint32_t)k;
        const float4 r0 = rays[2 * (size_t)i];
        const float4 r1 = rays[2 * (size_t)i + 1];
        WideRay r;
        r.pos = mk3(r0.x, r0.y, r0.z);
        r.dir = mk3(r1.x, r1.y, r1.z);
        WideHit h;
        h.t = h.t2 = 0.0f;
        float u = 0.0f, v = 0.0f;
        if (kAny) {
            h.best = finish_any(w, r, occ[i], r0.w);
        } else {
            const float4 raw = hits[i];
            h.t = raw.x;
            h.t2 = raw.y;
            h.best = __float_as_uint(raw.w);
            finish_closest(w, r, h, r0.w, u, v);
        }
        store_result<kAny>(i, h.best, r0.w, h.t, u, v, w.perm, hits, occ);
    }
}

// The rays of an NMH of at most kTinyTris triangles (aur_wide.cuh), in one
// launch: 4099 rays in the 34 triangles of the Cornell box take 18 us a call,
// 23 us with the general launches. Any hit collects the accepted triangles
// and takes the one whose node intersectAny() visits first for the ray's
// octant (preorder ranks, near child first).
template <bool kAny>
__global__ void __launch_bounds__(kTraceThreads) k_trace_tiny(WideView w, uint32_t count,
                                                              const float4* __restrict__ rays, uint32_t n,
                                                              float4* __restrict__ hits, uint32_t* __restrict__ occ,
                                                              uint32_t* __restrict__ ctr) {
    __shared__ __align__(16) TinyStage s_stage;
    __shared__ uint8_t s_rank[8][kTinyTris / 2];
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr[2] = 0u;  // no chunk is deferred
    if (kAny) {
        for (uint32_t j = threadIdx.x; j < 8u * w.nodes; j += blockDim.x) {
            const uint32_t oct = j & 7u, node = j >> 3, lvl = 31u - (uint32_t)__clz(node + 1u);
            uint32_t rank = 0;
            for (uint32_t l = 1; l <= lvl; ++l) {          // down the path: the node before, and a far child's sibling
                const uint32_t k = ((node + 1u) >> (lvl - l)) - 1u;
                const bool second = !(k & 1u), far = second != (((oct >> (l % 3u)) & 1u) != 0u);
                uint32_t size = 0;                         // of the sibling's subtree
                if (far)
                    for (uint32_t f = second ? k - 1u : k + 1u, m = 1; f < w.nodes; f = 2u * f + 1u, m <<= 1)
                        size += min(m, w.nodes - f);
                rank += 1u + size;
            }
            s_rank[oct][node] = (uint8_t)rank;
        }
    }
    stage_tiny(s_stage, w.verts, w.perm, count);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 r0 = rays[2 * (size_t)i];
    const float4 r1 = rays[2 * (size_t)i + 1];
    WideRay r;
    r.pos = mk3(r0.x, r0.y, r0.z);
    r.dir = mk3(r1.x, r1.y, r1.z);
    WideHit h;
    h.t = h.t2 = r0.w;
    h.best = kNoPrim;
    if (kAny) {
        const uint32_t oct = dir_octant(r.dir);
        uint32_t first = ~0u;
        for (uint64_t kept = tiny_filter(s_stage, count, r.pos, r.dir); kept; kept &= kept - 1ull) {
            const uint32_t j = (uint32_t)__ffsll((long long)kept) - 1u;
            float t;
            uint32_t id;
            if (tiny_tri(s_stage, j, r.pos, r.dir, t, id) && t < r0.w)
                first = min(first, ((uint32_t)s_rank[oct][j >> 1] << 8) | j);
        }
        if (first != ~0u) h.best = first & 255u;
    } else {
        tiny_closest(s_stage, count, r.pos, r.dir, r0.w, h);
    }
    float u = 0.0f, v = 0.0f;
    if (kAny) h.best = finish_any(w, r, h.best, r0.w);
    else finish_closest(w, r, h, r0.w, u, v);
    store_result<kAny>(i, h.best, r0.w, h.t, u, v, w.perm, hits, occ);
}

inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

}  // namespace

// Up to this many rays per SM are in flight at once in k_trace_packets, so
// nothing is gained by handing the mixed chunks to a second launch.
constexpr uint32_t kSmallPerSm = 6 * kTraceThreads;

template <typename K>
aur_status persistent_grid(aur_ctx* ctx, K kernel, size_t smem, uint32_t n, uint32_t& grid) {
    int per_sm = 0;
    AUR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTraceThreads, smem));
    grid = std::max(1u, std::min<uint32_t>(cdiv(n, kTraceThreads), (uint32_t)(ctx->sm_count * per_sm)));
    return AUR_OK;
}

// The counting kernel over every ray.
template <bool kAny, bool kBoxes>
aur_status launch_count(aur_ctx* ctx, const aur_nmh* nmh, const float4* r, uint32_t n, float4* h, uint32_t* occ,
                        unsigned long long* counters, cudaStream_t stream, int slot) {
    const int cap = (int)nmh->levels + 1;
    const size_t smem = (size_t)2 * cap * kTraceThreads * sizeof(uint32_t);
    uint32_t* ctr = ctx->d_flags + 16 + 4 * slot;
    AUR_CUDA(cudaMemsetAsync(ctr, 0, 3 * sizeof(uint32_t), stream));
    uint32_t grid = 0;
    const aur_status st = persistent_grid(ctx, k_trace<kAny, kBoxes>, smem, n, grid);
    if (st != AUR_OK) return st;
    k_trace<kAny, kBoxes><<<grid, kTraceThreads, smem, stream>>>(nmh->node_recs, nmh->nodes, nmh->perm, r, n, h, occ,
                                                                 counters, ctr, cap);
    AUR_CUDA(cudaGetLastError());
    return AUR_OK;
}

// The shipped trace: k_trace_packets over all rays, then k_trace_wide and
// k_trace_finish over the chunks it deferred.
template <bool kAny>
aur_status launch_wide(aur_ctx* ctx, const aur_nmh* nmh, const float4* r, uint32_t n, float4* h, uint32_t* occ,
                       cudaStream_t stream, int slot) {
    uint32_t* ctr = ctx->d_flags + 16 + 4 * slot;
    const WideView w = wide_view(nmh);
    if (nmh->count <= kTinyTris) {
        const uint32_t threads = n <= (uint32_t)ctx->sm_count * 64u ? 32u : kTraceThreads;   // a block per SM when they are few
        k_trace_tiny<kAny><<<cdiv(n, threads), threads, 0, stream>>>(w, nmh->count, r, n, h, occ, ctr);
        AUR_CUDA(cudaGetLastError());
        return AUR_OK;
    }
    AUR_CUDA(cudaMemsetAsync(ctr, 0, 3 * sizeof(uint32_t), stream));
    Scratch& d = ctx->defer[slot];
    const size_t need = (size_t)cdiv(n, 32) * sizeof(uint32_t);
    if (d.bytes < need) {
        if (d.ptr) cudaFreeAsync(d.ptr, stream);
        d.ptr = nullptr;
        d.bytes = 0;
        AUR_CHECK(::aur::dev_malloc_async(&d.ptr, need, stream) == cudaSuccess, AUR_ERR_OOM,
                  "trace: out of device memory for %u rays", n);
        d.bytes = need;
    }
    uint32_t* defer = static_cast<uint32_t*>(d.ptr);
    uint32_t grid = 0;
    aur_status st = persistent_grid(ctx, k_trace_packets<kAny>, 0, n, grid);
    if (st != AUR_OK) return st;
    const bool small = n <= (uint32_t)ctx->sm_count * kSmallPerSm;
    k_trace_packets<kAny><<<grid, kTraceThreads, 0, stream>>>(w, r, n, h, occ, ctr, defer, packet_span(nmh), dir_span(nmh), small);
    AUR_CUDA(cudaGetLastError());
    if (!small) {
        st = persistent_grid(ctx, k_trace_wide<kAny>, 0, n, grid);
        if (st != AUR_OK) return st;
        k_trace_wide<kAny><<<grid, kTraceThreads, 0, stream>>>(w, r, n, h, occ, ctr, defer);
        AUR_CUDA(cudaGetLastError());
    }
    st = persistent_grid(ctx, k_trace_finish<kAny>, 0, n, grid);
    if (st != AUR_OK) return st;
    k_trace_finish<kAny><<<grid, kTraceThreads, 0, stream>>>(w, r, n, h, occ);
    AUR_CUDA(cudaGetLastError());
    return AUR_OK;
}

aur_status launch_trace(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, aur_hit* hits,
                        uint32_t* occluder, unsigned long long* counters, cudaStream_t stream, bool pruned,
                        int slot) {
    if (n == 0) return AUR_OK;
    const float4* r = reinterpret_cast<const float4*>(rays);
    float4* h = reinterpret_cast<float4*>(hits);
    if (counters && !pruned)
        return occluder ? launch_count<true, false>(ctx, nmh, r, n, nullptr, occluder, counters, stream, slot)
                        : launch_count<false, false>(ctx, nmh, r, n, h, nullptr, counters, stream, slot);
    if (counters)
        return occluder ? launch_count<true, true>(ctx, nmh, r, n, nullptr, occluder, counters, stream, slot)
                        : launch_count<false, true>(ctx, nmh, r, n, h, nullptr, counters, stream, slot);
    return occluder ? launch_wide<true>(ctx, nmh, r, n, nullptr, occluder, stream, slot)
                    : launch_wide<false>(ctx, nmh, r, n, h, nullptr, stream, slot);
}

}  // namespace aur

using namespace aur;

namespace {

aur_status check_trace_args(aur_ctx* ctx, const aur_nmh* nmh, const void* rays, uint32_t n, const void* out) {
    AUR_CHECK(ctx && nmh, AUR_ERR_INVALID, "trace: null context or NMH");
    AUR_CHECK(n == 0 || (rays && out), AUR_ERR_INVALID, "trace: null ray or result buffer for %u rays", n);
    AUR_CHECK(nmh->device == ctx->device, AUR_ERR_INVALID, "trace: NMH lives on device %d, context on %d",
              nmh->device, ctx->device);
    AUR_CHECK(((uintptr_t)rays & 15) == 0 && ((uintptr_t)out & 3) == 0, AUR_ERR_INVALID,
              "trace: rays must be 16-byte aligned");
    return AUR_OK;
}

// Host-buffer pipeline: chunks of rays alternate between two device slots
// and two launch streams (the context's and an internal one), so the H2D copy
// of chunk c+1 and the D2H copy of chunk c-1 overlap the traversal of c, and
// the traversal of c+1 starts while the last rays of c drain. Each slot has
// its own counters and deferred list, as its kernels may run concurrently
// with the other's. Chunks hold 8M rays, except a first chunk of 2M (its
// copy in waits for nothing to overlap) and, where the rays allow, a last
// chunk of 2M (its copy out likewise): 2^24 rays go as 2M, 8M, 4M, 2M, which
// measured 636 Mrays/s end to end against 605 for even chunks of 4M.
aur_status trace_host(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, void* out, bool any) {
    aur_status st = check_trace_args(ctx, nmh, rays, n, out);
    if (st != AUR_OK) return st;
    if (n == 0) return AUR_OK;
    AUR_CUDA(cudaSetDevice(ctx->device));
    const uint32_t chunk = 1u << 23;
    const size_t out_sz = any ? sizeof(uint32_t) : sizeof(aur_hit);
    for (int s = 0; s < 2; ++s) {
        const size_t need_in = (size_t)chunk * sizeof(aur_ray), need_out = (size_t)chunk * out_sz;
        if (ctx->pipe[s].bytes < need_in) {
            cudaFree(ctx->pipe[s].ptr);
            ctx->pipe[s].ptr = nullptr; ctx->pipe[s].bytes = 0;
            AUR_CHECK(::aur::dev_malloc(&ctx->pipe[s].ptr, need_in) == cudaSuccess, AUR_ERR_OOM, "trace_host: out of memory");
            ctx->pipe[s].bytes = need_in;
        }
        if (ctx->out[s].bytes < need_out) {
            cudaFree(ctx->out[s].ptr);
            ctx->out[s].ptr = nullptr; ctx->out[s].bytes = 0;
            AUR_CHECK(::aur::dev_malloc(&ctx->out[s].ptr, need_out) == cudaSuccess, AUR_ERR_OOM, "trace_host: out of memory");
            ctx->out[s].bytes = need_out;
        }
    }
    cudaEvent_t* in_done = ctx->ev;
    cudaEvent_t* comp_done = ctx->ev + 2;
    cudaEvent_t* out_done = ctx->ev + 4;
    // the copy and second launch streams start after work already queued on the launch stream
    AUR_CUDA(cudaEventRecord(ctx->ev[6], ctx->stream));
    AUR_CUDA(cudaStreamWaitEvent(ctx->copy_in, ctx->ev[6], 0));
    AUR_CUDA(cudaStreamWaitEvent(ctx->compute2, ctx->ev[6], 0));
    cudaStream_t const launch[2] = {ctx->stream, ctx->compute2};
    bool used[2] = {false, false};
    uint32_t m = 0;
    for (uint32_t c0 = 0, c = 0; c0 < n; c0 += m, ++c) {
        const int s = (int)(c & 1);
        // a quarter chunk first (the first copy is not overlapped) and last
        // (nor is the last copy back); full chunks between
        const uint32_t left = n - c0;
        uint32_t want = c == 0 ? chunk / 4 : chunk;
        if (c > 0 && left > chunk / 2 && left <= chunk + chunk / 4) want = left - chunk / 4;
        m = left < want ? left : want;
        if (used[s]) AUR_CUDA(cudaStreamWaitEvent(ctx->copy_in, out_done[s], 0));
        AUR_CUDA(cudaMemcpyAsync(ctx->pipe[s].ptr, rays + c0, (size_t)m * sizeof(aur_ray), cudaMemcpyHostToDevice,
                                 ctx->copy_in));
        AUR_CUDA(cudaEventRecord(in_done[s], ctx->copy_in));
        AUR_CUDA(cudaStreamWaitEvent(launch[s], in_done[s], 0));
        st = launch_trace(ctx, nmh, (const aur_ray*)ctx->pipe[s].ptr, m, any ? nullptr : (aur_hit*)ctx->out[s].ptr,
                          any ? (uint32_t*)ctx->out[s].ptr : nullptr, nullptr, launch[s], true, s);
        if (st != AUR_OK) return st;
        AUR_CUDA(cudaEventRecord(comp_done[s], launch[s]));
        AUR_CUDA(cudaStreamWaitEvent(ctx->copy_out, comp_done[s], 0));
        AUR_CUDA(cudaMemcpyAsync((char*)out + (size_t)c0 * out_sz, ctx->out[s].ptr, (size_t)m * out_sz,
                                 cudaMemcpyDeviceToHost, ctx->copy_out));
        AUR_CUDA(cudaEventRecord(out_done[s], ctx->copy_out));
        used[s] = true;
    }
    AUR_CUDA(cudaStreamSynchronize(ctx->copy_out));
    AUR_CUDA(cudaStreamSynchronize(ctx->compute2));
    AUR_CUDA(cudaStreamSynchronize(ctx->stream));
    return AUR_OK;
}

}  // namespace

extern "C" {

aur_status aur_trace_closest(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, aur_hit* hits) {
    AUR_RANGE("aur_trace_closest");
    aur_status st = check_trace_args(ctx, nmh, rays, n, hits);
    if (st != AUR_OK) return st;
    AUR_CUDA(cudaSetDevice(ctx->device));
    return launch_trace(ctx, nmh, rays, n, hits, nullptr, nullptr, ctx->stream, true);
}

aur_status aur_trace_any(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, uint32_t* occluder) {
    AUR_RANGE("aur_trace_any");
    aur_status st = check_trace_args(ctx, nmh, rays, n, occluder);
    if (st != AUR_OK) return st;
    AUR_CUDA(cudaSetDevice(ctx->device));
    return launch_trace(ctx, nmh, rays, n, nullptr, occluder, nullptr, ctx->stream, true);
}

aur_status aur_trace_closest_host(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, aur_hit* hits) {
    AUR_RANGE("aur_trace_closest_host");
    return trace_host(ctx, nmh, rays, n, hits, false);
}

aur_status aur_trace_any_host(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, uint32_t* occluder) {
    AUR_RANGE("aur_trace_any_host");
    return trace_host(ctx, nmh, rays, n, occluder, true);
}

namespace {

// Runs closest hit and any hit over n device rays with the counting kernels;
// out[0..2] closest (fetches, crossings, inner crossings), out[3..5] any hit.
aur_status count_work(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n, bool pruned,
                      unsigned long long out[6]) {
    for (int q = 0; q < 6; ++q) out[q] = 0;
    if (n == 0) return AUR_OK;
    void* scratch = nullptr;
    const size_t bytes = 256 + (size_t)n * sizeof(aur_hit);
    AUR_CHECK(::aur::dev_malloc_async(&scratch, bytes, ctx->stream) == cudaSuccess, AUR_ERR_OOM,
              "trace counters: out of memory");
    unsigned long long* cnt = (unsigned long long*)scratch;
    aur_hit* hits = (aur_hit*)((char*)scratch + 256);
    cudaMemsetAsync(cnt, 0, 48, ctx->stream);
    aur_status st = launch_trace(ctx, nmh, rays, n, hits, nullptr, cnt, ctx->stream, pruned);
    if (st == AUR_OK) st = launch_trace(ctx, nmh, rays, n, nullptr, (uint32_t*)hits, cnt + 3, ctx->stream, pruned);
    unsigned long long host[6] = {0, 0, 0, 0, 0, 0};
    cudaMemcpyAsync(host, cnt, 48, cudaMemcpyDeviceToHost, ctx->stream);
    cudaFreeAsync(scratch, ctx->stream);
    AUR_CUDA(cudaStreamSynchronize(ctx->stream));
    if (st != AUR_OK) return st;
    for (int q = 0; q < 6; ++q) out[q] = host[q];
    return AUR_OK;
}

}  // namespace

aur_status aur_trace_count_visits(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n,
                                  unsigned long long node_visits[2]) {
    AUR_RANGE("aur_trace_count_visits");
    AUR_CHECK(node_visits, AUR_ERR_INVALID, "aur_trace_count_visits: null output");
    aur_status st = check_trace_args(ctx, nmh, rays, n, rays);
    if (st != AUR_OK) return st;
    AUR_CUDA(cudaSetDevice(ctx->device));
    unsigned long long c[6];
    st = count_work(ctx, nmh, rays, n, false, c);
    node_visits[0] = c[0];
    node_visits[1] = c[3];
    return st;
}

aur_status aur_debug_trace_deferred(aur_ctx* ctx, uint32_t* chunks) {
    AUR_CHECK(ctx && chunks, AUR_ERR_INVALID, "aur_debug_trace_deferred: null argument");
    AUR_CUDA(cudaSetDevice(ctx->device));
    AUR_CUDA(cudaMemcpyAsync(chunks, ctx->d_flags + 16 + 2, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
    AUR_CUDA(cudaStreamSynchronize(ctx->stream));
    return AUR_OK;
}

aur_status aur_trace_stats(aur_ctx* ctx, const aur_nmh* nmh, const aur_ray* rays, uint32_t n,
                           aur_trace_work* closest, aur_trace_work* any) {
    AUR_RANGE("aur_trace_stats");
    AUR_CHECK(closest && any, AUR_ERR_INVALID, "aur_trace_stats: null output");
    aur_status st = check_trace_args(ctx, nmh, rays, n, rays);
    if (st != AUR_OK) return st;
    AUR_CUDA(cudaSetDevice(ctx->device));
    unsigned long long c[6];
    st = count_work(ctx, nmh, rays, n, true, c);
    closest->node_fetches = c[0];
    closest->slab_crossings = c[1];
    closest->box_loads = c[2];
    any->node_fetches = c[3];
    any->slab_crossings = c[4];
    any->box_loads = c[5];
    return st;
}

}  // extern "C"
