// adjoint.cu — path-replay backpropagation through the integrator.
//
// Gradients of a loss L(image) with respect to every shader's diffuse colour,
// every shader's emission colour and every light's colour, given dL/dimage.
// No counterpart in the
// reference. Method: path replay backpropagation (D. Vicini, S. Speierer,
// W. Jakob, "Path Replay Backpropagation", ACM TOG 40(4), 2021), in one pass
// per camera sample: the integrator's ray stack (monteCarloRaytracer.cu:26-88,
// the same estimator and counter-RNG draws as aur_render) is walked again,
// and at vertex k with throughput T_k and Lambert colour
// c_k = diffuse_color * diffuse the replay adds
//   dL/dc_k  += g * (T_k * D_k / c_k + L_after_k / c_k)
//   dL/dcolor_l += g * T_k * dD_k/dcolor_l
// where D_k is the direct light at k (ambient, delta and area terms,
// radiance.cuh:13-80), g = dL/dpixel / spp, and L_after_k the radiance of
// the rays that descend from k's diffuse bounce (c_k enters the throughput
// f*|cos|/pdf of every later vertex, BSDF::samplef, bsdf.cuh:222-236). The
// rays that descend from a bounce are exactly those traced between its pop
// and the stack's return to its height before the push (depth first), so a
// marker per pending bounce sums that radiance and hands it over when the
// subtree ends; no primal pass is needed. D_k / c_k is evaluated directly
// (f replaced by 1/pi), so the direct part needs no division; the
// later-vertex part divides by c_k and is skipped for colour channels that
// are exactly zero.
// Emission E_s of shader s enters linearly: at every vertex on s as T_k * E_s
// (times the emission's MIS weight in AUR_MODE_PATH_MIS,
// monteCarloRaytracer.cu:42), and in AUR_MODE_PATH_MIS through the emitter
// sample of every vertex, f * E_s * G with G the sample's geometric factor
// over its density. So
//   dL/dE_s += g * T_k * w_k  (vertex on s),  g * T_k * f_k * G  (emitter on s, visible).
// Neither the MIS weights nor the light-selection table depend on E_s: the
// table weighs triangles by the shader's scalar `emission` times area
// (emitter.cu's weight), not by its emission colour.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "aur_integrate.cuh"
#include "aur_internal.h"

namespace aur {
namespace {

constexpr int kAdjThreads = 128;
// Resident blocks per SM that the replay kernel is compiled for: its lanes
// diverge and it waits on latency and instruction fetch, so more warps pay for
// the spills. Without a ray stack (replay_diffuse), 256x256: per-warp sums, 16
// samples of a 4130-triangle box with a shader each: 3.80 ms at 8 blocks, 3.65
// at 10, 3.73 at 12, 3.97 at 14, in the MIS mode (8 samples) 2.81, 2.70, 2.69
// and 2.58; a thread's own sums, the 34-triangle box (8 samples): 0.64 ms at 8,
// 0.65 at 9, 0.66 at 10, 0.67 at 12. With the stack: 4.49 ms at 8, 4.33 at 10,
// 4.35 at 12, 4.42 at 14, in the MIS mode 3.41, 3.11, 2.99 and 2.88; own sums
// (100k-triangle spheres) 2.13 at 8, 2.14 at 10, 2.25 at 12.
constexpr int adj_blocks(bool generic, bool few) { return generic ? (few ? 10 : 12) : (few ? 8 : 10); }
constexpr uint32_t kSharedLights = 64;

// Per-unit-colour radiance of a light sample (Lr = color * s), light.cuh:228-259.
__device__ __forceinline__ float light_scale(const aur_light& L, const f3& dir, float t) {
    if (L.type == AUR_LIGHT_AMBIENT) return L.intensity * (1.0f - L.ambient);
    if (L.type == AUR_LIGHT_POINT) return L.intensity / (t * t);
    if (L.type == AUR_LIGHT_DIRECTIONAL) return L.intensity;
    return L.intensity * fmaxf(0.0f, dot(from(L.direction), -dir));
}

// Where a thread's shader gradients go. kFew (at most kFewShaders shaders):
// into the thread's own sums (local memory: the shader is known at run time
// only), which the block adds up once its samples are done; else to the
// result, summed first over the lanes of the warp that hit the same shader
// (large triangles are hit by most of a warp), one atomic per shader and
// component. A library reduction per shader group ran the groups one after
// the other: 5.2 ms on a 4130-triangle box with a shader each, 4.3 ms in
// rounds over all groups at once. The own sums pay where a warp meets few
// shaders often: 0.58 ms against 0.78 in rounds on the 34-triangle box (three
// shaders, 256x256, 8 samples), 1.30 against 1.43 in the MIS mode on the
// emissive box; on 100k-triangle spheres both take 1.77 ms with 2 to 64
// shaders. Room for 16 shaders costs the box 5 % (0.61 ms), for 32 the spheres
// 6 % (1.88).
constexpr uint32_t kFewShaders = 8;

template <bool kFew>
struct ShaderGrads {
    float* diffuse;      // 3 per shader
    float* emission;     // 3 per shader, or null
    float sum[kFew ? 6 * kFewShaders : 1];

    __device__ __forceinline__ void clear() {
        if (kFew)
            for (uint32_t k = 0; k < 6 * kFewShaders; ++k) sum[k] = 0.0f;
    }
    // Adds g to shader si's entry.
    __device__ __forceinline__ void add(bool to_emission, uint32_t si, const f3& g) {
        if constexpr (kFew) {
            float* s = sum + (to_emission ? 3 * kFewShaders : 0u) + 3 * si;
            s[0] += g.x;
            s[1] += g.y;
            s[2] += g.z;
        } else {
            // lanes of one shader in pairs, neighbours in rank first, all
            // shaders at once: at most five rounds
            const uint32_t here = __activemask(), lane = threadIdx.x & 31;
            const uint32_t peers = __match_any_sync(here, si);
            uint32_t rank = __popc(peers & ((1u << lane) - 1u));
            uint32_t above = peers & (0xFFFFFFFEu << lane);
            const bool first = rank == 0;
            f3 x = g;
            while (__any_sync(here, above != 0u)) {
                const int next = __ffs(above);
                const int src = next ? next - 1 : (int)lane;
                const float ax = __shfl_sync(here, x.x, src), ay = __shfl_sync(here, x.y, src),
                            az = __shfl_sync(here, x.z, src);
                if (next) x = x + mk3(ax, ay, az);
                above &= __ballot_sync(here, !(rank & 1u));
                rank >>= 1;
            }
            if (first && (x.x != 0.0f || x.y != 0.0f || x.z != 0.0f)) {
                float* d = (to_emission ? emission : diffuse) + 3 * (size_t)si;
                atomicAdd(d + 0, x.x);
                atomicAdd(d + 1, x.y);
                atomicAdd(d + 2, x.z);
            }
        }
    }
    // Adds g_c1 * d(colour1)/d(diffuse_color) = g_c1 * diffuse to shader si's
    // gradient (colour1 = diffuse_color * diffuse; a textured shader's colour
    // is not its diffuse_color, so it gets none).
    __device__ __forceinline__ void add_diffuse(uint32_t si, const aur_shader* sh, const f3& g_c1) {
        add(false, si, sh->texture > 0 ? mk3(0.0f) : g_c1 * sh->diffuse);
    }
};

// Direct light at a hit as the primal computes it (direct_light), with its
// derivatives: Dp receives the direct light per unit Lambert colour, and the
// light-colour gradients g * thr * d(direct)/d(colour_l) are added (light 0
// into gl0, the others to d_light). ew: the emission's MIS weight; bounce:
// whether a diffuse bounce follows the hit (both for AUR_MODE_PATH_MIS).
// With an emission result, the emission gradients of the hit's own shader si and of
// the emitter sample's shader are added too.
template <bool kMis, typename Trav, typename Grads>
__device__ __forceinline__ f3 direct_grad(const SceneView& sc, const aur_shader* sh, const Bsdf& b, const f3& f,
                                          const f3& position, const f3& wo, float ew, bool bounce, uint32_t seed,
                                          uint32_t scene, uint32_t pixel, uint32_t sample, uint32_t rix, const f3& thr,
                                          const f3& g, float* __restrict__ d_light, f3& gl0, f3& Dp,
                                          Grads& grads, uint32_t si, const Trav& trav) {
    f3 Li = kMis ? from(sh->emission_color) * ew : from(sh->emission_color);
    if (grads.emission) grads.add(true, si, kMis ? (g * thr) * ew : g * thr);
    Dp = mk3(0.0f);   // direct light per unit Lambert colour
    for (uint32_t i = 0; i < sc.num_lights; ++i) {
        const aur_light& L = sc.lights[i];
        f3 dl = mk3(0.0f);   // d(direct)/d(light colour), per channel
        if (L.type == AUR_LIGHT_AMBIENT) {
            const f3 X = (from(L.color) * L.intensity) * L.ambient;
            Li = Li + f * X;
            Dp = Dp + X * kInvPi;
            dl = dl + f * (L.intensity * L.ambient);
        }
        if (L.type != AUR_LIGHT_AREA) {
            f3 wdir; float wt, pdf;
            const f3 Ls = sample_light(L, position, seed, scene, pixel, sample, rix, 0u, wdir, wt, pdf);
            if (pdf > 0.0f && !zero(Ls)) {
                if (!zero(f) && !occluded(sc, trav, position, wdir, wt)) {
                    const float cs = fmaxf(0.0f, dot(wdir, b.N));
                    Li = Li + f * Ls * cs;
                    Dp = Dp + Ls * (kInvPi * cs);
                    dl = dl + f * (light_scale(L, wdir, wt) * cs);
                }
            }
        } else if (kMis) {
            // both strategies of every sample, as in direct_light_mis
            f3 acc = mk3(0.0f), accp = mk3(0.0f), accl = mk3(0.0f);
            const AreaLightMis q = area_light_setup(L, f);
            if (q.active) {
                for (int32_t j = 0; j < L.samples; ++j) {
                    f3 Ls = mk3(0.0f);
                    for (int h2 = 0; h2 < 2; ++h2) {
                        const ShadowSample ss =
                            h2 == 0 ? area_light_sample(q, i, (uint32_t)j, b, f, position, wo, seed, scene, pixel,
                                                        sample, rix)
                                    : area_bsdf_sample(q, i, (uint32_t)j, b, f, position, wo, seed, scene, pixel,
                                                       sample, rix);
                        const float tt = ss.tmax;
                        if (ss.cand && !occluded(sc, trav, ss.o, ss.d, tt)) {
                            Ls = Ls + ss.c;
                            accp = accp + ss.e * (ss.geo * kInvPi);
                            accl = accl + f * (L.intensity * ss.geo);
                        }
                    }
                    acc = acc + Ls;
                }
            }
            const float ns = (float)L.samples;
            Li = Li + mk3(acc.x / ns, acc.y / ns, acc.z / ns);
            Dp = Dp + mk3(accp.x / ns, accp.y / ns, accp.z / ns);
            dl = dl + mk3(accl.x / ns, accl.y / ns, accl.z / ns);
        } else {
            f3 acc = mk3(0.0f), accp = mk3(0.0f), accl = mk3(0.0f);
            for (int32_t j = 0; j < L.samples; ++j) {
                f3 wdir; float wt, lpdf;
                const f3 Lr = sample_light(L, position, seed, scene, pixel, sample, rix, light_slot(i, (uint32_t)j),
                                           wdir, wt, lpdf);
                f3 wpos = position;
                wpos.x += kEpsilon * wdir.x;
                wpos.y += kEpsilon * wdir.y;
                wpos.z += kEpsilon * wdir.z;
                wt += kEpsilon;
                if (lpdf > 0.0f && !zero(Lr)) {
                    if (!zero(f) && !occluded(sc, trav, wpos, wdir, wt)) {
                        const float cs = fmaxf(0.0f, dot(wdir, b.N));
                        acc = acc + f * Lr * cs;
                        accp = accp + Lr * (kInvPi * cs);
                        accl = accl + f * (light_scale(L, wdir, wt - kEpsilon) * cs);
                    }
                }
            }
            const float ns = (float)L.samples;
            Li = Li + mk3(acc.x / ns, acc.y / ns, acc.z / ns);
            Dp = Dp + mk3(accp.x / ns, accp.y / ns, accp.z / ns);
            dl = dl + mk3(accl.x / ns, accl.y / ns, accl.z / ns);
        }
        const f3 gl = g * thr * dl;
        if (i == 0) {
            gl0 = gl0 + gl;
        } else if (gl.x != 0.0f || gl.y != 0.0f || gl.z != 0.0f) {
            atomicAdd(d_light + 3 * i + 0, gl.x);
            atomicAdd(d_light + 3 * i + 1, gl.y);
            atomicAdd(d_light + 3 * i + 2, gl.z);
        }
    }
    if (kMis) {   // the emitter sample (direct_light_mis)
        const ShadowSample ss =
            emitter_shadow_sample(sc, b, f, position, wo, bounce, seed, scene, pixel, sample, rix);
        const float tt = ss.tmax;
        const bool vis = ss.cand && !occluded(sc, trav, ss.o, ss.d, tt);
        Li = Li + (vis ? ss.c : mk3(0.0f));
        if (vis) Dp = Dp + ss.e * (ss.geo * kInvPi);
        if (grads.emission && vis) grads.add(true, ss.esi, (g * thr) * (f * ss.geo));
    }
    return Li;
}

// The replay of one camera sample: integrate()'s ray stack
// (monteCarloRaytracer.cu:26-88) walked again with the same draws. A hit's
// colour Li * thr depends on its own vertex's colour through the direct
// light, and on the colour of every vertex whose diffuse bounce lies on its
// way from the camera through thr, as a factor. The rays that descend from a
// diffuse bounce are exactly those traced between its pop and the return of
// the stack to the height it had before the bounce was pushed (depth first),
// so a marker per pending bounce sums its subtree's radiance; when the
// subtree ends, g * subtree / c_k goes to the bouncing vertex's shader.
// Gradients of light 0 are summed in `gl0` (reduced once per block by the
// caller); those of further lights go to d_light with atomics. kMis:
// AUR_MODE_PATH_MIS, whose MIS weights do not depend on the colours (Lambert
// densities are |cos| / pi), so every direct term stays linear in the vertex
// colour and in the light colour. One pass replaces a primal pass (each
// sample's radiance) plus a replay: 29.3 -> 21.1 ms on the differentiable
// workload (256x256, 64 spp, path mode).
template <bool kMis, typename Trav, typename Grads>
__device__ void replay_stack(const SceneView& sc, uint32_t max_depth, uint32_t mode, uint32_t seed, uint32_t scene,
                             uint32_t pixel, uint32_t sample, const PathRay& primary, const Trav& trav,
                             const f3& g, Grads& grads, float* __restrict__ d_light, f3& gl0, uint32_t* err) {
    struct Marker {
        f3 col0, c1;          // colour before the subtree, the bouncing vertex's Lambert colour
        const aur_shader* sh;
        uint32_t si;
        int base;             // stack height before the bounce was pushed
    };
    PathRay stack[AUR_MAX_DEPTH + 2];
    Marker mk[AUR_MAX_DEPTH + 2];
    int sp = 0, nm = 0;
    stack[sp++] = primary;
    int depth = 0;
    f3 col = mk3(0.0f);
    uint32_t ray_index = 0;
    const int maxd = (int)max_depth;
    const bool path = kMis || mode == AUR_MODE_PATH;
    auto close = [&](const Marker& m) {
        const f3 sub = col - m.col0;
        f3 dc;
        dc.x = m.c1.x != 0.0f ? sub.x / m.c1.x : 0.0f;
        dc.y = m.c1.y != 0.0f ? sub.y / m.c1.y : 0.0f;
        dc.z = m.c1.z != 0.0f ? sub.z / m.c1.z : 0.0f;
        grads.add_diffuse(m.si, m.sh, g * dc);
    };
    for (;;) {
        while (nm > 0 && sp <= mk[nm - 1].base) close(mk[--nm]);
        if (!(depth <= maxd && sp > 0)) break;
        PathRay ray = stack[--sp];
        const uint32_t rix = ray_index++;
        float t = kInfinity, u = 0.0f, v = 0.0f;
        const uint32_t tri = closest_hit(sc, trav, ray.pos, ray.dir, t, u, v);
        if (tri == kNoPrim) continue;
        const f3 position = ray.pos + (ray.dir * t);
        const f3 wo = -ray.dir;
        const uint32_t sid = sc.sids[tri];
        const uint32_t si = sid > 0 ? sid - 1 : 0;
        const aur_shader* sh = sc.shaders + si;
        const float refl = sh->reflectivity, trans = sh->translucence;
        const Bsdf b = get_bsdf(sc, sh, tri, u, v);
        const f3 f = bsdf_f(b);
        const bool specular = refl > 0.0f || trans > 0.0f;
        const bool bounce_follows = !specular && depth + 1 <= maxd;   // as direct_light is told in the primal
        const float ew = kMis ? emission_weight(sc, tri, ray.dir, t, ray.pdf) : 1.0f;
        // the continuation changes the ray's throughput before the colour
        // update; the direct light's derivatives scale with that throughput
        PathRay cur = ray;
        const Continuation kc =
            continue_ray<kMis>(sh, b, cur, position, wo, path, depth, maxd, seed, scene, pixel, sample, rix);
        f3 Dp;
        const f3 Li = direct_grad<kMis>(sc, sh, b, f, position, wo, ew, bounce_follows, seed, scene, pixel, sample, rix,
                                        cur.thr, g, d_light, gl0, Dp, grads, si, trav);
        grads.add_diffuse(si, sh, g * (cur.thr * Dp));
        col = col + Li * cur.thr;
        for (int q = 0; q < kc.n; ++q) {
            if (kc.bounced && q == kc.n - 1) {   // the diffuse bounce: its subtree scales with this vertex's colour
                Marker m;
                m.col0 = col;
                m.c1 = b.color1;
                m.sh = sh;
                m.si = si;
                m.base = sp;
                mk[nm++] = m;
            }
            if (sp < AUR_MAX_DEPTH + 2) stack[sp++] = kc.ray[q]; else atomicOr(err, 2u);
        }
    }
    while (nm > 0) close(mk[--nm]);
}

// The same replay for scenes without specular shaders: one ray in flight per
// sample, no ray stack, and every subtree is the rest of the path, so all of
// them end where the path does. Same operations in the same order as
// replay_stack(). What bounds the replay is instruction fetch and the local
// memory of its stack: without stack, reflection and refraction the box of
// adj_blocks takes 3.65 ms (4.35 with them), the 34-triangle box 0.64 (0.86).
template <bool kMis, typename Trav, typename Grads>
__device__ __forceinline__ void replay_diffuse(const SceneView& sc, uint32_t max_depth, uint32_t mode, uint32_t seed,
                                               uint32_t scene, uint32_t pixel, uint32_t sample, const PathRay& primary,
                                               const Trav& trav, const f3& g, Grads& grads,
                                               float* __restrict__ d_light, f3& gl0) {
    struct Marker {
        f3 col0, c1;          // colour before the subtree, the bouncing vertex's Lambert colour
        uint32_t si;
    };
    Marker mk[AUR_MAX_DEPTH];
    uint32_t nm = 0;          // bounces, also the depth
    f3 pos = primary.pos, dir = primary.dir, thr = primary.thr, col = mk3(0.0f);
    float prev_pdf = 0.0f;
    const bool path = kMis || mode == AUR_MODE_PATH;
    for (;;) {
        float t = kInfinity, u = 0.0f, v = 0.0f;
        const uint32_t tri = closest_hit(sc, trav, pos, dir, t, u, v);
        if (tri == kNoPrim) break;
        const f3 position = pos + (dir * t);
        const f3 wo = -dir;
        const uint32_t sid = sc.sids[tri];
        const uint32_t si = sid > 0 ? sid - 1 : 0;
        const aur_shader* sh = sc.shaders + si;
        const Bsdf b = get_bsdf(sc, sh, tri, u, v);
        const f3 f = bsdf_f(b);
        const float ew = kMis ? emission_weight(sc, tri, dir, t, prev_pdf) : 1.0f;
        f3 Dp;
        const f3 Li = direct_grad<kMis>(sc, sh, b, f, position, wo, ew, nm + 1 <= max_depth, seed, scene, pixel, sample,
                                        nm, thr, g, d_light, gl0, Dp, grads, si, trav);
        grads.add_diffuse(si, sh, g * (thr * Dp));
        col = col + Li * thr;
        if (!path || nm + 1 > max_depth) break;
        f3 wi, nthr;
        if (!(kMis ? mis_bounce(b, wo, thr, seed, scene, pixel, sample, nm, wi, nthr, prev_pdf)
                   : diffuse_bounce(b, wo, thr, seed, scene, pixel, sample, nm, wi, nthr, prev_pdf)))
            break;
        mk[nm].col0 = col;
        mk[nm].c1 = b.color1;
        mk[nm].si = si;
        ++nm;
        pos = position;
        dir = wi;
        thr = nthr;
    }
    while (nm > 0) {
        const Marker m = mk[--nm];
        const f3 sub = col - m.col0;
        f3 dc;
        dc.x = m.c1.x != 0.0f ? sub.x / m.c1.x : 0.0f;
        dc.y = m.c1.y != 0.0f ? sub.y / m.c1.y : 0.0f;
        dc.z = m.c1.z != 0.0f ? sub.z / m.c1.z : 0.0f;
        grads.add_diffuse(m.si, sc.shaders + m.si, g * dc);
    }
}

// Replay kernel: one thread per camera sample of samples [s0, s0 + nb). kGeneric: the scene has specular shaders;
// kFew: at most kFewShaders shaders.
template <bool kGeneric, bool kMis, bool kTiny, bool kFew>
__global__ void __launch_bounds__(kAdjThreads, adj_blocks(kGeneric, kFew)) k_adj_replay(SceneView sc, aur_camera cam,
                                                                            aur_render_params p, uint32_t s0,
                                                                            uint32_t nb,
                                                                            const float4* __restrict__ d_image,
                                                                            float* __restrict__ d_diffuse,
                                                                            float* __restrict__ d_light,
                                                                            float* __restrict__ d_emission,
                                                                            uint32_t shaders,
                                                                            uint32_t* __restrict__ err) {
    const auto trav = make_trav<kTiny>(sc);
    __shared__ float s_light[3 * kSharedLights];
    // light gradients are reduced in shared memory first (one light is hit by every sample)
    const bool shared_lights = sc.num_lights <= kSharedLights;
    if (shared_lights)
        for (uint32_t i = threadIdx.x; i < 3 * sc.num_lights; i += kAdjThreads) s_light[i] = 0.0f;
    __syncthreads();
    const uint64_t P = (uint64_t)p.width * p.height;
    f3 gl0 = mk3(0.0f);
    ShaderGrads<kFew> grads;
    grads.diffuse = d_diffuse;
    grads.emission = d_emission;
    grads.clear();
    const uint64_t t = (uint64_t)blockIdx.x * kAdjThreads + threadIdx.x;
    if (t < P * nb) {
        const uint32_t pix = (uint32_t)(t % P);
        const uint32_t s = s0 + (uint32_t)(t / P);
        const PathRay r = camera_ray(cam, p.width, p.height, pix % p.width, pix / p.width, s, p.spp);
        const float4 di = d_image[pix];
        const float w = 1.0f / (float)p.spp;
        const f3 g = mk3(di.x * w, di.y * w, di.z * w);
        float* dl = shared_lights ? s_light : d_light;
        if constexpr (kGeneric)
            replay_stack<kMis>(sc, p.max_depth, p.mode, p.seed, p.scene_id, pix, s, r, trav, g, grads, dl, gl0, err);
        else
            replay_diffuse<kMis>(sc, p.max_depth, p.mode, p.seed, p.scene_id, pix, s, r, trav, g, grads, dl, gl0);
    }
    if constexpr (kFew) {      // the block's sums, one atomic per entry
        __shared__ float s_sum[kAdjThreads / 32][6 * kFewShaders];
        const uint32_t lane = threadIdx.x & 31;
        for (uint32_t k = 0; k < 6 * kFewShaders; ++k) {
            float x = grads.sum[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == 0) s_sum[threadIdx.x >> 5][k] = x;
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < 6 * kFewShaders; k += kAdjThreads) {
            const bool em = k >= 3 * kFewShaders;
            const uint32_t e = em ? k - 3 * kFewShaders : k;
            float x = 0.0f;
            for (int q = 0; q < kAdjThreads / 32; ++q) x += s_sum[q][k];
            if (e < 3 * shaders && x != 0.0f && (!em || d_emission)) atomicAdd((em ? d_emission : d_diffuse) + e, x);
        }
    }
    // light 0: warp sum, then one shared atomic per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gl0.x += __shfl_down_sync(0xffffffffu, gl0.x, o);
        gl0.y += __shfl_down_sync(0xffffffffu, gl0.y, o);
        gl0.z += __shfl_down_sync(0xffffffffu, gl0.z, o);
    }
    if ((threadIdx.x & 31) == 0 && sc.num_lights > 0) {
        float* dst = shared_lights ? s_light : d_light;
        atomicAdd(dst + 0, gl0.x);
        atomicAdd(dst + 1, gl0.y);
        atomicAdd(dst + 2, gl0.z);
    }
    __syncthreads();
    if (shared_lights)
        for (uint32_t i = threadIdx.x; i < 3 * sc.num_lights; i += kAdjThreads)
            if (s_light[i] != 0.0f) atomicAdd(d_light + i, s_light[i]);
}

inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

}  // namespace


}  // namespace aur

using namespace aur;

extern "C" {

aur_status aur_render_adjoint(aur_ctx* ctx, const aur_scene* scene, const aur_camera* camera,
                              const aur_render_params* params, const float* d_image, float* d_diffuse,
                              float* d_light_color, float* d_emission) {
    AUR_RANGE("aur_render_adjoint");
    clear_error();
    AUR_CHECK(ctx && scene && camera && d_image && d_diffuse && (d_light_color || scene->num_lights == 0),
              AUR_ERR_INVALID, "aur_render_adjoint: null argument");
    aur_status st = check_params(params);
    if (st == AUR_OK) st = check_scene_textures(scene);
    if (st != AUR_OK) return st;
    const bool mis = params->mode == AUR_MODE_PATH_MIS;
    AUR_CHECK(!mis || scene->num_lights < 32767, AUR_ERR_INVALID,
              "aur_render_adjoint: AUR_MODE_PATH_MIS takes at most 32766 lights (scene has %u)", scene->num_lights);
    AUR_CUDA(cudaSetDevice(ctx->device));
    if (mis) {
        st = build_mis_table(ctx, scene);
        if (st != AUR_OK) return st;
    }
    const aur_render_params p = *params;
    const uint32_t s0 = p.sample_begin, s1 = p.sample_end ? p.sample_end : p.spp;
    if (s1 == s0) return AUR_OK;
    const uint64_t P = (uint64_t)p.width * p.height;
    const uint32_t batch = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(s1 - s0, (1ull << 24) / P));
    const SceneView sv = scene_view(scene);
    const float4* di = (const float4*)d_image;
    for (uint32_t s = s0; s < s1; s += batch) {
        const uint32_t nb = std::min(batch, s1 - s);
        const uint32_t grid = cdiv(P * nb, kAdjThreads);
        auto go = [&](auto spec, auto m, auto tiny, auto few) {
            k_adj_replay<spec.value, m.value, tiny.value, few.value><<<grid, kAdjThreads, 0, ctx->stream>>>(
                sv, *camera, p, s, nb, di, d_diffuse, d_light_color, d_emission, scene->num_shaders, ctx->d_flags);
        };
        launch_variant(scene, mis, [&](auto spec, auto m, auto tiny) {
            if (scene->num_shaders <= kFewShaders) go(spec, m, tiny, std::true_type{});
            else go(spec, m, tiny, std::false_type{});
        });
    }
    AUR_CUDA(cudaGetLastError());
    return AUR_OK;
}

}  // extern "C"
