// trace.cu -- grid traversal (uniform and two-level 3D-DDA), Moller-Trumbore
// intersection and the primary / ambient-occlusion / path-tracing integrators.
//
// Reference path (javorkk/happyray):
//   uniform DDA            src/RT/Algorithm/UGridTraverser.h:44-177
//   two-level DDA          src/RT/Algorithm/TLGridTraverser.h:45-354
//   intersector            src/RT/Algorithm/RayTriangleIntersector.h:38-92
//   trace kernel           src/RT/Algorithm/RayTracingKernels.h:47-152
//   camera                 src/RT/Primitive/Camera.h:35-72
//   primary shading        src/RT/Integrator/SimpleIntegrator.h:41-126
//   ambient occlusion      src/RT/Integrator/AOIntegrator.h:64-191, 234-351; RayGenerators.h:286-342
//   path tracing           src/RT/Integrator/PathTracer.h:41-372
//
// Differences in arithmetic (all deterministic, bit-identical to the oracle):
//   * rays keep the direction and its IEEE reciprocal; the intersector and the entry
//     points use the direction itself instead of re-deriving it with __fdividef;
//   * primary ray directions are normalised, so t is a distance;
//   * no fast-math: IEEE division / square root, no FMA contraction.
//
// The traversal itself (warp-synchronous DDA + intersection) lives in traverse.cuh.
#include "traverse.cuh"

#include <type_traits>

#ifndef HR_AO_REFILL_MIN
#define HR_AO_REFILL_MIN 12   // idle lanes that make k_ao_samples refill
#endif
#ifndef HR_AO_LEAF_STEPS
#define HR_AO_LEAF_STEPS 6   // AO camera and sample rays: empty leaves stepped over per warp step
#endif
// Idle lanes that make a warp of a ray query, or of a shadow-ray query, refill: 1M random
// closest-hit rays in a 500k-triangle scene at 8 / 20 / 28 / 32 lanes 0.428 / 0.423 / 0.436 /
// 0.495 ms, shadow rays from its surfaces at 8 / 12 / 16 / 20 1.348 / 1.358 / 1.376 / 1.393;
// cheap rays (300k in a heightfield of 100k, most of them misses) 0.258 / 0.253 / 0.248 /
// 0.254, and 0.247 unrefilled with one ray per thread.
constexpr uint32_t kQueryRefill = 24, kShadowRefill = 12;
#ifndef HR_TRACE_MIN_BLOCKS
#define HR_TRACE_MIN_BLOCKS 8   // blocks of kTT per SM the ray kernels' register budget must allow (8: 64 registers)
#endif

namespace hr {

namespace {

// The traverser of ray and shadow-ray queries.  Their rays are long and incoherent more
// often than not, so on a two-level grid they test occupancy bits before cell records and
// step over up to six empty leaves (1M random rays 0.450 -> 0.428 ms, shadow rays 1.41 ->
// 1.36); walks over empty top cells paced as the path tracer's measured no better.
template <int KIND, bool STATS>
using QueryTrav = std::conditional_t<KIND == kUniform, TravUG<STATS>, TravTL<STATS, true, 0, 6>>;

__device__ __forceinline__ void load_ray(const float* __restrict__ org, const float* __restrict__ dir, uint32_t i, f3& o,
                                         f3& d) {
    o = mk(__ldg(org + 3 * (size_t)i), __ldg(org + 3 * (size_t)i + 1), __ldg(org + 3 * (size_t)i + 2));
    d = mk(__ldg(dir + 3 * (size_t)i), __ldg(dir + 3 * (size_t)i + 1), __ldg(dir + 3 * (size_t)i + 2));
}

template <bool STATS>
__device__ __forceinline__ void store_hit(const Scene& s, uint32_t i, f3 o, f3 d, Hit& h, int32_t* __restrict__ oid,
                                          float* __restrict__ ot, float* __restrict__ ou, float* __restrict__ ov,
                                          uint32_t* __restrict__ stats) {
    if (h.hit) refine_uv(s, h.tri, o, d, &h.u, &h.v);
    oid[i] = h.hit ? (int32_t)h.tri : -1;
    ot[i] = h.hit ? h.t : FLT_MAX;
    ou[i] = h.u;
    ov[i] = h.v;
    if (STATS) { stats[2 * (size_t)i] = h.cells; stats[2 * (size_t)i + 1] = h.tests; }
}

// the rays of a query: `width` a warp, or (POOL) from a pool
struct RayShare {
    RayPool pool;
    uint32_t width;
};
template <class T, int HM, bool STATS, bool POOL, class Gen, class Fin>
__device__ __forceinline__ void trace_query(const Scene& s, const G& g, const RayShare& w, Gen gen, Fin fin) {
    if constexpr (POOL) trace_pool<T, HM, STATS>(s, g, w.pool, gen, fin);
    else trace_shares<T, HM, STATS>(s, g, w.pool.n, w.width, gen, fin);
}

template <int KIND, bool STATS, bool POOL>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_trace_rays(Scene s, const float* __restrict__ org, const float* __restrict__ dir,
                                                    RayShare w, int32_t* __restrict__ oid, float* __restrict__ ot,
                                                    float* __restrict__ ou, float* __restrict__ ov,
                                                    uint32_t* __restrict__ stats) {
    const G g = load_g(s.desc);
    gate_scene(s);
    trace_query<QueryTrav<KIND, STATS>, kHitClosest, STATS, POOL>(
        s, g, w, [&](uint32_t i, f3& o, f3& d, Hit&) { load_ray(org, dir, i, o, d); },
        [&](uint32_t i, f3 o, f3 d, Hit& h) { store_hit<STATS>(s, i, o, d, h, oid, ot, ou, ov, stats); });
}

// Camera rays by pixel tile, `width` consecutive slots of the tile order per warp and
// step (grid stride); body(slot) traces the slot's ray with the whole warp, slots past the
// warp's width or the image are kNoSlot.
constexpr uint32_t kNoSlot = 0xffffffffu;
template <class F>
__device__ __forceinline__ void for_camera_slots(const Cam& cam, uint32_t width, F body) {
    const uint32_t lane = threadIdx.x & 31u, units = tile_slots(cam) / width;
    for (uint32_t u = blockIdx.x * (kTT / 32) + (threadIdx.x >> 5); u < units; u += gridDim.x * (kTT / 32))
        body(lane < width ? u * width + lane : kNoSlot);
}

template <int KIND, bool STATS>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_trace_primary(Scene s, Cam cam, uint32_t width, int32_t* __restrict__ oid,
                                                       float* __restrict__ ot, float* __restrict__ ou,
                                                       float* __restrict__ ov, uint32_t* __restrict__ stats) {
    const G g = load_g(s.desc);
    gate_scene(s);
    const f3 o = mk(cam.pos[0], cam.pos[1], cam.pos[2]);
    for_camera_slots(cam, width, [&](uint32_t slot) {
        uint32_t i = 0;
        const bool valid = slot != kNoSlot && tile_pixel(cam, slot, &i);
        Hit h;
        const f3 d = valid ? primary_dir(cam, i) : mk(1.0f, 0.0f, 0.0f);
        trace_one<KIND, STATS>(s, g, o, d, FLT_MAX, h, valid);
        if (valid) store_hit<STATS>(s, i, o, d, h, oid, ot, ou, ov, stats);
    });
}

// the ray-file form of render mode 0 (SimpleRayTraverser::integrate,
// SimpleRayTraverser.h:166-180): ray i traced (closest hit) and shaded by simpleShade into
// pixel i, progressive blend
template <int KIND, bool POOL>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_render_rays(Scene s, const float* __restrict__ org,
                                                                     const float* __restrict__ dir, RayShare w,
                                                                     int32_t image_id, float* __restrict__ fb,
                                                                     unsigned long long* counter) {
    const G g = load_g(s.desc);
    gate_scene(s);
    uint32_t nrays = 0;
    trace_query<QueryTrav<KIND, false>, kHitClosest, false, POOL>(
        s, g, w, [&](uint32_t i, f3& o, f3& d, Hit&) { load_ray(org, dir, i, o, d); },
        [&](uint32_t i, f3 o, f3 d, Hit& h) {
            float rgb[3];
            simple_shade(s, h.hit, h.tri, o, d, rgb);
            for (int k = 0; k < 3; ++k) fb[3 * (size_t)i + k] = blend(fb[3 * (size_t)i + k], rgb[k], image_id);
            nrays += 1;
        });
    add_rays<false>(counter, false, nrays);
}

template <int KIND, bool POOL>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_occluded(Scene s, const float* __restrict__ org, const float* __restrict__ dir,
                                                  const float* __restrict__ tmax, RayShare w, uint8_t* __restrict__ occ) {
    const G g = load_g(s.desc);
    gate_scene(s);
    trace_query<QueryTrav<KIND, false>, kHitAny, false, POOL>(
        s, g, w,
        [&](uint32_t i, f3& o, f3& d, Hit& h) {
            load_ray(org, dir, i, o, d);
            h.t = __ldg(tmax + i);
        },
        [&](uint32_t i, f3, f3, Hit& h) { occ[i] = h.hit ? 1 : 0; });
}

// mode 0: primary rays with barycentric false colour (SimpleIntegrator.h:41-126)
template <int KIND, bool STATS>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_render_primary(Scene s, Cam cam, uint32_t width, int32_t image_id, uint64_t seed,
                                                        float* __restrict__ fb, unsigned long long* counter) {
    const G g = load_g(s.desc);
    gate_scene(s);
    const f3 o = mk(cam.pos[0], cam.pos[1], cam.pos[2]);
    for_camera_slots(cam, width, [&](uint32_t slot) {
        uint32_t i = 0;
        const bool valid = slot != kNoSlot && tile_pixel(cam, slot, &i);
        const f3 d = valid ? primary_sample_dir(cam, i, image_id, seed) : mk(1.0f, 0.0f, 0.0f);
        Hit h;
        trace_one<KIND, STATS>(s, g, o, d, FLT_MAX, h, valid);
        if (valid) {
            float rgb[3];
            simple_shade(s, h.hit, h.tri, o, d, rgb);
            fb[3 * (size_t)i] = blend(fb[3 * (size_t)i], rgb[0], image_id);
            fb[3 * (size_t)i + 1] = blend(fb[3 * (size_t)i + 1], rgb[1], image_id);
            fb[3 * (size_t)i + 2] = blend(fb[3 * (size_t)i + 2], rgb[2], image_id);
        }
        add_rays<STATS>(counter, false, valid ? 1u : 0u, h.cells, h.tests);
    });
}

// mode 3, ambient occlusion (AOIntegrator.h:234-351: primary trace, AO rays, shading), as
// a wavefront of three kernels:
//   k_ao_primary  camera rays in pixel tiles; misses are shaded at once, hit pixels are
//                 appended (warp-aggregated) to a queue with their t and triangle;
//   k_ao_samples  one ray per (hit pixel, sample): AO ray generation as
//                 RayGenerators.h:286-342 with the configured radius and PCG32 stream of
//                 the pixel (sample k uses draws 2k and 2k+1), any-hit traversal, and the
//                 unoccluded count of the pixel (match_any-aggregated atomics);
//   k_ao_finish   visibility = unoccluded / samples, progressive blend (AOIntegrator.h:168-175).
template <int KIND, bool STATS>
using AoTrav = std::conditional_t<KIND == kUniform, TravUG<STATS>, TravTL<STATS, false, 0, HR_AO_LEAF_STEPS>>;

// AO camera rays, with lanes refilled inside the traversal loop: once
// all `width` lanes a warp uses are done (their pixels shaded or queued), they take that
// many consecutive pixel slots of the tile order from the pool.
template <int KIND, bool STATS>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_ao_primary(Scene s, Cam cam, int32_t image_id,
                                                              float* __restrict__ fb, float* __restrict__ hit_t,
                                                              uint32_t* __restrict__ hit_tri, uint32_t* __restrict__ unocc,
                                                              uint32_t* __restrict__ queue, uint32_t* qcount,
                                                              unsigned long long* counter, uint32_t* work, uint32_t width) {
    const G g = load_g(s.desc);
    gate_scene(s);
    const uint32_t slots = tile_slots(cam);
    const f3 o = mk(cam.pos[0], cam.pos[1], cam.pos[2]);
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    AoTrav<KIND, STATS> q;
    q.st = 0;
    Hit h;
    h.t = FLT_MAX; h.u = 0.0f; h.v = 0.0f; h.tri = 0; h.hit = false; h.cells = 0; h.tests = 0;
    f3 d = mk(1.0f, 0.0f, 0.0f);
    uint32_t pix = 0, nrays = 0, ncells = 0, ntests = 0;
    bool has = false, valid = false, dry = false;
    while (true) {
        const uint32_t need = __ballot_sync(kFullMask, !has && lane < width);
        if (!dry && ((uint32_t)__popc(need) == width || (need && !__any_sync(kFullMask, q.st != 0)))) {   // warp-uniform
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(work, (uint32_t)__popc(need));
            base = __shfl_sync(kFullMask, base, leader);
            if (base + (uint32_t)__popc(need) >= slots) dry = true;
            const uint32_t slot = base + __popc(need & lt);
            if (((need >> lane) & 1u) && slot < slots) {
                has = true;
                valid = tile_pixel(cam, slot, &pix);
                h.t = FLT_MAX; h.u = 0.0f; h.v = 0.0f; h.tri = 0; h.hit = false; h.cells = 0; h.tests = 0;
                if (valid) {
                    d = primary_dir(cam, pix);
                    if (s.ntri != 0u) q.start(s, g, o, d, h);
                }
            }
        }
        if (!__any_sync(kFullMask, has)) break;   // the pool is dry and no ray is in flight
        const uint2 r = q.range(s, h);
        const bool done = test_lists<kHitClosest, STATS>(s, o, d, r.x, r.y, false, h);
        q.next(s, g, o, d, h, done);
        const bool fin = has && q.st == 0;
        const bool hit = fin && valid && h.hit;
        if (hit) {
            hit_t[pix] = h.t;
            hit_tri[pix] = h.tri;
            unocc[pix] = 0u;
        } else if (fin && valid) {
            const float val = blend(fb[3 * (size_t)pix], 1.0f, image_id);
            fb[3 * (size_t)pix] = val;
            fb[3 * (size_t)pix + 1] = val;
            fb[3 * (size_t)pix + 2] = val;
        }
        const uint32_t m = __ballot_sync(kFullMask, hit);
        if (m) {
            const int leader = __ffs(m) - 1;
            uint32_t qb = 0;
            if ((int)lane == leader) qb = atomicAdd(qcount, (uint32_t)__popc(m));
            qb = __shfl_sync(kFullMask, qb, leader);
            if (hit) queue[qb + __popc(m & lt)] = pix;
        }
        if (fin) {
            if (valid) {
                nrays += 1;
                ncells += h.cells;
                ntests += h.tests;
            }
            has = false;
        }
    }
    add_rays<STATS>(counter, false, nrays, ncells, ntests);
}

// AO samples, with lanes refilled inside the traversal loop: a lane
// whose ray is done (occluded, or out of the grid or past the radius) retires it and
// waits; once HR_AO_REFILL_MIN lanes wait (or no ray is left in flight) they take the next
// (hit pixel, sample) items from the pool together, so a warp keeps most of its lanes
// busy until the pool runs dry instead of waiting for its longest ray, and the divergent
// ray set-up runs for many lanes at once.  A launch traces samples k0 .. k0 + spp - 1 of every
// hit pixel: items are counted in 32 bits, so the host cuts the samples of a large image into
// launches of at most kAoItems items (what the warps take past the end then fits too).
constexpr uint32_t kAoItems = 1u << 31;
template <int KIND, bool STATS>
__global__ __launch_bounds__(kTT, HR_TRACE_MIN_BLOCKS) void k_ao_samples(Scene s, Cam cam, uint32_t k0, uint32_t spp, float alpha_frac,
                                                              float alpha_abs, uint64_t seed, int32_t image_id,
                                                              const float* __restrict__ hit_t,
                                                              const uint32_t* __restrict__ hit_tri,
                                                              const uint32_t* __restrict__ queue, const uint32_t* qcount,
                                                              uint32_t* __restrict__ unocc, unsigned long long* counter,
                                                              uint32_t* work) {
    const G g = load_g(s.desc);
    gate_scene(s);
    float alpha = alpha_abs;
    if (!(alpha > 0.0f)) {
        const f3 dd = mk(g.bmax[0] - g.bmin[0], g.bmax[1] - g.bmin[1], g.bmax[2] - g.bmin[2]);
        alpha = alpha_frac * sqrtf(dot(dd, dd));
    }
    const float off = 0.01f * alpha;
    const f3 cpos = mk(cam.pos[0], cam.pos[1], cam.pos[2]);
    const uint32_t nitems = *qcount * spp;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    // rays a warp holds at a time (as ray_width): fewer where the items would not fill the warps,
    // at least 8
    uint32_t width = 32u;
    while (width > 8u && nitems < gridDim.x * (kTT / 32u) * width) width /= 2u;
    AoTrav<KIND, STATS> q;
    q.st = 0;
    Hit h;
    h.t = alpha; h.u = 0.0f; h.v = 0.0f; h.tri = 0; h.hit = false; h.cells = 0; h.tests = 0;
    f3 o = mk(0.0f, 0.0f, 0.0f), w = mk(1.0f, 0.0f, 0.0f);
    uint32_t pix = 0xffffffffu, nrays = 0, ncells = 0, ntests = 0;
    bool has = false, dry = s.ntri == 0u;
    while (true) {
        const uint32_t need = __ballot_sync(kFullMask, !has && lane < width);
        if (need && !dry && (__popc(need) >= HR_AO_REFILL_MIN ||
                             !__any_sync(kFullMask, q.st != 0))) {   // warp-uniform
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(work, (uint32_t)__popc(need));
            base = __shfl_sync(kFullMask, base, leader);
            if (base + (uint32_t)__popc(need) >= nitems) dry = true;
            const uint32_t item = base + __popc(need & lt);
            if (((need >> lane) & 1u) && item < nitems) {
                has = true;
                const uint32_t qi = item / spp, k = k0 + item % spp;
                pix = queue[qi];
                const f3 d = primary_dir(cam, pix);
                const float t = hit_t[pix];
                const f3 p = mk(cpos.x + t * d.x, cpos.y + t * d.y, cpos.z + t * d.z);
                const f3 nrm = face_normal(s, hit_tri[pix], d);
                Pcg32 rng;
                pcg_seed(rng, ((uint64_t)(uint32_t)image_id << 32) | pix, seed);
                pcg_skip_pairs(rng, k);
                const float u1 = pcg_float(rng), u2 = pcg_float(rng);
                w = cosine_dir(nrm, u1, u2);
                o = mk(p.x + off * w.x, p.y + off * w.y, p.z + off * w.z);
                h.t = alpha; h.hit = false; h.cells = 0; h.tests = 0;
                q.start(s, g, o, w, h);
            }
        }
        if (!__any_sync(kFullMask, has)) break;   // the pool is dry and no ray is in flight
        const uint2 r = q.range(s, h);
        const bool done = test_lists<kHitAny, STATS>(s, o, w, r.x, r.y, true, h);
        q.next(s, g, o, w, h, done);
        const bool fin = has && q.st == 0;
        const uint32_t peers = __match_any_sync(kFullMask, fin ? pix : 0xffffffffu);
        const uint32_t nfree = __popc(__ballot_sync(kFullMask, fin && !h.hit) & peers);
        if (fin && nfree && (int)lane == __ffs(peers) - 1) atomicAdd(unocc + pix, nfree);
        if (fin) {
            nrays += 1;
            ncells += h.cells;
            ntests += h.tests;
            has = false;
        }
    }
    add_rays<STATS>(counter, true, nrays, ncells, ntests);
}

__global__ void k_ao_finish(const uint32_t* __restrict__ queue, const uint32_t* qcount, const uint32_t* __restrict__ unocc,
                            int32_t spp, int32_t image_id, float* __restrict__ fb) {
    const uint32_t n = *qcount;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const uint32_t pix = queue[q];
        const float vis = (float)unocc[pix] / (float)spp;
        const float val = blend(fb[3 * (size_t)pix], vis, image_id);
        fb[3 * (size_t)pix] = val;
        fb[3 * (size_t)pix + 1] = val;
        fb[3 * (size_t)pix + 2] = val;
    }
}

#ifndef HR_PT_SMEM_STATE
#define HR_PT_SMEM_STATE 1   // path state in shared memory (registers left to the traversal)
#endif
#ifndef HR_PT_MIN_BLOCKS
#define HR_PT_MIN_BLOCKS 7   // blocks of kTT per SM the path tracer's register budget must allow (7: 72 registers)
#endif

// mode 1/2: path tracing with next-event estimation (PathTracer.h:41-372 structure), one
// path per pixel.  Persistent: each warp takes 32-pixel tiles from *work, and a lane whose
// path ends takes the next pixel at once (path_refill / path_step / path_retire), so lanes
// do not idle through the bounces of their warp's longest path.
template <int KIND, bool STATS>
__global__ __launch_bounds__(kTT, HR_PT_MIN_BLOCKS) void k_render_pt(Scene s, Cam cam, const LightSet* __restrict__ ls, int32_t bounces,
                                                                  float albedo, float eps_frac, uint64_t seed,
                                                                  int32_t image_id, float* __restrict__ fb,
                                                                  unsigned long long* counter, uint32_t* work, uint32_t width) {
    const G g = load_g(s.desc);
    gate_scene(s);
    const PtConsts k = pt_consts(g, ls, bounces, albedo, eps_frac);
    const uint32_t nunits = tile_slots(cam) / width;   // a warp takes `width` pixel slots at a time
    const uint32_t lane = threadIdx.x & 31u;
#if HR_PT_SMEM_STATE
    // the path state lives in shared memory, so the traversal has the registers to itself
    __shared__ __align__(16) unsigned char s_lanes[sizeof(PathLane) * kTT];
    PathLane& ln = reinterpret_cast<PathLane*>(s_lanes)[threadIdx.x];
    ln.pix = 0;
    ln.sample = 0;
    ln.val = 0.0f;
    ln.has = false;
#else
    PathLane ln;
#endif
    PtCounts n;
    uint32_t slot0 = 0, next = width;
    bool more = true;
    while (true) {
        while (more) {
            if (next >= width) {
                uint32_t t = 0;
                if (lane == 0) t = atomicAdd(work, 1u);
                t = __shfl_sync(kFullMask, t, 0);
                if (t >= nunits) {
                    more = false;
                    break;
                }
                slot0 = t * width;
                next = 0;
            }
            if (path_refill(ln, cam, slot0, &next, width, image_id, seed, fb) == 0u) break;
        }
        if (!__any_sync(kFullMask, ln.has)) break;
        const bool cont = path_step<KIND, STATS>(s, g, k, ln.p, ln.has, n);
        path_retire(ln, cont, cam, image_id, 1, seed, fb);
    }
    add_rays<STATS>(counter, false, n.rays, n.cells, n.tests);
    add_rays<STATS>(counter, true, n.srays, n.scells, n.stests);
}

Scene make_scene(hr_ctx* c) {
    Scene s;
    s.tris = c->tris.as<float4>();
    s.cells = c->g.cells.as<uint2>();
    s.leaves = c->g.leaves.as<uint2>();
    s.prims = c->g.prims.as<uint32_t>();
    s.desc = c->g.desc.as<GridDesc>();
    s.ntri = c->ntri;
    s.kind = c->built_kind;
    // shading normals and materials given for the current mesh
    s.nrm3 = c->nrm_ntri && c->nrm_ntri == c->ntri ? c->tri_nrm.as<float4>() : nullptr;
    s.alb = c->alb_ntri && c->alb_ntri == c->ntri ? c->tri_alb.as<float>() : nullptr;
    s.occ = c->built_kind == kTwoLevel ? c->g.occ.as<uint32_t>() : nullptr;
    s.occ_bit0 = 0;
    return s;
}

Cam make_cam(const hr_ctx* c) {
    Cam k;
    for (int i = 0; i < 3; ++i) {
        k.pos[i] = c->cam.pos[i]; k.tl[i] = c->cam.top_left[i];
        k.sx[i] = c->cam.step_x[i]; k.sy[i] = c->cam.step_y[i];
    }
    k.w = c->cam.w; k.h = c->cam.h;
    return k;
}

// Rays a warp holds at a time when n rays are shared out to `warps` resident warps: 32, or
// a smaller power of two (at least `least`) while n rays would not fill them `waves` times.
// A warp step costs the longest of its lanes' walks, and a small launch is as long as its
// slowest warp: with fewer rays per warp the walks are shorter, a ray's list is still
// tested by all 32 lanes, and the GPU's other warps take the rest; the launch as a whole
// does more work.
uint32_t ray_width(uint64_t n, uint64_t warps, uint32_t waves, uint32_t least) {
    uint32_t w = 32u;
    while (w > least && n < warps * w * waves) w /= 2u;
    return w;
}

// Camera rays.  Coherent rays share their walk, so a narrower warp saves less of a step than
// it gives up, and next to other work on the GPU the work counts, not the launch's tail.
// Two-level grids: 32 rays unless the image does not fill a quarter of the warps, at least 8
// (a frame, passes overlapping / alone, at 32 / 16 / 8 / 4 rays: 128 x 128 113 / 86 / 87 / 92 us
// and 194 / 198 / 167 / 141, 313 x 308 160 / 165 / 183 / 209 and 294 / 275 / 263 / 276).
// Uniform grids, whose crowded cells make tiles of very uneven cost: warps filled four
// times over, at least 4 rays (256 x 256 97 us at 32, 87 at 4; 801 x 601 with lists of
// thousands 883 at 32, 679 at 16; kernels alone 0.067 -> 0.051 and 2.56 -> 1.45 ms).  AO
// camera rays on two-level grids: four times over, at least 16 (641 x 479, where 32-ray
// tiles are just over two per warp: 0.212 -> 0.155 ms).
uint32_t camera_width(const hr_ctx* c, bool ao) {
    const uint64_t slots = (((uint64_t)c->cam.w + 7u) / 8u) * (((uint64_t)c->cam.h + 3u) / 4u) * 32u;
    const uint64_t warps = (uint64_t)c->num_sms * HR_TRACE_MIN_BLOCKS * (kTT / 32);
    if (c->built_kind == kUniform) return ray_width(slots, warps, 4, 4);
    return ao ? ray_width(slots, warps, 4, 16) : ray_width(slots, warps / 4u, 1, 8);
}

// Whether a launch on the context's stream may run beside another one of this context: a
// launch that is being captured (its graph may be replayed on any stream) or one on the
// per-thread stream.
bool may_overlap(const hr_ctx* c) {
    if (c->stream == cudaStreamPerThread) return true;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess) cudaGetLastError();
    return st != cudaStreamCaptureStatusNone;
}

// How a query over n rays is shared out, and its block count (the launch bounds allow
// HR_TRACE_MIN_BLOCKS blocks per SM at once).  A query that fits takes the fewest rays per warp
// that still have all of them in flight at once; a larger one refills from the pool, whose
// words are the context's, unless the launch may overlap another one.
//
// A launch is as long as its slowest warp, and a warp with few rays is through sooner: its
// lists are tested by all 32 lanes, its walks by the few.  So long lists cost no more work in
// narrow warps, empty cells do.  Shadow rays from the surfaces of 6,366 clustered triangles,
// 7,366 of them, at 1 / 2 / 4 / 8 / 32 a warp: 128 / 148 / 230 / 319 / 830 us.  Where cells
// are mostly empty the time alone is shorter too, but beside other queries the work counts:
// random rays in a 100k heightfield (first line) and rays from above into a uniform grid of
// it, us a query alone / among three streams' / among eight's:
//   rays     one ray per lane     this rule            32 a warp
//   1024     121 / 40.1 / 15.6    76 / 26.6 / 10.8     118 / 40.6 / 15.6
//            46 / 15.7 / 6.3      22 / 7.9 / 3.6       47 / 16.2 / 6.5
//   8192     151 / 51.5 / 21.5    94 / 34.1 / 16.3     146 / 50.3 / 20.4
//            52 / 18.1 / 7.9      33 / 13.4 / 12.3     54 / 18.8 / 8.0
//   20,000   129 / 45.6 / 21.3    92 / 34.8 / 22.7     111 / 40.0 / 18.7
//            57 / 20.2 / 9.3      41 / 15.8 / 12.6     52 / 18.4 / 8.2
//   65,536   145 / 59.2 / 46.1    114 / 52.9 / 51.8    125 / 49.3 / 38.4
//            61 / 24.9 / 22.0     49 / 28.0 / 27.5     55 / 23.1 / 20.0
// Half of the warps for widths up to 4 and a third for 8 and 16 would lose nothing among eight
// (8192: 36 / 12.9 / 6.0 in the second line), but took 1.5 times as long for the shadow rays
// above, 652 us against 471 for 48,774 rays into crowded uniform cells, and rebuilds of 2M
// triangles with 7,349 rays 404 us a pass against 382.
RayShare ray_share(const hr_ctx* c, uint32_t n, uint32_t refill, bool* pool, int* blocks) {
    const uint64_t wpb = kTT / 32, warps = (uint64_t)c->num_sms * HR_TRACE_MIN_BLOCKS * wpb;
    RayShare w = {{n, refill, c->counters.as<unsigned long long>() + 9}, 32u};
    while (w.width > 1u && n <= warps * (w.width / 2u)) w.width /= 2u;
    const uint64_t want = ((uint64_t)n + w.width - 1) / w.width;   // warps
    *pool = want > warps && !may_overlap(c);
    *blocks = (int)((std::min(want, *pool ? warps : 2 * warps) + wpb - 1) / wpb);
    return w;
}

int grid_for(const hr_ctx* c, uint32_t n) {
    uint32_t b = (n + kTT - 1) / kTT;
    uint32_t cap = (uint32_t)c->num_sms * 16u;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

uint32_t slots_for(const hr_ctx* c) {
    return (((uint32_t)c->cam.w + 7u) / 8u) * (((uint32_t)c->cam.h + 3u) / 4u) * 32u;
}

template <int V> using IntC = std::integral_constant<int, V>;
template <bool V> using BoolC = std::integral_constant<bool, V>;

// f(IntC<kind>, BoolC<stats>): picks the kernel instance of the built grid's kind
template <class F>
void by_kind(int32_t kind, bool stats, F&& f) {
    if (kind == kUniform) {
        if (stats) f(IntC<kUniform>{}, BoolC<true>{});
        else f(IntC<kUniform>{}, BoolC<false>{});
    } else {
        if (stats) f(IntC<kTwoLevel>{}, BoolC<true>{});
        else f(IntC<kTwoLevel>{}, BoolC<false>{});
    }
}

}  // namespace

int launch_trace_rays(hr_ctx* c, const float* org, const float* dir, uint32_t n, int32_t* id, float* t, float* u,
                      float* v, uint32_t* stats) {
    if (n == 0) return 0;
    Scene s = make_scene(c);
    bool pool;
    int nb;
    const RayShare w = ray_share(c, n, kQueryRefill, &pool, &nb);
    c->launches += 1;
    by_kind(s.kind, stats != nullptr, [&](auto K, auto S) {
        if (pool) k_trace_rays<K(), S(), true><<<nb, kTT, 0, c->stream>>>(s, org, dir, w, id, t, u, v, stats);
        else k_trace_rays<K(), S(), false><<<nb, kTT, 0, c->stream>>>(s, org, dir, w, id, t, u, v, stats);
    });
    return cuda_check(c, cudaGetLastError(), "trace_rays launch");
}

int launch_trace_primary(hr_ctx* c, int32_t* id, float* t, float* u, float* v, uint32_t* stats) {
    Scene s = make_scene(c);
    Cam k = make_cam(c);
    const uint32_t n = (uint32_t)k.w * (uint32_t)k.h;
    if (n == 0) return 0;
    c->launches += 1;
    const uint32_t width = camera_width(c, false);
    by_kind(s.kind, stats != nullptr, [&](auto K, auto S) {
        k_trace_primary<K(), S()><<<grid_for(c, slots_for(c) / width * 32u), kTT, 0, c->stream>>>(s, k, width, id, t, u, v,
                                                                                                 stats);
    });
    return cuda_check(c, cudaGetLastError(), "trace_primary launch");
}

int launch_render_rays(hr_ctx* c, const float* org, const float* dir, uint32_t n, int32_t image_id, float* fb) {
    if (n == 0) return 0;
    bool pool;
    int nb;
    const RayShare w = ray_share(c, n, kQueryRefill, &pool, &nb);
    c->launches += 1;
    const Scene s = make_scene(c);
    unsigned long long* ctr = c->counters.as<unsigned long long>();
    by_kind(s.kind, false, [&](auto K, auto) {
        if (pool) k_render_rays<K(), true><<<nb, kTT, 0, c->stream>>>(s, org, dir, w, image_id, fb, ctr);
        else k_render_rays<K(), false><<<nb, kTT, 0, c->stream>>>(s, org, dir, w, image_id, fb, ctr);
    });
    return cuda_check(c, cudaGetLastError(), "render_rays launch");
}

int launch_occluded(hr_ctx* c, const float* org, const float* dir, const float* tmax, uint32_t n, uint8_t* occ) {
    if (n == 0) return 0;
    bool pool;
    int nb;
    const RayShare w = ray_share(c, n, kShadowRefill, &pool, &nb);
    c->launches += 1;
    const Scene s = make_scene(c);
    by_kind(s.kind, false, [&](auto K, auto) {
        if (pool) k_occluded<K(), true><<<nb, kTT, 0, c->stream>>>(s, org, dir, tmax, w, occ);
        else k_occluded<K(), false><<<nb, kTT, 0, c->stream>>>(s, org, dir, tmax, w, occ);
    });
    return cuda_check(c, cudaGetLastError(), "occluded launch");
}

int launch_render(hr_ctx* c, int32_t mode, int32_t image_id, float* d_fb) {
    Scene s = make_scene(c);
    Cam k = make_cam(c);
    const uint32_t n = (uint32_t)k.w * (uint32_t)k.h;
    if (n == 0) return 0;
    unsigned long long* ctr = c->counters.as<unsigned long long>();
    const bool st = c->collect_stats;
    cudaStream_t strm = c->stream;
    auto mark = [&](int i) { if (c->timing && i < 8) cudaEventRecord(c->rev[i], strm); };
    c->nrender_ev = 0;
    switch (mode) {
    case 0: {
        const uint32_t width = camera_width(c, false);
        const int gw = grid_for(c, slots_for(c) / width * 32u);
        c->launches += 1;
        mark(0);
        by_kind(s.kind, st, [&](auto K, auto S) { k_render_primary<K(), S()><<<gw, kTT, 0, strm>>>(s, k, width, image_id, c->ip.seed, d_fb, ctr); });
        mark(1);
        c->nrender_ev = 2;
        break;
    }
    case 1:
    case 2: {
        const LightSet* l = c->lights_dev.as<LightSet>();
        uint32_t* work = reinterpret_cast<uint32_t*>(ctr + 7);
        int rc;
        if ((rc = cuda_check(c, cudaMemsetAsync(work, 0, sizeof(uint32_t), strm), "tile counter reset"))) return rc;
        c->launches += 1;
        mark(0);
        by_kind(s.kind, st, [&](auto K, auto S) {
            int nb = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_render_pt<K(), S()>, kTT, 0) != cudaSuccess || nb < 1) {
                cudaGetLastError();
                nb = 1;
            }
            // 320 x 200 at 32 / 16 / 8 / 4 paths per warp: 718 / 596 / 532 / 539 us a four-image pass
            const uint32_t width = ray_width(slots_for(c), (uint64_t)nb * c->num_sms * (kTT / 32), 1, 8);
            const uint32_t need = (slots_for(c) / width + kTT / 32 - 1) / (kTT / 32);   // blocks
            const int gp = (int)std::min(need, (uint32_t)(nb * c->num_sms));
            k_render_pt<K(), S()><<<gp, kTT, 0, strm>>>(s, k, l, c->ip.pt_bounces, c->ip.albedo, c->ip.ray_eps_frac,
                                                        c->ip.seed, image_id, d_fb, ctr, work, width);
        });
        mark(1);
        c->nrender_ev = 2;
        break;
    }
    case 3: {
        int rc;
        if ((rc = ensure(c, c->hit_t, sizeof(float) * n)) || (rc = ensure(c, c->hit_tri, sizeof(uint32_t) * n)) ||
            (rc = ensure(c, c->unocc, sizeof(uint32_t) * n)) || (rc = ensure(c, c->queue, sizeof(uint32_t) * n)))
            return rc;
        // word 7: the hit-pixel queue length and the sample pool; word 8: the camera-ray pool
        uint32_t* qcount = reinterpret_cast<uint32_t*>(ctr + 7);
        if ((rc = cuda_check(c, cudaMemsetAsync(qcount, 0, 4 * sizeof(uint32_t), strm), "queue reset"))) return rc;
        const uint32_t spp = (uint32_t)c->ip.ao_samples, part = std::max(1u, std::min(spp, kAoItems / n));
        c->launches += 2;
        mark(0);
        // blocks of both kernels: all resident at once (the launch bounds allow HR_TRACE_MIN_BLOCKS per SM)
        const int nb = HR_TRACE_MIN_BLOCKS * c->num_sms;
        const uint32_t width = camera_width(c, true);
        by_kind(s.kind, st, [&](auto K, auto S) {
            k_ao_primary<K(), S()><<<std::min(grid_for(c, slots_for(c) / width * 32u), nb), kTT, 0, strm>>>(
                s, k, image_id, d_fb, c->hit_t.as<float>(), c->hit_tri.as<uint32_t>(), c->unocc.as<uint32_t>(),
                c->queue.as<uint32_t>(), qcount, ctr, qcount + 2, width);
        });
        mark(1);
        for (uint32_t k0 = 0; k0 == 0 || k0 < spp; k0 += part) {
            if (k0 && (rc = cuda_check(c, cudaMemsetAsync(qcount + 1, 0, sizeof(uint32_t), strm), "sample pool reset"))) return rc;
            c->launches += 1;
            by_kind(s.kind, st, [&](auto K, auto S) {
                k_ao_samples<K(), S()><<<nb, kTT, 0, strm>>>(
                    s, k, k0, std::min(part, spp - k0), c->ip.ao_radius_frac, c->ip.ao_radius_abs, c->ip.seed, image_id,
                    c->hit_t.as<float>(), c->hit_tri.as<uint32_t>(), c->queue.as<uint32_t>(), qcount, c->unocc.as<uint32_t>(),
                    ctr, qcount + 1);
            });
        }
        mark(2);
        k_ao_finish<<<c->num_sms * 4, 256, 0, strm>>>(c->queue.as<uint32_t>(), qcount, c->unocc.as<uint32_t>(), (int32_t)spp,
                                                      image_id, d_fb);
        mark(3);
        c->nrender_ev = 4;
        break;
    }
    default:
        return set_error(c, 1, "render: unknown mode %d", mode);
    }
    return cuda_check(c, cudaGetLastError(), "render launch");
}

}  // namespace hr
