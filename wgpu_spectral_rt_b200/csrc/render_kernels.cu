// render_kernels.cu — per-frame kernels of the spectral path tracer.
//
// One frame = one sample per pixel (src/renderer/mod.rs:168-207):
//   photon pass   photon_emit.wgsl:154-331 as a wavefront (emit and
//                 cull, per bounce trace + shade, emitter-ordered compaction
//                 of the stored photons) and the grid (build_grid.wgsl:25-73)
//                 as cell keys + radix sort + ranges
//   camera paths  shader.wgsl:708-823 as a wavefront: raygen, then per
//                 bounce trace_closest -> shade -> trace_shadow over SoA
//                 queues compacted with warp ballots; finalize converts the
//                 hero tuple to sRGB, accumulates and tonemaps.
#include <algorithm>

#include "radix_sort.cuh"
#include "render_kernels.h"

// Resident blocks of TRACE_BLOCK threads per SM the shading kernels are
// compiled for.  8 caps them at 64 registers (the unbounded build takes 87,
// 108 with guiding, and runs 20 warps per SM): the spills stay in L1 and the
// doubled warp count hides the photon-gather latency better (measured shading
// per frame: config 2 1.98 -> 1.79 ms, the guiding scene 2.94 -> 2.58 ms).
#ifndef SRT_SHADE_MIN_BLOCKS
#define SRT_SHADE_MIN_BLOCKS 8
#endif

namespace srt {

namespace {

constexpr uint32_t FLAG_DIFFUSE = 0x1u;  // has_hit_diffuse (shader.wgsl:554)
constexpr uint32_t FLAG_CAUSTIC = 0x2u;  // is_caustic_path (shader.wgsl:555)
constexpr uint32_t FLAG_LIGHT = 0x4u;    // pb.light holds the path's radiance at the first light's temperature

// A light's unit normal and area (shader.wgsl:493-497, photon_emit.wgsl:172-176).
SRT_DEV float4 light_frame(const float4* light) {
    const float3 c = cross(xyz(light[1]) - xyz(light[0]), xyz(light[2]) - xyz(light[0]));
    const float3 n = normalize(c);
    return f4(n.x, n.y, n.z, length(c) * 0.5f);
}
__global__ void k_light_frames(const float4* __restrict__ lights, uint32_t n, float4* __restrict__ frames) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) frames[i] = light_frame(lights + 4ull * i);
}

SRT_DEV uint32_t warp_push(bool pred, uint32_t* counter) {
    uint32_t mask = __ballot_sync(0xFFFFFFFFu, pred);
    int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (mask) {
        int leader = __ffs(mask) - 1;
        if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
        base = __shfl_sync(0xFFFFFFFFu, base, leader);
    }
    return base + __popc(mask & ((1u << lane) - 1u));
}

SRT_DEV GatherConst gather_const(const GatherArgs& g, uint32_t frame) {
    GatherConst k;
    k.j = grid_jitter(frame, g.cell);
    k.r = g.r0 * powf((float)(frame + 1u), g.rexp);
    k.r2 = k.r * k.r;
    k.density = (3.0f / (PI * k.r2)) * (1.0f / g.spectral_radius) * g.inv_norm_count;
    return k;
}

// gather_photons: shader.wgsl:297-342 over a sorted range: a point's bucket,
// walked from its highest photon index down (the LIFO order of the
// reference's linked list for in-order insertion), at most `cap` photons.
// gather_range is what the walk covers: [.x, .y).
SRT_DEV uint2 gather_range(const GatherArgs& g, const GatherConst& k, float3 hit_pos) {
    const uint2 rg = __ldg(&g.ranges[grid_hash(hit_pos, k.j, g.cell, g.hash_bits)]);
    return make_uint2(rg.y - min(rg.y - rg.x, g.cap), rg.y);
}

// A photon adds zeros unless it lies within the radius and one of the path's
// four wavelengths lies within spectral_radius of its own (two usually
// cannot: they are 100 nm apart), and zeros are left out of the sum.  They are
// zeros only if every energy is finite and the radius positive: a map with a
// non-finite energy (ranges' last entry) weights every photon within the radius.
SRT_DEV bool gather_all(const GatherArgs& g) {
    return !(g.spectral_radius > 0.f) || __ldg(&g.ranges[(size_t)1 << g.hash_bits]).x != 0u;
}
SRT_DEV bool gather_near(float4 pa, float3 hit_pos, float4 wl, float r2, float sr, bool all) {
    const float3 dd = hit_pos - xyz(pa);
    const float a =
        fminf(fminf(fabsf(wl.x - pa.w), fabsf(wl.y - pa.w)), fminf(fabsf(wl.z - pa.w), fabsf(wl.w - pa.w)));
    return dot(dd, dd) < r2 && (a < sr || all);
}
// What a near photon (pa: position + wavelength, pb: direction + energy) adds.
SRT_DEV float4 gather_weight(float4 pa, float4 pb, float3 hit_pos, float4 wl, float r, float sr, bool all) {
    const float3 dd = hit_pos - xyz(pa);
    const float sw = 1.0f - (sqrtf(dot(dd, dd)) / r);
    const float e = pb.w * sw;
    const float a0 = fabsf(wl.x - pa.w), a1 = fabsf(wl.y - pa.w), a2 = fabsf(wl.z - pa.w), a3 = fabsf(wl.w - pa.w);
    if ((a0 < sr) + (a1 < sr) + (a2 < sr) + (a3 < sr) == 1 && !all) {
        const float w = fmaxf(1.0f - fminf(fminf(a0, a1), fminf(a2, a3)) / sr, 0.f) * e;
        return f4(a0 < sr ? w : 0.f, a1 < sr ? w : 0.f, a2 < sr ? w : 0.f, a3 < sr ? w : 0.f);
    }
    return f4(fmaxf(1.0f - a0 / sr, 0.f), fmaxf(1.0f - a1 / sr, 0.f), fmaxf(1.0f - a2 / sr, 0.f),
              fmaxf(1.0f - a3 / sr, 0.f)) * e;
}

// One thread walks a range: which of 32 photons are near, GATHER_BATCH loads
// at a time (the loads are independent, and every lane of the warp weighs its
// near photons in one loop per 32), then their weights in order.  In the
// shading kernel a loop per batch of 4 took 1.99 ms per slab frame, a loop per 32
// 1.86 (batches of 2 / 8: 1.81 / 1.85), a plain walk 2.35.
#ifndef SRT_GATHER_BATCH
#define SRT_GATHER_BATCH 2
#endif
constexpr uint32_t GATHER_BATCH = SRT_GATHER_BATCH;
SRT_DEV float4 gather(const GatherArgs& g, const GatherConst& k, uint2 range, float3 hit_pos, float3 normal, float4 wl) {
    float4 total = splat4(0.f);
    const float sr = g.spectral_radius;
    const bool all = gather_all(g);
    for (uint32_t i = range.y; i > range.x;) {
        const uint32_t m = min(i - range.x, 32u);
        uint32_t near = 0u;
        for (uint32_t c = 0; c < m; c += GATHER_BATCH) {
            float4 p[GATHER_BATCH];
#pragma unroll
            for (uint32_t b = 0; b < GATHER_BATCH; ++b) p[b] = __ldg(&g.pos[i - 1u - min(c + b, m - 1u)]);
#pragma unroll
            for (uint32_t b = 0; b < GATHER_BATCH; ++b)
                if (gather_near(p[b], hit_pos, wl, k.r2, sr, all)) near |= 1u << (c + b);
        }
        near &= 0xFFFFFFFFu >> (32u - m);
        while (near != 0u) {
            const uint32_t at = i - (uint32_t)__ffs(near);
            near &= near - 1u;
            const float4 pb = __ldg(&g.dir[at]), pa = __ldg(&g.pos[at]);
            if (dot(normal, xyz(pb)) > 0.0f) total = total + gather_weight(pa, pb, hit_pos, wl, k.r, sr, all);
        }
        i -= m;
    }
    return total * k.density;
}

// The same walk by a group of eight lanes (called by all 32 lanes of a warp;
// the result in all lanes of the group): a lane weighs one photon, and the
// weights of eight are added in order.
SRT_DEV float4 gather_group(const GatherArgs& g, const GatherConst& k, bool active, uint2 range, float3 hit_pos,
                            float3 normal, float4 wl) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t c = threadIdx.x & 7u, shift = threadIdx.x & 24u;
    float4 total = splat4(0.f);
    const float sr = g.spectral_radius;
    const bool all = gather_all(g);
    uint32_t i = range.y;
    while (__any_sync(FULL, active && i > range.x)) {
        float4 w = splat4(0.f);
        bool near = active && i > range.x + c;
        if (near) {
            const float4 pa = __ldg(&g.pos[i - 1u - c]);
            near = gather_near(pa, hit_pos, wl, k.r2, sr, all);
            if (near) {
                const float4 pb = __ldg(&g.dir[i - 1u - c]);
                near = dot(normal, xyz(pb)) > 0.0f;
                if (near) w = gather_weight(pa, pb, hit_pos, wl, k.r, sr, all);
            }
        }
        // the lanes any group of the warp has to add (a lane without a weight adds zeros)
        uint32_t add = __ballot_sync(FULL, near);
        add |= add >> 16;
        add = (add | (add >> 8)) & 0xFFu;
        while (add != 0u) {
            const int from = (int)(shift | ((uint32_t)__ffs(add) - 1u));
            add &= add - 1u;
            total = total + f4(__shfl_sync(FULL, w.x, from), __shfl_sync(FULL, w.y, from), __shfl_sync(FULL, w.z, from),
                               __shfl_sync(FULL, w.w, from));
        }
        i = i > range.x + 8u ? i - 8u : range.x;
    }
    return total * k.density;
}

// ------------------------------------------------------------------ photon pass
// The photon pass of photon_emit.wgsl:154-331 as a wavefront: emit every
// photon path (one thread per emitter id), then per bounce: the shared
// closest-hit kernel over the live queue and a shading kernel for the
// photon's material logic.  A stored photon lands in its emitter's slot and is
// flagged; an emitter-ordered compaction afterwards reproduces the order a
// sequential run of the reference's atomicAdd gives.
//
// Emission culls first: a photon path whose first surface does not scatter
// (diffuse, emitter) ends there without storing anything, so an emitted ray
// that meets no leaf box with a scattering triangle (scatter_step: a walk of
// the scene's tree restricted to those subtrees) needs no closest hit, and
// none of its state is written.  Config 2 (4.2M emitted, 31k scatter): photon pass 2.12 -> 1.59 ms alone (closest hits of bounce 0
// 1.42 -> 0.50 ms, emission 0.09 -> 0.66 ms), frame 8.87 -> 8.35 ms; eight
// seeded scenes in a batch 17.1 -> 15.6 ms for two iterations.

// Octahedral 12+12-bit direction code, Morton-interleaved (24 bits).
SRT_DEV uint32_t dir_key(float3 d) {
    float s = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    float px = d.x / s, py = d.y / s;
    if (d.z < 0.0f) {
        float qx = (1.0f - fabsf(py)) * (px >= 0.0f ? 1.0f : -1.0f);
        float qy = (1.0f - fabsf(px)) * (py >= 0.0f ? 1.0f : -1.0f);
        px = qx;
        py = qy;
    }
    uint32_t ux = (uint32_t)fminf(fmaxf((px * 0.5f + 0.5f) * 4096.0f, 0.0f), 4095.0f);
    uint32_t uy = (uint32_t)fminf(fmaxf((py * 0.5f + 0.5f) * 4096.0f, 0.0f), 4095.0f);
    uint32_t k = 0;
#pragma unroll
    for (int b = 0; b < 12; ++b) k |= (((ux >> b) & 1u) << (2 * b)) | (((uy >> b) & 1u) << (2 * b + 1));
    return k;
}

// Sort key of a secondary camera ray: direction first (octahedral 7+7 bits,
// Morton order), then origin (6 bits per axis of the scene bounds, Morton).
SRT_DEV uint32_t ray_sort_key(float3 o, float3 d, float4 bmin, float4 binv) {
    uint32_t dk = dir_key(d) >> 10;  // top 7 bits of each octahedral coordinate
    uint32_t q[3];
    q[0] = (uint32_t)fminf(fmaxf((o.x - bmin.x) * binv.x * 64.0f, 0.0f), 63.0f);
    q[1] = (uint32_t)fminf(fmaxf((o.y - bmin.y) * binv.y * 64.0f, 0.0f), 63.0f);
    q[2] = (uint32_t)fminf(fmaxf((o.z - bmin.z) * binv.z * 64.0f, 0.0f), 63.0f);
    uint32_t ok = 0;
#pragma unroll
    for (int b = 0; b < 6; ++b)
        ok |= (((q[0] >> b) & 1u) << (3 * b)) | (((q[1] >> b) & 1u) << (3 * b + 1)) | (((q[2] >> b) & 1u) << (3 * b + 2));
    return (dk << 18) | ok;
}

constexpr uint32_t PH_CAUSTIC = 0x1u;

// Emission (photon_emit.wgsl:159-214) in persistent warps: a lane takes an
// emitter id, draws its light point and direction and walks (scatter_step);
// once SRT_EMIT_REFILL lanes are done, the rays that may scatter get their
// wavelength, energy and state and are queued for bounce 0 (any order: a
// path's results go to its emitter's slot), and the lanes take new ids.  The
// walks end after 1 to ~10 nodes; one ray per thread, a warp waited for its
// longest.  Config-2 photon pass alone 1.46 -> 1.25 ms (refill at 4 / 8 / 12 / 16 /
// 24 idle lanes: 1.36 / 1.27 / 1.25 / 1.25 / 1.30).
#ifndef SRT_EMIT_REFILL
#define SRT_EMIT_REFILL 16
#endif
constexpr int EMIT_FETCH = MAX_BOUNCES;  // the emission's id counter: fetch[TRAV_PHOTON][EMIT_FETCH]
static_assert(MAX_PHOTON_BOUNCES < EMIT_FETCH, "photon bounces use the counters below");

template <int STACK>
__global__ void __launch_bounds__(TRACE_BLOCK, SRT_SHADE_MIN_BLOCKS) k_photon_emit(FrameArgs a) {
    extern __shared__ uint2 stack_smem[];
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const DevScene& S = a.scene;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t n = a.photons_per_frame, nl = S.n_lights;  // nl > 0: the pass is skipped without lights
    const uint32_t seed = a.cam->frame_count * 927163u + a.seed;
    uint32_t* fetch = &a.counters->fetch[TRAV_PHOTON][EMIT_FETCH];
    if (blockIdx.x == 0 && threadIdx.x == 0) a.counters->photons_emitted = n;
    // what the rest of the pass starts from: no photon stored, no deposit tile
    // done, no digit counted
    rs_clear(reinterpret_cast<uint32_t*>(a.ph.flags), deposit_tiles(n) * (DEPOSIT_TILE / 4u));
    rs_clear(a.ph.deposit, deposit_words(n));
    rs_clear(a.ph.sort_scratch, RS_HEAD);
    rs_clear_status(a.ph.sort_scratch, n);
    ScatterWalk W;
    float3 dir = f3(0.f, 0.f, 0.f);
    uint32_t e = 0u, s = 0u, li = 0u;
    int state = WALK_DONE;
    bool exhausted = false;
    while (true) {
        const uint32_t idle = __ballot_sync(FULL, state != WALK_ON);
        if (idle == FULL || (!exhausted && __popc(idle) >= SRT_EMIT_REFILL)) {
            const bool live = state == WALK_MAY_SCATTER;
            if (live) {
                const float4 LP = S.lights[4 * li + 3], lf = S.light_frames[li];
                float cmin = cauchy_cdf(LAMBDA_MIN), cmax = cauchy_cdf(LAMBDA_MAX), crange = cmax - cmin;
                float lambda =
                    clampf(555.0f + 40.0f * tanf(PI * ((cmin + rng_next(s) * crange) - 0.5f)), LAMBDA_MIN, LAMBDA_MAX);
                float dw = (lambda - 555.0f) / 40.0f;
                float pdf = (1.0f / (crange * PI * 40.0f)) / (1.0f + dw * dw);
                float energy = (blackbody(lambda, LP.y) / pdf) * lf.w * PI * LP.z;
                a.ph.ray_o[e] = f4(W.o.x, W.o.y, W.o.z, 0.0001f);
                a.ph.ray_d[e] = f4(dir.x, dir.y, dir.z, 100.0f);
                a.ph.state[e] = f4(lambda, energy, __uint_as_float(s), __uint_as_float(0u));
            }
            const uint32_t slot = warp_push(live, &a.counters->photon_paths[0]);
            if (live) a.ph.queue[0][slot] = e;
            if (state != WALK_ON) state = WALK_DONE;
            if (exhausted) break;  // every lane is done
            uint32_t base = 0u;
            if (lane == 0u) base = atomicAdd(fetch, (uint32_t)__popc(idle));
            base = __shfl_sync(FULL, base, 0);
            exhausted = base + (uint32_t)__popc(idle) >= n;
            if (state != WALK_ON) {
                e = base + __popc(idle & lt);
                if (e < n) {
                    s = pcg_hash(e + seed);
                    li = min(__float2uint_rz(rng_next(s) * (float)nl), nl - 1u);
                    const float4 L0 = S.lights[4 * li], L1 = S.lights[4 * li + 1], L2 = S.lights[4 * li + 2],
                                 lf = S.light_frames[li];
                    float r1 = rng_next(s);
                    float r2 = rng_next(s);
                    float sr1 = sqrtf(r1);
                    float u = 1.0f - sr1, v = r2 * sr1, w = 1.0f - u - v;
                    float3 emit_pos = xyz(L0) * u + xyz(L1) * v + xyz(L2) * w;
                    dir = normalize(xyz(lf) + random_unit_vector(s));
                    if (scatter_init(W, S, emit_pos + dir * 0.001f, dir)) state = WALK_ON;
                }
            }
            continue;
        }
        if (state == WALK_ON)
            state = scatter_step<STACK>(S, W, 0.0001f, 100.0f, stack_smem + threadIdx.x, TRACE_BLOCK, a.err);
    }
}

// One bounce of the photon loop after its closest-hit query
// (photon_emit.wgsl:227-330).  Material type 5 (no reference counterpart)
// reflects with the probability of the film's Airy reflectance, else absorbs.
__global__ void __launch_bounds__(TRACE_BLOCK, SRT_SHADE_MIN_BLOCKS) k_photon_shade(FrameArgs a, uint32_t bounce) {
    const uint32_t n = a.counters->photon_paths[bounce];
    const DevScene& S = a.scene;
    const uint32_t* qin = a.ph.queue[bounce & 1];
    for (uint32_t base = blockIdx.x * TRACE_BLOCK; base < n; base += gridDim.x * TRACE_BLOCK) {
        const uint32_t q = base + threadIdx.x;
        bool alive = false;
        uint32_t e = q < n ? qin[q] : 0u;
        if (q < n) {
            float4 h = a.ph.hit[e];
            uint32_t prim = __float_as_uint(h.y);
            if (prim != MISS) {
                float4 o4 = a.ph.ray_o[e], d4 = a.ph.ray_d[e], st = a.ph.state[e];
                float3 pos = xyz(o4), dir = xyz(d4);
                float lambda = st.x, energy = st.y;
                uint32_t s = __float_as_uint(st.z), fl = __float_as_uint(st.w);
                Surface sf = surface_at(S, prim, h.z, h.w, dir);
                float4 extra = S.materials[2 * sf.mat + 1];
                float3 ffn = sf.front ? sf.wn : -sf.wn;
                uint32_t type = (uint32_t)extra.x;
                float3 hp = pos + dir * h.x;
                bool caustic = (fl & PH_CAUSTIC) != 0u;
                if (type == 0u) {
                    if (caustic) {
                        a.ph.staging[2 * e] = f4(hp.x, hp.y, hp.z, lambda);
                        a.ph.staging[2 * e + 1] = f4(-dir.x, -dir.y, -dir.z, energy);
                        a.ph.flags[e] = 1u;
                    }
                } else if (type == 1u) {
                    dir = reflect(normalize(dir), ffn);
                    pos = hp + ffn * 0.001f;
                    alive = true;
                } else if (type == 2u) {
                    float lum = lambda / 1000.0f;
                    float ir = extra.z + (extra.w / (lum * lum));
                    float ratio = sf.front ? 1.0f / ir : ir;
                    float3 ud = normalize(dir);
                    float ct = fminf(dot(-ud, ffn), 1.0f);
                    float stn = sqrtf(1.0f - ct * ct);
                    if (ratio * stn > 1.0f || schlick(ct, ratio) > rng_next(s)) {
                        dir = reflect(ud, ffn);
                    } else {
                        caustic = true;
                        dir = refract(ud, ffn, ratio);
                    }
                    pos = hp + (dot(dir, ffn) > 0.0f ? ffn : -ffn) * 0.001f;
                    alive = true;
                } else if (type == 4u) {
                    float3 ud = normalize(dir);
                    float ct = fminf(dot(-ud, ffn), 1.0f);
                    // select(n1 / n3, n3 / n1, is_front_face) with n1 = 1
                    float ratio = sf.front ? extra.w / 1.0f : 1.0f / extra.w;
                    float stt = ratio * ratio * (1.0f - ct * ct);
                    if (stt > 1.0f) {
                        dir = reflect(ud, ffn);
                    } else {
                        bool tir;
                        float F = thin_film1(ct, 1.0f, extra.z, extra.w, fmaxf(extra.y, 50.0f), lambda, tir);
                        dir = rng_next(s) < F ? reflect(ud, ffn) : refract(ud, ffn, ratio);
                    }
                    caustic = true;  // the position is not advanced (photon_emit.wgsl:291-326)
                    alive = true;
                } else if (type == 5u) {
                    float3 ud = normalize(dir);
                    float ct = fminf(dot(-ud, ffn), 1.0f);
                    bool tir;
                    float F = thin_film1(ct, 1.0f, extra.z, extra.w, fmaxf(extra.y, 50.0f), lambda, tir);
                    if (rng_next(s) < F) {
                        dir = reflect(ud, ffn);
                        pos = hp + ffn * 0.001f;
                        caustic = true;
                        alive = true;
                    }
                }
                if (bounce + 1u >= a.photon_max_bounces) alive = false;
                if (alive) {
                    a.ph.ray_o[e] = f4(pos.x, pos.y, pos.z, 0.0001f);
                    a.ph.ray_d[e] = f4(dir.x, dir.y, dir.z, 100.0f);
                    a.ph.state[e] = f4(lambda, energy, __uint_as_float(s), __uint_as_float(caustic ? PH_CAUSTIC : 0u));
                }
            }
        }
        uint32_t slot = warp_push(alive, &a.counters->photon_paths[bounce + 1]);
        if (alive) a.ph.queue[(bounce + 1) & 1][slot] = e;
    }
}

// The grid key of a photon (build_grid.wgsl:54-73): its cell's hash, or the
// sentinel bucket for a photon without energy.
SRT_DEV uint32_t photon_key(float4 p0, float4 p1, float3 jitter, float cell, uint32_t hash_bits) {
    return p1.w == 0.0f ? (1u << hash_bits) : grid_hash(xyz(p0), jitter, cell, hash_bits);
}
constexpr int GRID_PASSES = RS_PASSES;  // digit counts kept by the key kernels: hash_bits <= 26, at most 4 passes
SRT_DEV void clear_counts(uint32_t* h) {
    for (uint32_t i = threadIdx.x; i < GRID_PASSES * 256u; i += blockDim.x) h[i] = 0u;
    __syncthreads();
}

// Emitter-ordered compaction of the stored photons and their grid keys, in one
// launch: a tile of emitter flags per block, the photons before it by
// look-back over the tiles (a warp reads 32 of them at once), each stored photon
// copied to its place with its key, the keys' digits counted for the sort.
// Against a count, a scan by one block (32 us for 4M emitters), the copy and the
// keys, 76 us in four launches, and three memsets: with the sort's passes the
// photon pass of config 2 1.25 -> 1.14 ms, Cornell 0.82 -> 0.77 ms.
static_assert(DEPOSIT_TILE == RS_THREADS * 16, "16 flags per thread");
__global__ void __launch_bounds__(RS_THREADS) k_deposit(FrameArgs a) {
    __shared__ uint32_t counts[GRID_PASSES * 256];
    __shared__ uint32_t warp_sums[RS_WARPS], ticket, before;
    clear_counts(counts);
    uint32_t* status = a.ph.deposit + 2;
    if (threadIdx.x == 0) ticket = atomicAdd(&a.ph.deposit[0], 1u);
    __syncthreads();
    const uint32_t tile = ticket, tiles = deposit_tiles(a.photons_per_frame);
    if (tile >= tiles) {  // (one block per tile: its counter was not cleared)
        if (threadIdx.x == 0) atomicOr(a.err, ERR_BAD_INDEX);
        return;
    }
    const uint32_t first = tile * DEPOSIT_TILE + threadIdx.x * 16u;
    const uint4 f = *reinterpret_cast<const uint4*>(a.ph.flags + first);  // (flags past the last emitter are clear)
    uint32_t stored = 0u;
    const uint32_t w[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)  // bytes of 0 or 1 to bits
        stored |= ((w[i] & 1u) | ((w[i] >> 7) & 2u) | ((w[i] >> 14) & 4u) | ((w[i] >> 21) & 8u)) << (4 * i);
    const uint32_t mine = __popc(stored);
    uint32_t dst = rs_block_exclusive(mine, warp_sums);
    if (threadIdx.x == RS_THREADS - 1) {
        const uint32_t total = dst + mine;
        atomicExch(&status[tile], (tile == 0u ? RS_PREFIX : RS_SUM) | total);
        warp_sums[0] = total;
    }
    __syncthreads();
    if (threadIdx.x < 32u) {
        // 32 tiles before this one at a time, up to the nearest that knows its prefix
        uint32_t sum = 0u;
        for (uint32_t t = tile; t > 0u;) {
            const bool in = threadIdx.x < t;
            const volatile uint32_t* p = status + (in ? t - 1u - threadIdx.x : 0u);
            uint32_t s = in ? *p : RS_PREFIX;
            for (uint32_t polls = 0; __any_sync(0xFFFFFFFFu, s == 0u) && polls < RS_POLLS; ++polls)
                if (s == 0u) s = *p;
            if (s == 0u) {
                atomicOr(a.err, ERR_WAIT_TIMEOUT);
                s = RS_PREFIX;
            }
            const uint32_t done = __ballot_sync(0xFFFFFFFFu, (s & RS_PREFIX) != 0u);
            const uint32_t last = done != 0u ? (uint32_t)__ffs(done) - 1u : 31u;
            sum += __reduce_add_sync(0xFFFFFFFFu, threadIdx.x <= last ? (s & RS_COUNT) : 0u);
            if (done != 0u) break;
            t -= 32u;
        }
        if (threadIdx.x == 0u) {
            before = sum;
            const uint32_t all = sum + warp_sums[0];
            if (tile > 0u) atomicExch(&status[tile], RS_PREFIX | all);
            if (tile + 1u == tiles) {
                a.counters->photons_stored = all;
                atomicAdd(&a.stats->photons_stored, (unsigned long long)all);
            }
        }
    }
    __syncthreads();
    dst += before;
    const float3 j = grid_jitter(a.cam->frame_count, a.gather.cell);
    const int passes = rs_passes(0, (int)a.gather.hash_bits + 1);
    while (stored != 0u) {
        const uint32_t e = first + (uint32_t)__ffs(stored) - 1u;
        stored &= stored - 1u;
        const float4 p0 = a.ph.staging[2ull * e], p1 = a.ph.staging[2ull * e + 1];
        const uint32_t key = photon_key(p0, p1, j, a.gather.cell, a.gather.hash_bits);
        a.ph.photons[2ull * dst] = p0;
        a.ph.photons[2ull * dst + 1] = p1;
        a.ph.keys[dst] = key;
        a.ph.vals[dst] = dst;
        rs_count_key(counts, key, 0, passes);
        ++dst;
    }
    __syncthreads();
    rs_flush_counts(counts, a.ph.sort_scratch, passes);
}

// Keys of a photon array, their digits counted for the sort (its scratch's
// head cleared before), and every bucket emptied.
__global__ void __launch_bounds__(GRID_KEYS_THREADS) k_grid_keys(const float4* __restrict__ photons, uint32_t n, uint32_t frame,
                                                          float cell, uint32_t hash_bits, uint32_t* __restrict__ keys,
                                                          uint32_t* __restrict__ vals, uint32_t* __restrict__ scratch,
                                                          uint2* __restrict__ ranges, uint32_t entries) {
    __shared__ uint32_t counts[GRID_PASSES * 256];
    clear_counts(counts);
    const float3 j = grid_jitter(frame, cell);
    const int passes = rs_passes(0, (int)hash_bits + 1);
    for (uint32_t i = blockIdx.x * GRID_KEYS_THREADS + threadIdx.x; i < n; i += gridDim.x * GRID_KEYS_THREADS) {
        const uint32_t key = photon_key(photons[2ull * i], photons[2ull * i + 1], j, cell, hash_bits);
        keys[i] = key;
        vals[i] = i;
        rs_count_key(counts, key, 0, passes);
    }
    rs_clear_status(scratch, n);
    if (ranges != nullptr)
        for (uint32_t i = blockIdx.x * GRID_KEYS_THREADS + threadIdx.x; i < entries; i += gridDim.x * GRID_KEYS_THREADS)
            ranges[i] = make_uint2(0u, 0u);
    __syncthreads();
    rs_flush_counts(counts, scratch, passes);
}

__global__ void k_grid_ranges(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                              const uint32_t* n_dev, uint32_t n_host, uint32_t hash_bits,
                              const float4* __restrict__ photons, float4* __restrict__ sorted, uint32_t capacity,
                              uint2* __restrict__ ranges, const uint32_t* __restrict__ scratch, uint32_t* err) {
    uint32_t n = n_dev ? *n_dev : n_host;
    uint32_t sentinel = 1u << hash_bits;
    if (n != 0u && scratch[RS_GAVE_UP] != 0u) {  // the sort's wait gave up: no grid
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, ERR_WAIT_TIMEOUT);
        return;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t h = keys[i];
        uint32_t v = vals[i];
        const float4 dir = photons[2 * v + 1];
        sorted[i] = photons[2 * v];
        sorted[capacity + i] = dir;
        if (!(fabsf(dir.w) < __int_as_float(0x7F800000))) ranges[sentinel].x = 1u;
        if (h >= sentinel) continue;
        if (i == 0 || keys[i - 1] != h) ranges[h].x = i;
        if (i + 1 == n || keys[i + 1] != h) ranges[h].y = i + 1;
    }
}

// ------------------------------------------------------------------ camera paths
// Bounce-0 queue order (SRT_RAYGEN_TILE): queue position q -> pixel, with
// the pixels of a warp in an 8 x 4 tile (bands of 4 rows, 8-column blocks
// within a band; narrower blocks and bands at the right and bottom edges)
// instead of a 32 x 1 strip.  A bijection of [0, w h).  Config-2 camera rays
// of bounce 0: 0.383 vs 0.428 ms (a warp's rays closer in both directions);
// a path's result does not depend on its queue position.
#ifndef SRT_RAYGEN_TILE
#define SRT_RAYGEN_TILE 1
#endif
SRT_DEV void tile_pixel(uint32_t q, uint32_t w, uint32_t h, uint32_t& x, uint32_t& y) {
    const uint32_t band = q / (4u * w), y0 = 4u * band;
    const uint32_t hb = min(4u, h - y0);
    const uint32_t r = q - y0 * w;  // position inside the band
    const uint32_t blk = r / (8u * hb), x0 = 8u * blk;
    const uint32_t wb = min(8u, w - x0);
    const uint32_t t = r - x0 * hb;  // position inside the block
    x = x0 + t % wb;
    y = y0 + t / wb;
}

__global__ void k_raygen(FrameArgs a) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t n = a.width * a.height;
    const srt_camera_uniform& cam = *a.cam;
    // the frame's matrix, once per block instead of per pixel (1080p 47 -> 39 us;
    // 31 us to write the paths' state)
    __shared__ float m[16];
    if (threadIdx.x < 16u) m[threadIdx.x] = camera_elem(cam, threadIdx.x >> 2, threadIdx.x & 3u);
    __syncthreads();
    if (q >= n) return;
    uint32_t x, y;
    if (SRT_RAYGEN_TILE) tile_pixel(q, a.width, a.height, x, y);
    else {
        x = q % a.width;
        y = q / a.width;
    }
    const uint32_t p = x + y * a.width;
    uint32_t s = pcg_hash(x + y * a.width + cam.frame_count * 927163u + a.seed);
    float3 o, d;
    camera_ray(cam, m, x, y, a.width, a.height, s, o, d);
    float4 wl = sample_hero(s);
    a.pb.ray_o[p] = f4(o.x, o.y, o.z, 0.0001f);
    a.pb.ray_d[p] = f4(d.x, d.y, d.z, 100.0f);
    a.pb.thr[p] = splat4(1.0f);
    a.pb.wl[p] = wl;
    a.pb.rad[p] = splat4(0.0f);
    a.pb.misc[p] = make_uint4(s, 0u, p, 0u);
    a.pb.queue[0][q] = p;
    if (q == 0) {
        a.counters->paths[0] = n;
        a.counters->gather = gather_const(a.gather, cam.frame_count);
    }
}

struct LightSample {
    float3 dir;
    float dist, pdf;
    float2 emission;  // temperature, power
};

// sample_random_light: shader.wgsl:477-528 (the emitted radiance is left to the caller)
SRT_DEV LightSample sample_light(const DevScene& S, float3 hp, uint32_t& s) {
    LightSample ls;
    ls.pdf = 0.f;
    uint32_t nl = S.n_lights;
    if (nl == 0u) return ls;
    uint32_t li = min(__float2uint_rz(rng_next(s) * (float)nl), nl - 1u);
    float4 L0 = S.lights[4 * li], L1 = S.lights[4 * li + 1], L2 = S.lights[4 * li + 2], LP = S.lights[4 * li + 3];
    const float4 frame = S.light_frames[li];
    float r1 = rng_next(s);
    float r2 = rng_next(s);
    float sr1 = sqrtf(r1);
    float u = 1.0f - sr1, v = r2 * sr1, w = 1.0f - u - v;
    float3 p = xyz(L0) * u + xyz(L1) * v + xyz(L2) * w;
    float3 to = p - hp;
    float d2 = dot(to, to);
    float dist = sqrtf(d2);
    float3 l = to / dist;
    float cl = fmaxf(dot(xyz(frame), -l), 0.0f);
    if (cl <= 0.0001f) return ls;
    ls.dir = l;
    ls.dist = dist;
    ls.pdf = d2 / (frame.w * (float)nl * cl);
    ls.emission = make_float2(LP.y, LP.z);
    return ls;
}

// blackbody4 of the path's wavelengths at temperature t.  Lights mostly share
// one temperature, and a path meets light samples at most of its vertices: its
// value at the first light's is kept with the path (pb.light) from the first
// vertex that needs it.  (Four powf, expf and two divisions each: 0.29 of the
// 1.72 ms of config-2 shading per frame; kept, and with the lights' frames
// computed once, shading 1.57 -> 1.47 ms, the frame 8.01 -> 7.84 ms.)
SRT_DEV float4 path_blackbody(const FrameArgs& a, uint32_t id, float4 wl, float t, uint32_t& flags) {
    if (a.scene.n_lights == 0u || t != __ldg(&a.scene.lights[3].y)) return blackbody4(wl, t);
    if (flags & FLAG_LIGHT) return a.pb.light[id];
    const float4 r = blackbody4(wl, t);
    a.pb.light[id] = r;
    flags |= FLAG_LIGHT;
    return r;
}

// What one path's vertex produced: the continuation (written to the path
// state when alive), a shadow ray, or a vertex deferred to the guide.
struct VertexOut {
    bool alive = false, shadow = false, dark = false, guided = false;
    float3 sh_o = f3(0.f, 0.f, 0.f), sh_d = f3(0.f, 0.f, 0.f);
    float sh_tmax = 0.f;
    float4 sh_c = splat4(0.f);
    uint32_t key = 0u;
    bool gather = false;                // TAIL only: photons to gather, over ga_range at ga_p
    uint2 ga_range = make_uint2(0u, 0u);
    float3 ga_p = f3(0.f, 0.f, 0.f), ga_n = f3(0.f, 0.f, 0.f);
    float4 ga_f = splat4(0.f);
    float4 g_p = splat4(0.f), g_n = splat4(0.f), g_wo = splat4(0.f), g_spec = splat4(0.f);
};

// One iteration of ray_color's bounce loop after the closest-hit query
// (shader.wgsl:568-700) for path `id`, whose hit is in a.pb.hit[id]: writes
// the path's radiance and, when it continues, its next ray and state.  The
// photon gather of a diffuse vertex is left to launch_gather (queued here) or,
// TAIL, to the caller; either adds it before the vertex's shadow ray.
// GUIDE: Lambert continuations of bounces < guide_bounces are left to
// k_guide_infer (guide.cu); every guided renderer records the radiance a
// training record's next vertex sees.
template <bool GUIDE, bool TAIL>
SRT_DEV VertexOut shade_vertex(const FrameArgs& a, uint32_t id, uint32_t bounce) {
    VertexOut out;
    const DevScene& S = a.scene;
    float4 h = a.pb.hit[id];
    uint32_t prim = __float_as_uint(h.y);
    if (prim == MISS) return out;
    float4 o4 = a.pb.ray_o[id], d4 = a.pb.ray_d[id];
    float3 o = xyz(o4), d = xyz(d4);
    float4 thr = a.pb.thr[id], wl = a.pb.wl[id];
    uint4 misc = a.pb.misc[id];
    uint32_t s = misc.x, flags = misc.y;
    // a training record of the previous vertex: radiance before this vertex
    if (GUIDE && misc.w != 0u) a.guide.rec.rad[misc.w - 1u] = a.pb.rad[id];
    Surface sf = surface_at(S, prim, h.z, h.w, d);
    float4 color = S.materials[2 * sf.mat], extra = S.materials[2 * sf.mat + 1];
    float3 ffn = sf.front ? sf.wn : -sf.wn;
    uint32_t type = (uint32_t)extra.x;
    if (type == 3u) {
        if (!(flags & FLAG_CAUSTIC) && (sf.front || extra.y > 0.0f)) {
            float4 em = path_blackbody(a, id, wl, color.x, flags) * color.y;
            a.pb.rad[id] = a.pb.rad[id] + em * thr;
        }
        return out;
    }
    if (type == 0u) flags = (flags | FLAG_DIFFUSE) & ~FLAG_CAUSTIC;
    else if (type == 2u && (flags & FLAG_DIFFUSE)) flags |= FLAG_CAUSTIC;
    if (type == 0u) {
        float4 spec = rgb_to_spectrum4(xyz(color), wl);
        float3 hp = o + d * h.x;
        if (a.gather.enabled) {
            const GatherConst& k = a.counters->gather;
            const uint2 rg = gather_range(a.gather, k, hp);
            const float4 f = thr * (spec / PI);
            const float inf = __int_as_float(0x7F800000);
            // an empty range adds zeros (unless a factor is not finite)
            if (rg.y > rg.x || !within4(f, inf) || !(fabsf(k.density) < inf)) {
                if (TAIL) {
                    out.gather = true;
                    out.ga_range = rg;
                    out.ga_p = hp;
                    out.ga_n = ffn;
                    out.ga_f = f;
                } else {
                    // a slot for each lane that is here (in any grouping)
                    const uint32_t here = __activemask();
                    const uint32_t lane = threadIdx.x & 31u, leader = (uint32_t)__ffs(here) - 1u;
                    uint32_t slot = 0u;
                    if (lane == leader) slot = atomicAdd(&a.counters->gathers[bounce], (uint32_t)__popc(here));
                    slot = __shfl_sync(here, slot, (int)leader) + __popc(here & ((1u << lane) - 1u));
                    a.pb.ga_p[slot] = f4(hp.x, hp.y, hp.z, __uint_as_float(id));
                    a.pb.ga_n[slot] = f4(ffn.x, ffn.y, ffn.z, __uint_as_float(rg.y));
                    a.pb.ga_f[slot] = f;
                    a.pb.ga_start[slot] = rg.x;
                }
            }
        }
        LightSample ls = sample_light(S, hp, s);
        if (ls.pdf > 0.0f) {
            float ct = fmaxf(dot(ffn, ls.dir), 0.0f);
            const float4 f = thr * (spec / PI);
            // a light behind the surface adds zeros, whether its shadow ray is
            // blocked or not: the ray counts but is not traced (the bounds keep
            // every factor of its contribution finite).  Config 2: shadow rays
            // 2.33 -> 1.96 ms per frame, the frame 7.84 -> 7.52 ms; animated
            // 512x384 shadow rays 0.66 -> 0.60 ms.
            out.dark = ct == 0.0f && within4(f, 1e15f) && ls.pdf > 1e-30f && ls.emission.x >= 1.0f &&
                       ls.emission.x <= 1e6f && fabsf(ls.emission.y) < 1e15f;
            if (!out.dark) {
                float bpdf = ct / PI;
                float mis = ls.pdf / (ls.pdf + bpdf);
                const float4 radiance = path_blackbody(a, id, wl, ls.emission.x, flags) * ls.emission.y;
                out.sh_c = f * radiance * ct * (mis / ls.pdf);
                out.sh_o = hp;
                out.sh_d = ls.dir;
                out.sh_tmax = ls.dist - 0.001f;
                out.shadow = true;
            }
        }
        if (GUIDE && bounce + 1u < a.max_depth && bounce < a.guide_bounces) {
            out.guided = true;
            out.g_p = f4(hp.x, hp.y, hp.z, wl.x);
            out.g_n = f4(ffn.x, ffn.y, ffn.z, 0.f);
            out.g_wo = f4(-d.x, -d.y, -d.z, 0.f);
            out.g_spec = spec;
            a.pb.misc[id] = make_uint4(s, flags, misc.z, 0u);
            return out;
        }
    }
    Scatter sc = sample_bsdf(d, ffn, color, extra, sf.front, wl, thr, s);
    if (!sc.absorbed) {
        thr = thr * sc.att;
        o = o + d * h.x;
        bool alive = true;
        if (bounce > 3u) {
            float p = max4(thr);
            if (rng_next(s) > p) alive = false;
            else thr = thr / p;
        }
        if (bounce + 1u >= a.max_depth) alive = false;
        if (alive) {
            a.pb.thr[id] = thr;
            a.pb.ray_o[id] = f4(o.x, o.y, o.z, 0.0001f);
            a.pb.ray_d[id] = f4(sc.dir.x, sc.dir.y, sc.dir.z, 100.0f);
            a.pb.misc[id] = make_uint4(s, flags, misc.z, 0u);
            if (a.ray_sort) out.key = ray_sort_key(o, sc.dir, S.bmin, S.binv);
        }
        out.alive = alive;
    }
    return out;
}

// One bounce of every live path: shade_vertex, then the live paths, shadow
// rays and guided vertices go to their queues (warp-aggregated slots).
// shade_slot is one thread's vertex, of path `id` (not valid: no vertex; the
// thread still takes part in the warp's queue pushes).
template <bool GUIDE>
SRT_DEV void shade_slot(const FrameArgs& a, uint32_t bounce, uint32_t id, bool valid) {
    VertexOut v;
    if (valid) v = shade_vertex<GUIDE, false>(a, id, bounce);
    // the warp's places in its queues: one atomic instruction, a lane per queue
    // (one after the other each waited for the last one's answer; config-2
    // shading 1.331 -> 1.313 ms per frame)
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t m_alive = __ballot_sync(FULL, v.alive), m_shadow = __ballot_sync(FULL, v.shadow),
                   m_dark = __ballot_sync(FULL, v.dark), m_guided = GUIDE ? __ballot_sync(FULL, v.guided) : 0u;
    uint32_t* counter = &a.counters->paths[bounce + 1];
    uint32_t add = m_alive;
    if (lane == 1u) {
        counter = &a.counters->shadow[bounce];
        add = m_shadow;
    } else if (lane == 2u) {
        counter = &a.counters->dark[bounce];
        add = m_dark;
    } else if (GUIDE && lane == 3u) {
        counter = &a.guide.gc->verts[bounce];
        add = m_guided;
    }
    uint32_t base = 0u;
    if (lane < (GUIDE ? 4u : 3u) && add != 0u) base = atomicAdd(counter, (uint32_t)__popc(add));
    const uint32_t slot = __shfl_sync(FULL, base, 0) + __popc(m_alive & lt);
    if (v.alive) {
        a.pb.queue[(bounce + 1) & 1][slot] = id;
        if (a.ray_sort) a.pb.sort_keys[slot] = v.key;
    }
    const uint32_t sslot = __shfl_sync(FULL, base, 1) + __popc(m_shadow & lt);
    if (v.shadow) {
        a.pb.sh_o[sslot] = f4(v.sh_o.x, v.sh_o.y, v.sh_o.z, 0.001f);
        a.pb.sh_d[sslot] = f4(v.sh_d.x, v.sh_d.y, v.sh_d.z, v.sh_tmax);
        a.pb.sh_c[sslot] = v.sh_c;
        a.pb.sh_id[sslot] = id;
    }
    if (GUIDE) {
        const uint32_t gslot = __shfl_sync(FULL, base, 3) + __popc(m_guided & lt);
        if (v.guided) {
            a.guide.gv.p[gslot] = v.g_p;
            a.guide.gv.n[gslot] = v.g_n;
            a.guide.gv.wo[gslot] = v.g_wo;
            a.guide.gv.spec[gslot] = v.g_spec;
            a.guide.gv.id[gslot] = id;
        }
    }
}

#ifndef SRT_SHADE_BLOCK
#define SRT_SHADE_BLOCK 256
#endif
constexpr uint32_t SHADE_BLOCK = SRT_SHADE_BLOCK, SHADE_WARPS = SHADE_BLOCK / 32;
// A block's vertices are dealt to its threads by kind of material, so that most
// warps run one branch of shade_vertex (on config 2 from bounce 1 on, 15 of 32
// lanes were active).  With the words a hit needs next in the instance record,
// shading per frame: config 2 1.53 -> 1.41 ms, caustic slab 1.52 -> 1.47, others
// within 2 %; blocks of 128 / 512: config 2 1.44, 1.46, slab 1.49, 1.53.
constexpr uint32_t SHADE_KINDS = 4;  // ends here (no hit, emitter); diffuse; glossy; dielectric or film

template <bool GUIDE>
__global__ void __launch_bounds__(SHADE_BLOCK, SRT_SHADE_MIN_BLOCKS * TRACE_BLOCK / SHADE_BLOCK)
    k_shade(FrameArgs a, uint32_t bounce) {
    __shared__ uint32_t ids[SHADE_BLOCK], counts[SHADE_KINDS][SHADE_WARPS];
    const uint32_t n = a.counters->paths[bounce];
    const uint32_t first = blockIdx.x * SHADE_BLOCK, q = first + threadIdx.x;
    if (first >= n) return;
    const bool valid = q < n;
    uint32_t id = valid ? a.pb.queue[bounce & 1][q] : 0u;
    uint32_t kind = 0u;
    if (valid) {
        const uint32_t prim = __float_as_uint(a.pb.hit[id].y);
        if (prim != MISS) {
            const uint32_t type = __float_as_uint(a.scene.inst[__ldg(&a.scene.tri_inst[prim])].w2o2.w);
            kind = type == 3u ? 0u : (type == 1u || type == 5u) ? 2u : (type == 2u || type == 4u) ? 3u : 1u;
        }
    }
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t mine = 0u;
#pragma unroll
    for (uint32_t k = 0; k < SHADE_KINDS; ++k) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, valid && kind == k);
        if (lane == 0u) counts[k][warp] = (uint32_t)__popc(m);
        if (kind == k) mine = m;
    }
    __syncthreads();
    uint32_t at = __popc(mine & lt);
    for (uint32_t k = 0; k < SHADE_KINDS; ++k)
        for (uint32_t w = 0; w < SHADE_WARPS; ++w)
            if (k < kind || (k == kind && w < warp)) at += counts[k][w];
    if (valid) ids[at] = id;
    __syncthreads();
    if (valid) id = ids[threadIdx.x];
    shade_slot<GUIDE>(a, bounce, id, valid);
}

// The photon gathers a bounce queued (shade_vertex): one per thread, or one
// per eight lanes where they are few (at most SRT_GATHER_GROUP_WAVES for each
// group of the grid's lanes).  Their own launch, so that the lanes of a warp
// all walk a range: in the shading kernel, where one vertex in three lies in a
// caustic and walks up to 64 photons, 11 of 32 lanes were active.  Shading with
// the gathers, per frame: caustic slab at 1080p 2.35 -> 1.53 ms, Cornell 640x480
// 0.72 -> 0.48, config 1 0.28 -> 0.16, config 2 1.72 -> 1.57; frames 5.19 -> 4.14,
// 2.30 -> 1.98, 0.91 -> 0.73, 8.17 -> 8.01 ms.  Threshold 0 / 1 / 2 / 4 / 8 / 64:
// slab 1.60 / 1.55 / 1.53 / 1.53 / 1.53 / 1.73, Cornell 0.59 / 0.53 / 0.50 / 0.48 /
// 0.48 / 0.48, config 1 0.23 / 0.17 / 0.16 / 0.17 / 0.16 / 0.17, config 2 1.56 / 1.56
// / 1.56 / 1.57 / 1.60 / 1.59.
#ifndef SRT_GATHER_GROUP_WAVES
#define SRT_GATHER_GROUP_WAVES 4
#endif
__global__ void __launch_bounds__(TRACE_BLOCK, SRT_SHADE_MIN_BLOCKS) k_gather(FrameArgs a, uint32_t bounce) {
    const uint32_t n = a.counters->gathers[bounce];
    const GatherConst& k = a.counters->gather;
    if (n <= gridDim.x * (TRACE_BLOCK / GROUP) * SRT_GATHER_GROUP_WAVES) {
        const uint32_t c = threadIdx.x & 7u, group = threadIdx.x / GROUP;
        for (uint32_t base = blockIdx.x * (TRACE_BLOCK / GROUP); base < n; base += gridDim.x * (TRACE_BLOCK / GROUP)) {
            const uint32_t q = base + group;
            const bool have = q < n;
            const float4 p = have ? a.pb.ga_p[q] : splat4(0.f), nn = have ? a.pb.ga_n[q] : splat4(0.f);
            const uint2 range = make_uint2(have ? a.pb.ga_start[q] : 0u, __float_as_uint(nn.w));
            const uint32_t id = __float_as_uint(p.w);
            const float4 gl = gather_group(a.gather, k, have, range, xyz(p), xyz(nn), have ? a.pb.wl[id] : splat4(0.f));
            if (have && c == 0u) a.pb.rad[id] = a.pb.rad[id] + a.pb.ga_f[q] * gl;
        }
        return;
    }
    for (uint32_t q = blockIdx.x * TRACE_BLOCK + threadIdx.x; q < n; q += gridDim.x * TRACE_BLOCK) {
        const float4 p = a.pb.ga_p[q], nn = a.pb.ga_n[q];
        const uint32_t id = __float_as_uint(p.w);
        const float4 gl = gather(a.gather, k, make_uint2(a.pb.ga_start[q], __float_as_uint(nn.w)), xyz(p), xyz(nn),
                                 a.pb.wl[id]);
        a.pb.rad[id] = a.pb.rad[id] + a.pb.ga_f[q] * gl;
    }
}

// Resident blocks per SM the tail kernel is compiled for (traversal and
// shading in one kernel: 4 blocks of 128 allow 128 registers).
#ifndef SRT_TAIL_MIN_BLOCKS
#define SRT_TAIL_MIN_BLOCKS 4
#endif

// The last bounces of the live paths in one persistent launch: a group of
// eight lanes takes a path entering bounce `first` and follows it to its end
// (closest hit on the group's lanes, shade_vertex on its first, its shadow ray
// on all again), then takes the next path.  Per path the operations and the
// order of its radiance updates are those of the bounce-by-bounce wavefront
// (a ray is answered alike by every kernel), so the image is bit-identical;
// where few paths remain, one launch replaces a chain of launches that each
// last as long as their slowest ray.  What bounds it is the chain of one path
// (closest hit, shading, shadow ray, next bounce): with a thread per path and
// lanes of a warp at different stages it took 0.89 ms on config 2 (bounces 5-11
// of 59k paths) and 0.73 ms on config 1 (bounces 1-7 of 65k); the lanes of a
// group share a ray's node visits and the groups of a warp keep in step, and
// with the launches before it (trace_groups) config 2 8.35 -> 8.17 ms per frame,
// config 1 15.6 -> 14.6 ms per 16 frames, prism 96x64 0.445 -> 0.330 ms.
template <bool GUIDE, bool COUNT, int STACK>
__global__ void __launch_bounds__(TRACE_BLOCK, SRT_TAIL_MIN_BLOCKS) k_tail(FrameArgs a, uint32_t first) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    __shared__ uint32_t n_closest[MAX_BOUNCES + 1], n_shadow[MAX_BOUNCES + 1];
    for (uint32_t i = threadIdx.x; i <= (uint32_t)MAX_BOUNCES; i += blockDim.x) n_closest[i] = n_shadow[i] = 0u;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, c = lane & 7u, shift = lane & 24u;
    const uint32_t n = a.counters->paths[first];
    uint32_t* fetch = &a.counters->fetch[TRAV_CLOSEST][first];
    const uint32_t* queue = a.pb.queue[first & 1];
    GroupTrav<STACK> T;
    T.sp = 0;
    T.axes = 0u;
    bool live = false, exhausted = false;
    uint32_t id = 0u, b = first;
    while (true) {
        const uint32_t idle = __ballot_sync(FULL, !live) & GROUP_LEADERS;
        if (!exhausted && idle) {
            uint32_t base = 0u;
            if (lane == 0u) base = atomicAdd(fetch, (uint32_t)__popc(idle));
            base = __shfl_sync(FULL, base, 0);
            if (base + (uint32_t)__popc(idle) >= n) exhausted = true;
            const uint32_t q = base + __popc(idle & ((1u << shift) - 1u));
            if (!live && q < n) {
                id = queue[q];
                b = first;
                live = true;
            }
        }
        if (__ballot_sync(FULL, live) == 0u) break;  // exhausted: a fetch that gave no path was past the end
        // two rays per bounce through one copy of the traversal: the closest
        // hit, then (after shading) the shadow ray.  A warp runs this loop's
        // code once per bounce and waits for it: with a copy for each ray the
        // kernel took 0.201 vs 0.174 ms on config 2, 0.176 vs 0.146 on the caustic
        // slab, 0.117 vs 0.100 on config 1.
        VertexOut vo;
        uint32_t alive = 0u;
#pragma unroll 1
        for (int ray = 0; ray < 2; ++ray) {
            uint32_t nodes = 0u, tris = 0u;
            float3 ro = f3(0.f, 0.f, 0.f), rd = ro;
            float rmin = 0.001f, rmax = 0.f;
            bool has = live;
            if (ray == 0) {
                if (live) {
                    // paths[first] was counted by the last shading step
                    if (b > first && c == 0u) atomicAdd(&n_closest[b], 1u);
                    const float4 o = a.pb.ray_o[id], d = a.pb.ray_d[id];
                    ro = xyz(o);
                    rd = xyz(d);
                    rmin = o.w;
                    rmax = d.w;
                }
            } else {
                const uint32_t shadow = __ballot_sync(FULL, vo.shadow);
                if (shadow == 0u) break;
                ro = f3(__shfl_sync(FULL, vo.sh_o.x, (int)shift), __shfl_sync(FULL, vo.sh_o.y, (int)shift),
                        __shfl_sync(FULL, vo.sh_o.z, (int)shift));
                rd = f3(__shfl_sync(FULL, vo.sh_d.x, (int)shift), __shfl_sync(FULL, vo.sh_d.y, (int)shift),
                        __shfl_sync(FULL, vo.sh_d.z, (int)shift));
                rmax = __shfl_sync(FULL, vo.sh_tmax, (int)shift);
                has = ((shadow >> shift) & 1u) != 0u;
            }
            T.id = MISS;
            bool act = has && group_init(T, a.scene, ro, rd, rmin, rmax);
            while (__any_sync(FULL, act))
                if (group_step(a.scene, T, act, ray == 1, a.err, nodes, tris)) act = false;
            if (COUNT && has) {
                const int kind = ray == 0 ? TRAV_CLOSEST : TRAV_SHADOW;
                atomicAdd(&a.stats->nodes_bounce[kind][b], (unsigned long long)nodes);
                atomicAdd(&a.stats->tris_bounce[kind][b], (unsigned long long)tris);
            }
            if (ray == 0) {
                float t, u, v;
                uint32_t prim;
                group_closest(T, t, prim, u, v);
                if (live && c == 0u) {
                    a.pb.hit[id] = prim != MISS ? make_float4(t, __uint_as_float(prim), u, v)
                                                : make_float4(0.f, __uint_as_float(MISS), 0.f, 0.f);
                    vo = shade_vertex<GUIDE, true>(a, id, b);
                }
                __syncwarp();  // the path's next ray, written by the group's first lane, is read by all
                alive = __ballot_sync(FULL, vo.alive);
                if (__any_sync(FULL, vo.gather)) {
                    const bool ga = __shfl_sync(FULL, (int)vo.gather, (int)shift) != 0;
                    const uint2 range = make_uint2(__shfl_sync(FULL, vo.ga_range.x, (int)shift),
                                                   __shfl_sync(FULL, vo.ga_range.y, (int)shift));
                    const float3 p =
                        f3(__shfl_sync(FULL, vo.ga_p.x, (int)shift), __shfl_sync(FULL, vo.ga_p.y, (int)shift),
                           __shfl_sync(FULL, vo.ga_p.z, (int)shift));
                    const float3 nn =
                        f3(__shfl_sync(FULL, vo.ga_n.x, (int)shift), __shfl_sync(FULL, vo.ga_n.y, (int)shift),
                           __shfl_sync(FULL, vo.ga_n.z, (int)shift));
                    const float4 gl = gather_group(a.gather, a.counters->gather, ga, range, p, nn,
                                                   ga ? a.pb.wl[id] : splat4(0.f));
                    if (ga && c == 0u) a.pb.rad[id] = a.pb.rad[id] + vo.ga_f * gl;
                }
            } else {
                const bool occluded = group_occluded(T);
                if (has && c == 0u) {
                    atomicAdd(&n_shadow[b], 1u);
                    if (!occluded) {  // as the shadow-ray kernel adds it (shader.wgsl:659-669)
                        const float4 r = a.pb.rad[id], k = vo.sh_c;
                        a.pb.rad[id] = make_float4(__fadd_rn(r.x, k.x), __fadd_rn(r.y, k.y), __fadd_rn(r.z, k.z),
                                                   __fadd_rn(r.w, k.w));
                    }
                }
            }
        }
        if (vo.dark) atomicAdd(&n_shadow[b], 1u);
        live = live && ((alive >> shift) & 1u) != 0u;
        ++b;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= (uint32_t)MAX_BOUNCES; i += blockDim.x) {
        if (n_closest[i]) atomicAdd(&a.counters->paths[i], n_closest[i]);
        if (n_shadow[i]) atomicAdd(&a.counters->shadow[i], n_shadow[i]);
    }
}

// Resident blocks per SM of one k_tail instantiation (its grid is one wave).
template <bool GUIDE, bool COUNT, int STACK>
int tail_per_sm() {
    static int per_sm = 0;
    if (per_sm == 0) {
        int x = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&x, k_tail<GUIDE, COUNT, STACK>, TRACE_BLOCK, 0) !=
                cudaSuccess ||
            x < 1)
            x = 1;
        per_sm = x;
    }
    return per_sm;
}

template <bool GUIDE, bool COUNT, int STACK>
int launch_tail_t(const FrameArgs& a, uint32_t first, cudaStream_t st) {
    const uint32_t grid = (uint32_t)(a.sm_count > 0 ? a.sm_count : 148) * (uint32_t)tail_per_sm<GUIDE, COUNT, STACK>();
    k_tail<GUIDE, COUNT, STACK><<<grid, TRACE_BLOCK, 0, st>>>(a, first);
    return 1;
}

// shader.wgsl:774-822: hero tuple -> XYZ / sum pdf -> linear sRGB ->
// accumulate (reset at frame 0) -> mean -> Reinhard on luma -> RGBA8.
__global__ void k_finalize(FrameArgs a) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.width * a.height) return;
    float4 L = a.pb.rad[p], wl = a.pb.wl[p];
    float3 c = f3(0.f, 0.f, 0.f);
    c = c + sample_cie_xyz(wl.x) * L.x;
    c = c + sample_cie_xyz(wl.y) * L.y;
    c = c + sample_cie_xyz(wl.z) * L.z;
    c = c + sample_cie_xyz(wl.w) * L.w;
    c = c * (1.0f / hero_pdf_sum(wl));
    float3 rgb = xyz_to_srgb(c);
    uint32_t frame = a.cam->frame_count;
    float4 acc = frame > 0u ? a.accum[p] : splat4(0.f);
    acc = acc + f4(rgb.x, rgb.y, rgb.z, 1.0f);
    a.accum[p] = acc;
    if (a.accum64) {
        double4 d = frame > 0u ? a.accum64[p] : make_double4(0, 0, 0, 0);
        a.accum64[p] = make_double4(d.x + rgb.x, d.y + rgb.y, d.z + rgb.z, d.w + 1.0);
    }
    float3 fc = f3(fmaxf(acc.x / acc.w * 1.0f, 0.f), fmaxf(acc.y / acc.w * 1.0f, 0.f), fmaxf(acc.z / acc.w * 1.0f, 0.f));
    float luma = fc.x * 0.2126f + fc.y * 0.7152f + fc.z * 0.0722f;
    float mapped = luma / (luma + 1.0f);
    if (luma > 0.00001f) fc = fc * (mapped / luma);
    a.ldr[p] = make_uchar4((unsigned char)__float2uint_rn(clampf(fc.x, 0.f, 1.f) * 255.0f),
                           (unsigned char)__float2uint_rn(clampf(fc.y, 0.f, 1.f) * 255.0f),
                           (unsigned char)__float2uint_rn(clampf(fc.z, 0.f, 1.f) * 255.0f), 255);
}

// After the ray sort of the paths entering bounce + 1: where its bounded wait
// gave up the queue may hold anything, so no path goes on and the frame reports it.
__global__ void k_check_sort(FrameArgs a, uint32_t bounce) {
    if (threadIdx.x != 0 || a.pb.sort_scratch[RS_GAVE_UP] == 0u || a.counters->paths[bounce + 1] == 0u) return;
    a.counters->paths[bounce + 1] = 0u;
    atomicOr(a.err, ERR_WAIT_TIMEOUT);
}

// One lane per bounce (a chain of loads per bounce on one thread took 6 us at
// the end of every frame).
__global__ void k_frame_stats(FrameArgs a) {
    static_assert(MAX_BOUNCES + 1 == 32 && MAX_PHOTON_BOUNCES < 32, "one warp");
    const uint32_t i = threadIdx.x;
    const bool camera = i < a.max_depth, photon = a.photons_per_frame > 0u && i < a.photon_max_bounces;
    const uint32_t c = camera ? a.counters->paths[i] : 0u;
    const uint32_t s = camera ? a.counters->shadow[i] + a.counters->dark[i] : 0u;
    // bounce 0: every emitted ray, also those the cull answered
    const uint32_t p = !photon ? 0u : i == 0u ? a.ph_counters->photons_emitted : a.ph_counters->photon_paths[i];
    unsigned long long all[3] = {c, s, p};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < 3; ++k) all[k] += __shfl_down_sync(0xFFFFFFFFu, all[k], o);
    if (camera) {
        a.stats->rays_bounce[TRAV_CLOSEST][i] += c;
        a.stats->rays_bounce[TRAV_SHADOW][i] += s;
    }
    if (photon) a.stats->rays_bounce[TRAV_PHOTON][i] += p;
    if (i == 0u) {
        a.stats->closest_rays += all[0];
        a.stats->shadow_rays += all[1];
        a.stats->photon_rays += all[2];
        a.stats->paths += c;
    }
}

// ------------------------------------------------------------------ batch / test kernels
__global__ void k_gather_queries(GatherArgs g, uint32_t frame, const float* __restrict__ q, uint32_t n,
                                 float4* __restrict__ out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* a = q + 10 * i;
    const GatherConst k = gather_const(g, frame);
    const float3 p = f3(a[0], a[1], a[2]);
    out[i] = gather(g, k, gather_range(g, k, p), p, f3(a[3], a[4], a[5]), f4(a[6], a[7], a[8], a[9]));
}

__global__ void k_test_math(int op, uint32_t n, const void* __restrict__ in, void* __restrict__ out,
                            const void* __restrict__ aux) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* fi = (const float*)in;
    const uint32_t* ui = (const uint32_t*)in;
    float* fo = (float*)out;
    uint32_t* uo = (uint32_t*)out;
    switch (op) {
        case 0:
            uo[i] = pcg_hash(ui[i]);
            break;
        case 1: {
            float3 c = sample_cie_xyz(fi[i]);
            fo[3 * i] = c.x;
            fo[3 * i + 1] = c.y;
            fo[3 * i + 2] = c.z;
        } break;
        case 2:
            fo[i] = blackbody(fi[2 * i], fi[2 * i + 1]);
            break;
        case 3: {
            const float* p = fi + 7 * i;
            float4 r = rgb_to_spectrum4(f3(p[0], p[1], p[2]), f4(p[3], p[4], p[5], p[6]));
            reinterpret_cast<float4*>(fo)[i] = r;
        } break;
        case 4: {
            const float* p = fi + 9 * i;
            reinterpret_cast<float4*>(fo)[i] = thin_film4(p[0], p[1], p[2], p[3], p[4], f4(p[5], p[6], p[7], p[8]));
        } break;
        case 5: {
            uint32_t s = ui[i];
            float4 w = sample_hero(s);
            float* o = fo + 5 * i;
            o[0] = w.x;
            o[1] = w.y;
            o[2] = w.z;
            o[3] = w.w;
            o[4] = hero_pdf_sum(w);
        } break;
        case 6: {
            const float* p = fi + 24 * i;
            uint32_t s = __float_as_uint(p[23]);
            Scatter sc = sample_bsdf(f3(p[0], p[1], p[2]), f3(p[3], p[4], p[5]), f4(p[6], p[7], p[8], p[9]),
                                     f4(p[10], p[11], p[12], p[13]), p[14] != 0.0f, f4(p[15], p[16], p[17], p[18]),
                                     f4(p[19], p[20], p[21], p[22]), s);
            float* o = fo + 10 * i;
            o[0] = sc.dir.x;
            o[1] = sc.dir.y;
            o[2] = sc.dir.z;
            o[3] = sc.att.x;
            o[4] = sc.att.y;
            o[5] = sc.att.z;
            o[6] = sc.att.w;
            o[7] = sc.absorbed ? 1.0f : 0.0f;
            o[8] = __uint_as_float(s);
            o[9] = 0.f;
        } break;
        case 7: {
            const float* p = fi + 5 * i;
            float3 j = grid_jitter(__float_as_uint(p[3]), p[4]);
            uo[i] = grid_hash(f3(p[0], p[1], p[2]), j, p[4], 22);
        } break;
        case 8: {
            const uint32_t* p = ui + 5 * i;
            uint32_t s = p[4];
            float3 o, d;
            const srt_camera_uniform& cam = *(const srt_camera_uniform*)aux;
            float m[16];
            for (uint32_t e = 0; e < 16u; ++e) m[e] = camera_elem(cam, e >> 2, e & 3u);
            camera_ray(cam, m, p[0], p[1], p[2], p[3], s, o, d);
            float* r = fo + 7 * i;
            r[0] = o.x;
            r[1] = o.y;
            r[2] = o.z;
            r[3] = d.x;
            r[4] = d.y;
            r[5] = d.z;
            r[6] = __uint_as_float(s);
        } break;
        case 9: {
            const float* p = fi + 5 * i;
            uo[i] = within4(f4(p[0], p[1], p[2], p[3]), p[4]) ? 1u : 0u;
        } break;
        default:
            break;
    }
}

inline uint32_t blocks_for(uint64_t n, uint32_t b) { return (uint32_t)((n + b - 1) / b); }

}  // namespace

// ------------------------------------------------------------------ launchers
int launch_photon_pass(FrameArgs& a, cudaStream_t st) {
    int launches = 0;
    const uint32_t n = a.photons_per_frame;
    cudaMemsetAsync(a.ph.ranges, 0, sizeof(uint2) * range_entries(a.gather.hash_bits), st);
    const uint32_t blocks = blocks_for(n, TRACE_BLOCK);
    const uint32_t grid_max = (uint32_t)(a.sm_count > 0 ? a.sm_count : 148) * SRT_SHADE_MIN_BLOCKS;
    const uint32_t pass_grid = std::min(blocks, grid_max);
    if (a.scene.depth <= (uint32_t)TRAV_STACK_SMALL)
        k_photon_emit<TRAV_STACK_SMALL><<<pass_grid, TRACE_BLOCK, sizeof(uint2) * TRAV_STACK_SMALL * TRACE_BLOCK, st>>>(a);
    else k_photon_emit<TRAV_STACK><<<pass_grid, TRACE_BLOCK, sizeof(uint2) * TRAV_STACK * TRACE_BLOCK, st>>>(a);
    ++launches;
    for (uint32_t b = 0; b < a.photon_max_bounces; ++b) {
        launches += launch_trace_queue(a.scene, b, a.ph.queue[b & 1], &a.counters->photon_paths[b],
                                       &a.counters->fetch[TRAV_PHOTON][b], n, a.ph.ray_o, a.ph.ray_d, a.ph.hit,
                                       TRAV_PHOTON, a.count_visits, a.err, a.stats, a.sm_count, st);
        k_photon_shade<<<pass_grid, TRACE_BLOCK, 0, st>>>(a, b);
        ++launches;
    }
    // stored photons in emitter order with their keys, then the grid
    k_deposit<<<deposit_tiles(n), RS_THREADS, 0, st>>>(a);
    ++launches;
    launches += sort_passes(a.ph.keys, a.ph.vals, a.ph.keys2, a.ph.vals2, a.ph.capacity, &a.counters->photons_stored, 0,
                            (int)a.gather.hash_bits + 1, a.ph.sort_scratch, st, &a.ph.sorted_keys, &a.ph.sorted_vals);
    k_grid_ranges<<<148 * 8, 256, 0, st>>>(a.ph.sorted_keys, a.ph.sorted_vals, &a.counters->photons_stored, 0,
                                           a.gather.hash_bits, a.ph.photons, a.ph.sorted, a.ph.capacity, a.ph.ranges,
                                           a.ph.sort_scratch, a.err);
    ++launches;
    return launches;
}

GridKeysKernel grid_keys_kernel() { return k_grid_keys; }

int launch_grid_build(const float4* photons, uint32_t n, uint32_t frame, float cell, uint32_t hash_bits,
                      PhotonBuffers& ph, uint32_t* err, cudaStream_t st) {
    int launches = 0;
    cudaMemsetAsync(ph.sort_scratch, 0, RS_HEAD * sizeof(uint32_t), st);
    k_grid_keys<<<grid_keys_blocks(n), GRID_KEYS_THREADS, 0, st>>>(photons, n, frame, cell, hash_bits, ph.keys, ph.vals,
                                                           ph.sort_scratch, ph.ranges,
                                                           (uint32_t)range_entries(hash_bits));
    ++launches;
    launches += sort_passes(ph.keys, ph.vals, ph.keys2, ph.vals2, n, nullptr, 0, (int)hash_bits + 1, ph.sort_scratch, st,
                            &ph.sorted_keys, &ph.sorted_vals);
    k_grid_ranges<<<148 * 8, 256, 0, st>>>(ph.sorted_keys, ph.sorted_vals, nullptr, n, hash_bits, photons, ph.sorted, n,
                                           ph.ranges, ph.sort_scratch, err);
    ++launches;
    return launches;
}

int launch_light_frames(const float4* lights, uint32_t n, float4* frames, cudaStream_t st) {
    if (n == 0) return 0;
    k_light_frames<<<blocks_for(n, 128), 128, 0, st>>>(lights, n, frames);
    return 1;
}

int launch_raygen(const FrameArgs& a, cudaStream_t st) {
    k_raygen<<<blocks_for((uint64_t)a.width * a.height, 256), 256, 0, st>>>(a);
    return 1;
}

int launch_bounce(const FrameArgs& a, uint32_t bounce, cudaStream_t st, int stage) {
    int launches = 0;
    const uint32_t grid = blocks_for((uint64_t)a.width * a.height, SHADE_BLOCK);
    if (stage == 1) launches += launch_trace_closest(a, bounce, st);
    if (stage == 2 || stage == 4) {
        if (a.guiding) k_shade<true><<<grid, SHADE_BLOCK, 0, st>>>(a, bounce);
        else k_shade<false><<<grid, SHADE_BLOCK, 0, st>>>(a, bounce);
        ++launches;
        if (a.guiding && stage != 4 && bounce + 1 < a.max_depth && bounce < a.guide_bounces)
            launches += launch_guide_infer(a, bounce, st);
        if (a.ray_sort && bounce + 1 < a.max_depth) {
            // 4 passes: the sorted queue lands back in the queue buffer
            uint32_t *sk, *sv;
            launches += sort_pairs(a.pb.sort_keys, a.pb.queue[(bounce + 1) & 1], a.pb.sort_keys_alt,
                                   a.pb.sort_vals_alt, a.width * a.height, &a.counters->paths[bounce + 1], 0, 32,
                                   a.pb.sort_scratch, st, &sk, &sv);
            k_check_sort<<<1, 32, 0, st>>>(a, bounce);
            ++launches;
        }
    }
    if (stage == 3) launches += launch_trace_shadow(a, bounce, st);
    return launches;
}

int launch_gather(const FrameArgs& a, uint32_t bounce, cudaStream_t st) {
    if (!a.gather.enabled) return 0;
    const uint32_t grid = std::min(blocks_for((uint64_t)a.width * a.height, TRACE_BLOCK / GROUP),
                                   (uint32_t)(a.sm_count > 0 ? a.sm_count : 148) * SRT_SHADE_MIN_BLOCKS);
    k_gather<<<grid, TRACE_BLOCK, 0, st>>>(a, bounce);
    return 1;
}

int launch_finalize(const FrameArgs& a, cudaStream_t st) {
    k_finalize<<<blocks_for((uint64_t)a.width * a.height, 256), 256, 0, st>>>(a);
    return 1;
}

int launch_frame_stats(const FrameArgs& a, cudaStream_t st) {
    k_frame_stats<<<1, 32, 0, st>>>(a);
    return 1;
}

uint32_t tail_paths(const FrameArgs& a) {
    const bool small = a.scene.depth <= (uint32_t)TRAV_STACK_SMALL;
    const bool g = a.guiding != 0, c = a.count_visits != 0;
    int per_sm;
    if (c) per_sm = g ? (small ? tail_per_sm<true, true, TRAV_STACK_SMALL>() : tail_per_sm<true, true, TRAV_STACK>())
                      : (small ? tail_per_sm<false, true, TRAV_STACK_SMALL>() : tail_per_sm<false, true, TRAV_STACK>());
    else per_sm = g ? (small ? tail_per_sm<true, false, TRAV_STACK_SMALL>() : tail_per_sm<true, false, TRAV_STACK>())
                    : (small ? tail_per_sm<false, false, TRAV_STACK_SMALL>() : tail_per_sm<false, false, TRAV_STACK>());
    return (uint32_t)(a.sm_count > 0 ? a.sm_count : 148) * (uint32_t)per_sm * (TRACE_BLOCK / GROUP);
}

int launch_tail(const FrameArgs& a, uint32_t first, cudaStream_t st) {
    if (first >= a.max_depth) return 0;
    const bool small = a.scene.depth <= (uint32_t)TRAV_STACK_SMALL;
    const bool g = a.guiding != 0;
    if (a.count_visits) {
        if (g) return small ? launch_tail_t<true, true, TRAV_STACK_SMALL>(a, first, st) : launch_tail_t<true, true, TRAV_STACK>(a, first, st);
        return small ? launch_tail_t<false, true, TRAV_STACK_SMALL>(a, first, st) : launch_tail_t<false, true, TRAV_STACK>(a, first, st);
    }
    if (g) return small ? launch_tail_t<true, false, TRAV_STACK_SMALL>(a, first, st) : launch_tail_t<true, false, TRAV_STACK>(a, first, st);
    return small ? launch_tail_t<false, false, TRAV_STACK_SMALL>(a, first, st) : launch_tail_t<false, false, TRAV_STACK>(a, first, st);
}

int launch_gather_queries(const GatherArgs& g, uint32_t frame, const float* queries, uint32_t n_q, float4* out,
                          cudaStream_t st) {
    if (n_q == 0) return 0;
    k_gather_queries<<<blocks_for(n_q, 128), 128, 0, st>>>(g, frame, queries, n_q, out);
    return 1;
}

int launch_test_math(int op, uint32_t n, const void* in, void* out, const void* aux, cudaStream_t st) {
    if (n == 0) return 0;
    k_test_math<<<blocks_for(n, 128), 128, 0, st>>>(op, n, in, out, aux);
    return 1;
}

}  // namespace srt
