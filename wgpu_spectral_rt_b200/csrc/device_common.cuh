// device_common.cuh — device data layouts and shading math of the spectral
// path tracer (sm_100a).
//
// The shading functions follow the reference WGSL (path:line cited at each
// one) in FP32; they are written for the GPU (float4 SIMD-style helpers,
// register-resident state) and checked against the CPU oracle.
#pragma once
#include <cuda_fp16.h>

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/srt.h"

#define SRT_DEV __device__ __forceinline__

namespace srt {

constexpr float PI = 3.14159265359f;  // shader.wgsl:6
constexpr float LAMBDA_MIN = 380.0f;  // shader.wgsl:81-83
constexpr float LAMBDA_MAX = 780.0f;
constexpr float LAMBDA_RANGE = LAMBDA_MAX - LAMBDA_MIN;
constexpr uint32_t MISS = 0xFFFFFFFFu;
constexpr int TRAV_STACK = 32;        // BVH8 traversal stack entries per thread (deepest supported tree)
constexpr int TRAV_STACK_SMALL = 16;  // stack for trees of at most 16 levels (less shared memory, more warps)

// Device error word bits (read back by the host after synchronising).
constexpr uint32_t ERR_STACK_OVERFLOW = 0x1u;
constexpr uint32_t ERR_QUEUE_OVERFLOW = 0x2u;
constexpr uint32_t ERR_BAD_INDEX = 0x4u;
constexpr uint32_t ERR_WAIT_TIMEOUT = 0x40u;  // a bounded look-back (deposit, sort) gave up

// ------------------------------------------------------------------ layouts
// Per instance (64 B): mesh/material ids, first flattened triangle and the
// rows of world_to_object (inverse of the instance's linear part).
struct InstDev {
    uint32_t mesh_id, mat_id, tri_offset, tri_count;
    // rows; the .w lanes hold words a hit needs next, a load earlier than from
    // the mesh and material tables: the mesh's first vertex, its first index - 3
    // tri_offset (mod 2^32), the material type
    float4 w2o0, w2o1, w2o2;
};

// Compressed 8-wide BVH node, 80 B = 5 x uint4 (layout of Ylitie, Karras and
// Laine, HPG 2017):
//  w0..2  origin p (float x3)     w3  exponent bytes ex, ey, ez, imask
//  w4     first child node index  w5  first triangle slot index
//  w6..7  meta[8]: 0 empty; (7 << 5) internal child; (count << 5) | offset
//         for a leaf of `count` (1..3) triangles starting at
//         first triangle slot + offset
//  w8..19 qlo.x[8] qlo.y[8] qlo.z[8] qhi.x[8] qhi.y[8] qhi.z[8]
// Child bounds = p + 2^(e-127) * q.
struct Node8 {
    uint4 a, b, c, d, e;
};
static_assert(sizeof(Node8) == 80, "Node8 must be 80 bytes");

// A leaf triangle slot (48 B): world-space v0.xyz + flattened triangle id
// (bits in .w), v1.xyz, v2.xyz.
struct TriSlot {
    float4 v0, v1, v2;
};

struct DevScene {
    const float4* vtx;          // srt_vertex: pos, normal
    const uint32_t* indices;
    const uint4* mesh_infos;    // srt_mesh_info
    const float4* materials;    // srt_material: color, extra
    const float4* lights;       // srt_light: v0, v1, v2, params
    const float4* light_frames; // per light: unit normal, area (k_light_frames)
    uint32_t n_lights;
    const InstDev* inst;
    const uint32_t* tri_inst;   // flattened triangle -> instance
    const Node8* nodes;
    const TriSlot* tris;
    const uint8_t* scatter;     // per node: child slots whose subtree holds a scattering triangle (k_scatter_mask)
    uint32_t n_nodes;
    uint32_t n_tris;
    uint32_t depth;  // 8-wide levels: a traversal stack needs at least this many entries
    float4 bmin;     // world bounds of the scene (xyz), for ray sort keys
    float4 binv;     // 1 / extent of the bounds (xyz)
};

// ------------------------------------------------------------------ vector helpers
SRT_DEV float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
SRT_DEV float3 xyz(float4 a) { return make_float3(a.x, a.y, a.z); }
SRT_DEV float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
SRT_DEV float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
SRT_DEV float3 operator-(float3 a) { return f3(-a.x, -a.y, -a.z); }
SRT_DEV float3 operator*(float3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
SRT_DEV float3 operator/(float3 a, float s) { return f3(a.x / s, a.y / s, a.z / s); }
SRT_DEV float dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
SRT_DEV float3 cross(float3 a, float3 b) {
    return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
SRT_DEV float length(float3 a) { return sqrtf(dot(a, a)); }
SRT_DEV float3 normalize(float3 a) { return a / length(a); }
SRT_DEV float3 reflect(float3 i, float3 n) { return i - n * (2.0f * dot(n, i)); }
SRT_DEV float3 refract(float3 i, float3 n, float eta) {
    float ni = dot(n, i);
    float k = 1.0f - eta * eta * (1.0f - ni * ni);
    if (k < 0.0f) return f3(0.f, 0.f, 0.f);
    return i * eta - n * (eta * ni + sqrtf(k));
}
SRT_DEV float4 f4(float x, float y, float z, float w) { return make_float4(x, y, z, w); }
SRT_DEV float4 splat4(float s) { return make_float4(s, s, s, s); }
SRT_DEV float4 operator+(float4 a, float4 b) { return f4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
SRT_DEV float4 operator-(float4 a, float4 b) { return f4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
SRT_DEV float4 operator*(float4 a, float4 b) { return f4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
SRT_DEV float4 operator/(float4 a, float4 b) { return f4(a.x / b.x, a.y / b.y, a.z / b.z, a.w / b.w); }
SRT_DEV float4 operator*(float4 a, float s) { return f4(a.x * s, a.y * s, a.z * s, a.w * s); }
SRT_DEV float4 operator/(float4 a, float s) { return f4(a.x / s, a.y / s, a.z / s, a.w / s); }
SRT_DEV float max4(float4 a) { return fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)); }
// Every component lies within (-bound, bound); a NaN among them does not
// (max4 drops one beside a number).
SRT_DEV bool within4(float4 a, float bound) {
    return fabsf(a.x) < bound && fabsf(a.y) < bound && fabsf(a.z) < bound && fabsf(a.w) < bound;
}
SRT_DEV float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
SRT_DEV float sq(float x) { return x * x; }
SRT_DEV float signf(float x) { return x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f); }

// ------------------------------------------------------------------ RNG (shader.wgsl:144-169)
SRT_DEV uint32_t pcg_hash(uint32_t input) {
    uint32_t state = input * 747796405u + 2891336453u;
    uint32_t word = ((state >> ((state >> 28u) + 4u)) ^ state) * 277803737u;
    return (word >> 22u) ^ word;
}
// rand(): f32(u32) / 4294967295.0 — the f32 constant is 2^32, so the
// quotient is an exact scaling of the rounded u32, and so is the product with
// 2^-32: the same bits without a division (config-2 frame 7.00 -> 6.90 ms,
// caustic slab 3.88 -> 3.84).  The guide's kernels keep the division
// (SRT_RNG_DIVIDE): they are compiled with contraction, and there the product
// moves which multiplies the compiler fuses, so a frozen guide's image changes
// in its last bits, and at a few pixels in its decisions.
SRT_DEV float rng_next(uint32_t& s) {
    s = pcg_hash(s);
#ifdef SRT_RNG_DIVIDE
    return __fdiv_rn(__uint2float_rn(s), 4294967296.0f);
#else
    return __fmul_rn(__uint2float_rn(s), 2.3283064365386963e-10f);
#endif
}
// powf out of line: the shading kernels call it at several places, and its
// inlined copies were a large part of the code their warps wait for (config-2
// shading 1.40 -> 1.33 ms per frame, caustic slab 1.47 -> 1.43; blackbody4 or
// sincosf out of line too: 1.35, 1.37).
static __device__ __noinline__ float powf_call(float a, float b) { return powf(a, b); }
SRT_DEV float3 random_unit_vector(uint32_t& s) {
    float u1 = rng_next(s);
    float u2 = rng_next(s);
    float z = 1.0f - 2.0f * u1;
    float r = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    float phi = 2.0f * PI * u2;
    float sp, cp;
    sincosf(phi, &sp, &cp);
    return f3(r * cp, r * sp, z);
}

// ------------------------------------------------------------------ spectra
// sample_cie_xyz: shader.wgsl:85-97 (pow(x, 2.0) read as x*x)
SRT_DEV float3 sample_cie_xyz(float l) {
    float x = expf(-sq((l - 599.8f) / 37.9f)) * 1.056f + expf(-sq((l - 442.0f) / 16.0f)) * 0.362f -
              expf(-sq((l - 501.1f) / 26.7f)) * 0.065f;
    float y = expf(-sq((l - 568.8f) / 46.9f)) * 0.821f + expf(-sq((l - 530.9f) / 16.3f)) * 0.286f;
    float z = expf(-sq((l - 437.0f) / 11.8f)) * 1.217f + expf(-sq((l - 459.0f) / 26.0f)) * 0.681f;
    return f3(fmaxf(0.0f, x), fmaxf(0.0f, y), fmaxf(0.0f, z));
}
// XYZ_TO_SRGB: shader.wgsl:100-104
SRT_DEV float3 xyz_to_srgb(float3 c) {
    return f3(3.2404542f * c.x - 1.5371385f * c.y - 0.4985314f * c.z,
              -0.9692660f * c.x + 1.8760108f * c.y + 0.0415560f * c.z,
              0.0556434f * c.x - 0.2040259f * c.y + 1.0572252f * c.z);
}
// rgb_to_spectrum_eval: shader.wgsl:106-117, at the path's four wavelengths.  A
// channel that does not exceed the white part adds zeros (grey walls have
// three, red and green ones two): its exponentials are not evaluated.  One
// loop over the wavelengths (the tuple turned by one each time), like
// blackbody4's and thin_film4's below: the shading kernels' and above all the
// tail kernel's warps wait for instructions (a third of its stall cycles), and
// each of these bodies was there four times.  Tail kernel per frame with the
// three loops: config 1 0.140 -> 0.126 ms, caustic slab 0.225 -> 0.193, Cornell
// 0.197 -> 0.163, config 2 0.255 -> 0.231; the shading launches within 2 %.
SRT_DEV float4 rgb_to_spectrum4(float3 rgb, float4 wl) {
    const float white = fminf(rgb.x, fminf(rgb.y, rgb.z));
    const float cr = fmaxf(rgb.x - white, 0.f), cg = fmaxf(rgb.y - white, 0.f), cb = fmaxf(rgb.z - white, 0.f);
    float4 o = splat4(0.f);
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const float l = wl.x;
        wl = f4(wl.y, wl.z, wl.w, l);
        float r = 0.f, g = 0.f, b = 0.f;
        if (cr != 0.f) r = cr * expf(-sq((l - 630.0f) / 20.0f));
        if (cg != 0.f) g = cg * expf(-sq((l - 525.0f) / 20.0f));
        if (cb != 0.f) b = cb * expf(-sq((l - 460.0f) / 20.0f));
        o = f4(o.y, o.z, o.w, clampf(white + r + g + b, 0.0f, 0.99f));
    }
    return o;
}
// blackbody_radiance: shader.wgsl:128-139
SRT_DEV float blackbody(float lambda_nm, float temp_k) {
    float lm = lambda_nm * 1e-9f;
    const float h = 6.62607015e-34f, c = 299792458.0f, k = 1.380649e-23f;
    float c1 = 2.0f * h * c * c;
    float c2 = (h * c) / (k * temp_k);
    return c1 / (powf_call(lm, 5.0f) * (expf(c2 / lm) - 1.0f)) * 1e-13f;
}
SRT_DEV float4 blackbody4(float4 wl, float t) {
    float4 o = splat4(0.f);
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const float l = wl.x;
        wl = f4(wl.y, wl.z, wl.w, l);
        o = f4(o.y, o.z, o.w, blackbody(l, t));
    }
    return o;
}

// ------------------------------------------------------------------ BSDF math
// Airy reflectance of a film, one wavelength (photon_emit.wgsl:107-132;
// the vec4 form shader.wgsl:233-262 runs the same per component).
// Returns 1 and sets tir on total internal reflection.
SRT_DEV float thin_film1(float cos1, float n1, float n2, float n3, float d, float lambda, bool& tir) {
    float s1 = fmaxf(0.0f, 1.0f - cos1 * cos1);
    float s2 = (n1 / n2) * (n1 / n2) * s1;
    tir = true;
    if (s2 >= 1.0f) return 1.0f;
    float c2 = sqrtf(1.0f - s2);
    float s3 = (n1 / n3) * (n1 / n3) * s1;
    if (s3 >= 1.0f) return 1.0f;
    tir = false;
    float c3 = sqrtf(1.0f - s3);
    float r12 = (n1 * cos1 - n2 * c2) / (n1 * cos1 + n2 * c2);
    float r23 = (n2 * c2 - n3 * c3) / (n2 * c2 + n3 * c3);
    float a = r12 * r12, b = r23 * r23;
    float cd = cosf((4.0f * PI * n2 * d * c2) / lambda);
    float num = a + b + 2.0f * r12 * r23 * cd;
    float den = 1.0f + a * b + 2.0f * r12 * r23 * cd;
    return clampf(num / den, 0.0f, 1.0f);
}
SRT_DEV float4 thin_film4(float cos1, float n1, float n2, float n3, float d, float4 wl) {
    bool tir;  // total reflection does not depend on the wavelength: 1 for all four
    float4 o = splat4(0.f);
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const float l = wl.x;
        wl = f4(wl.y, wl.z, wl.w, l);
        o = f4(o.y, o.z, o.w, thin_film1(cos1, n1, n2, n3, d, l, tir));
    }
    return o;
}
// reflectance (Schlick): shader.wgsl:264-268
SRT_DEV float schlick(float cosine, float ri) {
    float r0 = (1.0f - ri) / (1.0f + ri);
    r0 = r0 * r0;
    return r0 + (1.0f - r0) * powf_call(1.0f - cosine, 5.0f);
}
SRT_DEV float g1_schlick_ggx(float nv, float r) {  // shader.wgsl:207-213
    float k = (r * r) / 2.0f;
    return nv / (nv * (1.0f - k) + k);
}
// GGX half vector in the frame of n (shader.wgsl:171-205; the basis keeps
// the reference's division by sign(n.z) + n.z).
SRT_DEV float3 ggx_half_vector(float3 n, float alpha, uint32_t& s) {
    float a2 = alpha * alpha;
    float r1 = rng_next(s);
    float r2 = rng_next(s);
    float phi = 2.0f * PI * r1;
    float ct = sqrtf((1.0f - r2) / (1.0f + (a2 - 1.0f) * r2));
    float st = sqrtf(fmaxf(0.0f, 1.0f - ct * ct));
    float sp, cp;
    sincosf(phi, &sp, &cp);
    float3 h = f3(cp * st, sp * st, ct);
    float sg = signf(n.z);
    float a = -1.0f / (sg + n.z);
    float b = n.x * n.y * a;
    float3 right = f3(1.0f + sg * n.x * n.x * a, sg * b, -sg * n.x);
    float3 up = f3(b, sg + n.y * n.y * a, -n.y);
    return normalize(right * h.x + up * h.y + n * h.z);
}

struct Scatter {
    float3 dir;
    float4 att;
    bool absorbed;
};

// sample_bsdf: shader.wgsl:347-471.  Type 5 (no reference counterpart):
// GGX sampling as type 1 with the film's Airy reflectance in place of
// Schlick's F; roughness in color.w, film d/n2/n3 in extra.yzw.
SRT_DEV Scatter sample_bsdf(float3 r_dir, float3 ffn, float4 color, float4 extra, bool front, float4 wl,
                            float4 thr, uint32_t& s) {
    Scatter rec;
    rec.absorbed = false;
    rec.dir = f3(0.f, 0.f, 0.f);
    rec.att = splat4(0.f);
    uint32_t type = (uint32_t)extra.x;
    float4 spec = rgb_to_spectrum4(xyz(color), wl);
    if (type == 1u || type == 5u) {
        float alpha = fmaxf(type == 1u ? extra.y : color.w, 0.001f);
        float3 v = normalize(-r_dir);
        float3 h = ggx_half_vector(ffn, alpha, s);
        float3 l = reflect(-v, h);
        float nl = dot(ffn, l), nv = dot(ffn, v);
        if (nl > 0.0f && nv > 0.0f) {
            float nh = fmaxf(dot(ffn, h), 0.0f);
            float vh = fmaxf(dot(v, h), 0.0f);
            float4 F;
            if (type == 1u) {
                float p = powf_call(clampf(1.0f - vh, 0.0f, 1.0f), 5.0f);
                F = spec + (splat4(1.0f) - spec) * p;
            } else {
                F = thin_film4(vh, 1.0f, extra.z, extra.w, fmaxf(extra.y, 50.0f), wl);
            }
            float G = g1_schlick_ggx(nl, alpha) * g1_schlick_ggx(nv, alpha);
            rec.att = (F * G * vh) / fmaxf(nv * nh, 0.0001f);
            rec.dir = l;
        } else {
            rec.absorbed = true;
        }
    } else if (type == 2u) {
        float lum = wl.x / 1000.0f;
        float ir = extra.z + (extra.w / (lum * lum));
        float ratio = front ? 1.0f / ir : ir;
        float3 u = normalize(r_dir);
        float ct = fminf(dot(-u, ffn), 1.0f);
        float si2 = fmaxf(0.0f, 1.0f - ct * ct);
        float st2 = ratio * ratio * si2;
        if (st2 >= 1.0f) {
            rec.dir = reflect(u, ffn);
            rec.att = splat4(1.0f);
        } else {
            float ctt = sqrtf(1.0f - st2);
            if (schlick(front ? ct : ctt, ratio) > rng_next(s)) {
                rec.dir = reflect(u, ffn);
                rec.att = splat4(1.0f);
            } else {
                rec.dir = refract(u, ffn, ratio);
                float4 base = spec * (ratio * ratio);
                if (extra.w > 0.0f) {
                    bool collapsed = thr.y < 0.0001f && thr.z < 0.0001f && thr.w < 0.0001f;
                    rec.att = f4(base.x * (collapsed ? 1.0f : 4.0f), 0.f, 0.f, 0.f);
                } else {
                    rec.att = base;
                }
            }
        }
    } else if (type == 4u) {
        float3 u = normalize(r_dir);
        float c1 = fminf(dot(-u, ffn), 1.0f);
        float4 F = thin_film4(c1, 1.0f, extra.z, extra.w, fmaxf(extra.y, 50.0f), wl);
        float p = F.x;
        if (rng_next(s) < p) {
            rec.dir = reflect(u, ffn);
            rec.att = F / p;
        } else {
            rec.dir = u;
            rec.att = (splat4(1.0f) - F) / (1.0f - p);
        }
    } else {
        float3 d = ffn + random_unit_vector(s);
        if (length(d) < 0.001f) d = ffn;
        rec.dir = normalize(d);
        rec.att = spec;
    }
    return rec;
}

// Hero wavelengths (shader.wgsl:734-767) and the sum of their pdfs (:782-797).
SRT_DEV float cauchy_cdf(float x) { return (1.0f / PI) * atanf((x - 555.0f) / 40.0f) + 0.5f; }
SRT_DEV float lambda_wrap(float x) {  // WGSL float %: e1 - e2 * trunc(e1 / e2)
    float a = x - LAMBDA_MIN;
    return LAMBDA_MIN + (a - LAMBDA_RANGE * truncf(a / LAMBDA_RANGE));
}
SRT_DEV float4 sample_hero(uint32_t& s) {
    float cmin = cauchy_cdf(LAMBDA_MIN), cmax = cauchy_cdf(LAMBDA_MAX);
    float u = cmin + rng_next(s) * (cmax - cmin);
    float hero = clampf(555.0f + 40.0f * tanf(PI * (u - 0.5f)), LAMBDA_MIN, LAMBDA_MAX);
    const float q = LAMBDA_RANGE / 4.0f;
    float4 w = f4(lambda_wrap(hero), lambda_wrap(hero + q), lambda_wrap(hero + q * 2.0f), lambda_wrap(hero + q * 3.0f));
    float rot = rng_next(s);
    if (rot < 0.25f) {
    } else if (rot < 0.5f) {
        w = f4(w.y, w.z, w.w, w.x);
    } else if (rot < 0.75f) {
        w = f4(w.z, w.w, w.x, w.y);
    } else {
        w = f4(w.w, w.x, w.y, w.z);
    }
    return w;
}
SRT_DEV float hero_pdf_sum(float4 w) {
    float cmin = cauchy_cdf(LAMBDA_MIN), cmax = cauchy_cdf(LAMBDA_MAX);
    float norm = 1.0f / ((cmax - cmin) * PI * 40.0f);
    float a = (w.x - 555.0f) / 40.0f, b = (w.y - 555.0f) / 40.0f, c = (w.z - 555.0f) / 40.0f,
          d = (w.w - 555.0f) / 40.0f;
    return norm / (1.0f + a * a) + norm / (1.0f + b * b) + norm / (1.0f + c * c) + norm / (1.0f + d * d);
}

// ------------------------------------------------------------------ photon grid hashing
// get_grid_jitter + hash_position: build_grid.wgsl:25-52.  Written with
// explicitly rounded intrinsics so that no multiply-add is contracted: the
// cell keys are compared bit for bit.
SRT_DEV float3 grid_jitter(uint32_t frame, float cell) {
    uint32_t seed = pcg_hash(frame * 114514u);
    float rx = __fdiv_rn(__uint2float_rn(seed & 0xFFu), 255.0f);
    float ry = __fdiv_rn(__uint2float_rn((seed >> 8u) & 0xFFu), 255.0f);
    float rz = __fdiv_rn(__uint2float_rn((seed >> 16u) & 0xFFu), 255.0f);
    return f3(__fmul_rn(__fsub_rn(rx, 0.5f), cell), __fmul_rn(__fsub_rn(ry, 0.5f), cell),
              __fmul_rn(__fsub_rn(rz, 0.5f), cell));
}
SRT_DEV uint32_t grid_hash(float3 p, float3 j, float cell, uint32_t hash_bits) {
    // f32 -> i32 conversion saturates as in WGSL (cvt.rzi.s32.f32 does)
    int gx = __float2int_rz(floorf(__fdiv_rn(__fadd_rn(p.x, j.x), cell)));
    int gy = __float2int_rz(floorf(__fdiv_rn(__fadd_rn(p.y, j.y), cell)));
    int gz = __float2int_rz(floorf(__fdiv_rn(__fadd_rn(p.z, j.z), cell)));
    uint32_t h = ((uint32_t)gx * 73856093u) ^ ((uint32_t)gy * 19349663u) ^ ((uint32_t)gz * 83492791u);
    return h & ((1u << hash_bits) - 1u);
}

// ------------------------------------------------------------------ camera ray (shader.wgsl:713-728)
// Element (r, c) of view_inv * proj_inv.
SRT_DEV float camera_elem(const srt_camera_uniform& cam, uint32_t r, uint32_t c) {
    const float* vi = cam.view_inverse;
    const float* pi = cam.proj_inverse;
    return vi[r] * pi[4u * c] + vi[4u + r] * pi[4u * c + 1u] + vi[8u + r] * pi[4u * c + 2u] +
           vi[12u + r] * pi[4u * c + 3u];
}
// m: camera_elem(r, c) at m[4 r + c].
SRT_DEV void camera_ray(const srt_camera_uniform& cam, const float* m, uint32_t x, uint32_t y, uint32_t w, uint32_t h,
                        uint32_t& s, float3& o, float3& d) {
    const float* vi = cam.view_inverse;
    float jx = rng_next(s);
    float jy = rng_next(s);
    float nx = ((float)x + jx) / (float)w * 2.0f - 1.0f;
    float ny = ((float)y + jy) / (float)h * 2.0f - 1.0f;
    float t[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) t[r] = m[4 * r] * nx + m[4 * r + 1] * ny + m[4 * r + 2] + m[4 * r + 3];
    o = f3(vi[12], vi[13], vi[14]);
    d = normalize(f3(t[0] / t[3], t[1] / t[3], t[2] / t[3]) - o);
}

// ------------------------------------------------------------------ traversal
struct Ray {
    float3 o, d;
    float tmin, tmax;
};

// Watertight ray/triangle test (Woop, Benthin, Wald, JCGT 2013) with the
// FP64 fallback for edge functions that evaluate to exactly zero.
struct RayShear {
    int kx, ky, kz;
    float sx, sy, sz;
};
SRT_DEV float comp(float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }
SRT_DEV RayShear make_shear(float3 d) {
    RayShear r;
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    r.kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    r.kx = r.kz == 2 ? 0 : r.kz + 1;
    r.ky = r.kx == 2 ? 0 : r.kx + 1;
    float dz = comp(d, r.kz);
    if (dz < 0.0f) {
        int t = r.kx;
        r.kx = r.ky;
        r.ky = t;
    }
    r.sx = comp(d, r.kx) / dz;
    r.sy = comp(d, r.ky) / dz;
    r.sz = 1.0f / dz;
    return r;
}
SRT_DEV float comp_i(float3 v, uint32_t k) { return k == 0u ? v.x : (k == 1u ? v.y : v.z); }
// The watertight test on vertices v0, v1, v2 for a ray from o sheared by
// (kx, ky, kz, sx, sy, sz).  Every rounding is written out (explicit fused
// multiply-adds and products), so the test gives the same bits in every
// translation unit whatever its contraction setting.  Returns true on a hit
// with tmin <= t <= tmax; u, v = weights of v1, v2.
SRT_DEV bool tri_test(float3 v0, float3 v1, float3 v2, float3 o, uint32_t kx, uint32_t ky, uint32_t kz, float sx,
                      float sy, float sz, float tmin, float tmax, float& t, float& u, float& v) {
    const float3 A = v0 - o, B = v1 - o, C = v2 - o;
    const float Az = comp_i(A, kz), Bz = comp_i(B, kz), Cz = comp_i(C, kz);
    const float Ax = fmaf(-sx, Az, comp_i(A, kx)), Ay = fmaf(-sy, Az, comp_i(A, ky));
    const float Bx = fmaf(-sx, Bz, comp_i(B, kx)), By = fmaf(-sy, Bz, comp_i(B, ky));
    const float Cx = fmaf(-sx, Cz, comp_i(C, kx)), Cy = fmaf(-sy, Cz, comp_i(C, ky));
    float U = fmaf(Cx, By, -__fmul_rn(Cy, Bx));
    float V = fmaf(Ax, Cy, -__fmul_rn(Ay, Cx));
    float W = fmaf(Bx, Ay, -__fmul_rn(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {  // FP64 fallback: exact products
        U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
        V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
        W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    const float inv = __frcp_rn(det);
    const float T = fmaf(W, __fmul_rn(sz, Cz), fmaf(V, __fmul_rn(sz, Bz), __fmul_rn(U, __fmul_rn(sz, Az))));
    const float tt = __fmul_rn(T, inv);
    if (!(tt >= tmin && tt <= tmax)) return false;
    t = tt;
    u = __fmul_rn(V, inv);
    v = __fmul_rn(W, inv);
    return true;
}
SRT_DEV bool intersect_tri(const Ray& ray, const RayShear& sh, float3 v0, float3 v1, float3 v2, float& t, float& u,
                           float& v) {
    return tri_test(v0, v1, v2, ray.o, (uint32_t)sh.kx, (uint32_t)sh.ky, (uint32_t)sh.kz, sh.sx, sh.sy, sh.sz,
                    ray.tmin, ray.tmax, t, u, v);
}

SRT_DEV uint32_t byte_of(uint32_t w, int i) { return (w >> (8 * i)) & 0xFFu; }
// A byte b as a float without the integer-to-float conversion unit is the bit
// pattern 0x4B0000bb (= 2^23 + b exactly).  The group's slab test (group_step)
// folds the 2^23 bias into its addend, t = fma(2^23 + q, a, b - 2^23 a), whose
// rounding moves a plane by at most half a quantum (node_hits' 1024: 2^-14 of
// one); the builder pads every child box by one quantum.
SRT_DEV float unbias(float a, float b) { return fmaf(-8388608.0f, a, b); }

// Two fused multiply-adds: one packed fma.rn.f32x2 with SRT_TRAV_FMA2 (the
// slab test of a child computes its near and far plane of an axis at once;
// measured 1.3 % off a config-2 frame), two scalar ones otherwise.  Both
// round each lane once, like fmaf.
#ifndef SRT_TRAV_FMA2
#define SRT_TRAV_FMA2 1
#endif
SRT_DEV float2 fma2(float2 a, float2 b, float2 c) {
#if SRT_TRAV_FMA2
    uint64_t x, y, z, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(z) : "f"(c.x), "f"(c.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
#else
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#endif
}

struct TravCounters {
    unsigned long long* nodes;
    unsigned long long* tris;
};

// Bytes 2p and 2p + 1 of w, each plus 1024, as floats (exact): one byte permute
// builds the half pair 0x64bb64bb, and its two conversions run beside the fused
// multiply-adds; the permutes share a half-rate unit with the minima and maxima.
SRT_DEV float2 qpair(uint32_t w, uint32_t p) {
    const uint32_t h = __byte_perm(w, 0x64646464u, p ? 0x4342u : 0x4140u);
    return __half22float2(*reinterpret_cast<const __half2*>(&h));
}

// Child slab tests of one node (words w0..w4) for a ray with inverse
// direction idir and octant oct: the slots whose box the ray meets within
// [tmin, tbest].  A slot without a child may be among them: it has no imask bit
// and no triangles.  (With a test per slot for a child, a compare and a select
// for the bit, and a byte permute per plane: closest hits 3.25 vs 3.17 ms per
// config-2 frame, shadow rays 1.88 vs 1.82.)
SRT_DEV uint32_t node_hits(uint4 w0, uint4 w1, uint4 w2, uint4 w3, uint4 w4, float3 o, float3 idir, uint32_t oct,
                           float tmin, float tbest) {
    float sx = __uint_as_float((w0.w & 0xFFu) << 23), sy = __uint_as_float(((w0.w >> 8) & 0xFFu) << 23),
          sz = __uint_as_float(((w0.w >> 16) & 0xFFu) << 23);
    float ax = sx * idir.x, ay = sy * idir.y, az = sz * idir.z;
    float bx = fmaf(-1024.0f, ax, (__uint_as_float(w0.x) - o.x) * idir.x),
          by = fmaf(-1024.0f, ay, (__uint_as_float(w0.y) - o.y) * idir.y),
          bz = fmaf(-1024.0f, az, (__uint_as_float(w0.z) - o.z) * idir.z);
    uint32_t nx0 = (oct & 1u) ? w3.z : w2.x, nx1 = (oct & 1u) ? w3.w : w2.y;
    uint32_t fx0 = (oct & 1u) ? w2.x : w3.z, fx1 = (oct & 1u) ? w2.y : w3.w;
    uint32_t ny0 = (oct & 2u) ? w4.x : w2.z, ny1 = (oct & 2u) ? w4.y : w2.w;
    uint32_t fy0 = (oct & 2u) ? w2.z : w4.x, fy1 = (oct & 2u) ? w2.w : w4.y;
    uint32_t nz0 = (oct & 4u) ? w4.z : w3.x, nz1 = (oct & 4u) ? w4.w : w3.y;
    uint32_t fz0 = (oct & 4u) ? w3.x : w4.z, fz1 = (oct & 4u) ? w3.y : w4.w;
    const float robust = 1.0000004f;
    uint32_t miss = 0u;
#pragma unroll
    for (int j = 3; j >= 0; --j) {  // children 2j and 2j + 1
        const uint32_t p = (uint32_t)(j & 1);
        const float2 qnx = qpair(j < 2 ? nx0 : nx1, p), qfx = qpair(j < 2 ? fx0 : fx1, p),
                     qny = qpair(j < 2 ? ny0 : ny1, p), qfy = qpair(j < 2 ? fy0 : fy1, p),
                     qnz = qpair(j < 2 ? nz0 : nz1, p), qfz = qpair(j < 2 ? fz0 : fz1, p);
#pragma unroll
        for (int e = 1; e >= 0; --e) {
            const float2 tx = fma2(make_float2(e ? qnx.y : qnx.x, e ? qfx.y : qfx.x), make_float2(ax, ax),
                                   make_float2(bx, bx));
            const float2 ty = fma2(make_float2(e ? qny.y : qny.x, e ? qfy.y : qfy.x), make_float2(ay, ay),
                                   make_float2(by, by));
            const float2 tz = fma2(make_float2(e ? qnz.y : qnz.x, e ? qfz.y : qfz.x), make_float2(az, az),
                                   make_float2(bz, bz));
            const float tn = fmaxf(fmaxf(tx.x, ty.x), fmaxf(tz.x, tmin));
            const float tf = fminf(fminf(tx.y, ty.y), fminf(tz.y, tbest));
            // the sign of tf * robust - tn shifted in: missed where it is negative
            miss = __funnelshift_l(__float_as_uint(fmaf(tf, robust, -tn)), miss, 1);
        }
    }
    return ~miss & 0xFFu;
}

// One node visit: the node's hit internal children (bits 24..31, ordered by
// octant) | imask, and its hit triangle bits.  The child loop (node_hits) only
// collects which slots are hit; the octant order of the internal children and
// the leaves' triangle bits follow once per node (config-2 closest-hit 3.35
// vs 3.43 ms per frame with both per child).
SRT_DEV void node_children(uint4 w0, uint4 w1, uint4 w2, uint4 w3, uint4 w4, float3 o, float3 idir, uint32_t oct,
                           float tmin, float tbest, uint2& g, uint2& tg) {
    const uint32_t imask = w0.w >> 24;
    const uint32_t hitmask = node_hits(w0, w1, w2, w3, w4, o, idir, oct, tmin, tbest);
    // internal children: slot i -> bit i ^ (oct ^ 7) (three conditional swaps)
    uint32_t ib = hitmask & imask;
    const uint32_t x = oct ^ 7u;
    ib = (x & 1u) ? (((ib & 0x55u) << 1) | ((ib >> 1) & 0x55u)) : ib;
    ib = (x & 2u) ? (((ib & 0x33u) << 2) | ((ib >> 2) & 0x33u)) : ib;
    ib = (x & 4u) ? (((ib & 0x0Fu) << 4) | ((ib >> 4) & 0x0Fu)) : ib;
    // leaves: their triangles' bits
    uint32_t lb = hitmask & ~imask, tris = 0u;
    while (lb != 0u) {
        const uint32_t i = (uint32_t)(__ffs(lb) - 1);
        lb &= lb - 1u;
        const uint32_t m = ((i < 4u ? w1.z : w1.w) >> (8u * (i & 3u))) & 0xFFu;
        tris |= ((1u << (m >> 5)) - 1u) << (m & 31u);
    }
    g = make_uint2(w1.x, (ib << 24) | imask);
    tg = make_uint2(w1.y, tris);
}

// Materials a photon path goes on from: types 1, 2, 4 and 5.  At any other
// surface a path ends, and its first surface stores nothing either (only
// diffuse surfaces reached after a refraction or a film store photons).
SRT_DEV bool scatters_photons(float4 extra) {
    const uint32_t type = (uint32_t)extra.x;
    return type == 1u || type == 2u || type == 4u || type == 5u;
}

// Walk of a ray over the subtrees that hold scattering triangles (S.scatter),
// one node per step, to the first leaf box of theirs that it meets.
// Conservative: the closest-hit traversal reaches a triangle through boxes that
// pass the same slab test with a t_max no larger than `tmax`, so a ray that
// meets no such leaf has no scattering triangle as its closest hit.
struct ScatterWalk {
    float3 o, idir;
    uint32_t oct;
    uint2 g;  // child base; child slots left (bits 8..15) | imask
    int sp;
};
constexpr int WALK_ON = 0, WALK_MAY_SCATTER = 1, WALK_DONE = 2;

// False: the ray cannot hit anything.
SRT_DEV bool scatter_init(ScatterWalk& W, const DevScene& S, float3 o, float3 d) {
    W.o = o;
    const float eps = 1e-12f;
    W.idir = f3(1.0f / (fabsf(d.x) > eps ? d.x : copysignf(eps, d.x)),
                1.0f / (fabsf(d.y) > eps ? d.y : copysignf(eps, d.y)),
                1.0f / (fabsf(d.z) > eps ? d.z : copysignf(eps, d.z)));
    W.oct = (d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u);
    W.g = make_uint2(0u, 0x101u);  // the root as child slot 0
    W.sp = 0;
    return S.n_nodes != 0u && (d.x != 0.0f || d.y != 0.0f || d.z != 0.0f);
}
// `stack`: STACK entries of this thread, stride `stride` (one entry per level at most).
template <int STACK>
SRT_DEV int scatter_step(const DevScene& S, ScatterWalk& W, float tmin, float tmax, uint2* stack, int stride,
                         uint32_t* err) {
    if ((W.g.y & 0xFF00u) == 0u) {
        if (W.sp == 0) return WALK_DONE;
        --W.sp;
        W.g = stack[W.sp * stride];
    }
    const uint32_t slot = (uint32_t)__ffs(W.g.y >> 8) - 1u;
    W.g.y &= ~(0x100u << slot);
    const uint32_t idx = W.g.x + __popc(W.g.y & ((1u << slot) - 1u) & 0xFFu);
    if (W.g.y & 0xFF00u) {
        if (W.sp >= STACK) {
            atomicOr(err, ERR_STACK_OVERFLOW);
            return WALK_DONE;
        }
        stack[W.sp * stride] = W.g;
        ++W.sp;
    }
    if (idx >= S.n_nodes) {
        atomicOr(err, ERR_BAD_INDEX);
        return WALK_DONE;
    }
    const uint32_t scatter = __ldg(S.scatter + idx);
    const uint4* np = reinterpret_cast<const uint4*>(S.nodes + idx);
    const uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    const uint32_t hits = node_hits(w0, w1, w2, w3, w4, W.o, W.idir, W.oct, tmin, tmax) & scatter;
    const uint32_t imask = w0.w >> 24;
    if (hits & ~imask) return WALK_MAY_SCATTER;
    W.g = make_uint2(w1.x, (hits << 8) | imask);
    return WALK_ON;
}

// Stack-based traversal of the compressed BVH8.  A node group holds the
// hit internal children of one node (bits 24..31 of .y, ordered so that the
// highest bit is the nearest child for this ray octant) plus the node's
// imask (bits 0..7); triangle hits go straight to the triangle loop.
// ANY: return at the first hit in [tmin, tmax].  Closest: lexicographic
// minimum of (t, flattened triangle id), independent of traversal order.
// `stack` is this thread's slice of shared memory, stride `stride` entries,
// STACK entries deep (at least the tree depth: one entry per level).
template <bool ANY, bool COUNT, int STACK = TRAV_STACK>
SRT_DEV bool traverse(const DevScene& S, Ray ray, uint2* stack, int stride, float& t_out, uint32_t& prim_out,
                      float& u_out, float& v_out, uint32_t* err, TravCounters cnt) {
    prim_out = MISS;
    if (S.n_nodes == 0u) return false;
    if (!(ray.d.x != 0.0f || ray.d.y != 0.0f || ray.d.z != 0.0f)) return false;
    if (!(ray.tmin <= ray.tmax)) return false;
    RayShear sh = make_shear(ray.d);
    const float eps = 1e-12f;
    float3 idir = f3(1.0f / (fabsf(ray.d.x) > eps ? ray.d.x : copysignf(eps, ray.d.x)),
                     1.0f / (fabsf(ray.d.y) > eps ? ray.d.y : copysignf(eps, ray.d.y)),
                     1.0f / (fabsf(ray.d.z) > eps ? ray.d.z : copysignf(eps, ray.d.z)));
    uint32_t oct = (ray.d.x < 0.f ? 1u : 0u) | (ray.d.y < 0.f ? 2u : 0u) | (ray.d.z < 0.f ? 4u : 0u);
    float tbest = ray.tmax;
    uint32_t best = MISS;
    float bu = 0.f, bv = 0.f;
    int sp = 0;
    uint32_t n_nodes = 0, n_tris = 0;
    // virtual group holding the root as child slot 0
    uint2 g = make_uint2(0u, (1u << (24 + (0u ^ (oct ^ 7u)))) | 1u);
    uint2 tg = make_uint2(0u, 0u);
    while (true) {
        // ---- triangles of the last node
        while (tg.y != 0u) {
            int b = __ffs(tg.y) - 1;
            tg.y &= tg.y - 1u;
            const TriSlot* ts = S.tris + tg.x + (uint32_t)b;
            float4 a0 = __ldg(&ts->v0), a1 = __ldg(&ts->v1), a2 = __ldg(&ts->v2);
            if (COUNT) ++n_tris;
            float t, u, v;
            Ray r = ray;
            r.tmax = tbest;
            if (intersect_tri(r, sh, xyz(a0), xyz(a1), xyz(a2), t, u, v)) {
                uint32_t id = __float_as_uint(a0.w);
                if (ANY) {
                    t_out = t;
                    prim_out = id;
                    if (COUNT) {
                        atomicAdd(cnt.nodes, (unsigned long long)n_nodes);
                        atomicAdd(cnt.tris, (unsigned long long)n_tris);
                    }
                    return true;
                }
                if (t < tbest || id < best) {  // (t, id) lexicographic; t <= tbest holds here
                    if (t < tbest || (t == tbest && id < best)) {
                        tbest = t;
                        best = id;
                        bu = u;
                        bv = v;
                    }
                }
            }
        }
        // ---- next node
        if ((g.y & 0xFF000000u) == 0u) {
            if (sp == 0) break;
            --sp;
            g = stack[sp * stride];
        }
        int bit = 31 - __clz(g.y & 0xFF000000u);
        g.y &= ~(1u << bit);
        uint32_t slot = (uint32_t)(bit - 24) ^ (oct ^ 7u);
        uint32_t idx = g.x + __popc(g.y & ((1u << slot) - 1u) & 0xFFu);
        if (g.y & 0xFF000000u) {
            if (sp >= STACK) {
                atomicOr(err, ERR_STACK_OVERFLOW);
                break;
            }
            stack[sp * stride] = g;
            ++sp;
        }
        if (idx >= S.n_nodes) {
            atomicOr(err, ERR_BAD_INDEX);
            break;
        }
        const uint4* np = reinterpret_cast<const uint4*>(S.nodes + idx);
        uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
        if (COUNT) ++n_nodes;
        node_children(w0, w1, w2, w3, w4, ray.o, idir, oct, ray.tmin, tbest, g, tg);
    }
    if (COUNT) {
        atomicAdd(cnt.nodes, (unsigned long long)n_nodes);
        atomicAdd(cnt.tris, (unsigned long long)n_tris);
    }
    if (ANY) return false;
    if (best == MISS) return false;
    t_out = tbest;
    prim_out = best;
    u_out = bu;
    v_out = bv;
    return true;
}

// ------------------------------------------------------------------ resumable traversal
// The same traversal as traverse<>, split into an init and a step so that a
// persistent warp can hand a finished lane a new ray between steps.  One
// step = the pending triangle tests of the warp's last node visits (pool_tris)
// + one node visit per lane (trav_step).
struct TravState {
    float3 o, idir;
    float tmin, tbest;
    float sx, sy, sz;
    uint32_t axes;  // kx | ky << 2 | kz << 4 | oct << 8
    uint2 g, tg;
    int sp;
    uint32_t best;
    float bu, bv;
};

// Returns false when the ray cannot hit anything (finished at once).
SRT_DEV bool trav_init(TravState& T, const DevScene& S, float3 o, float3 d, float tmin, float tmax) {
    T.best = MISS;
    T.tbest = tmax;
    T.tmin = tmin;
    T.sp = 0;
    T.tg = make_uint2(0u, 0u);
    T.g = make_uint2(0u, 0u);
    T.bu = T.bv = 0.f;
    T.o = o;
    if (S.n_nodes == 0u || !(d.x != 0.0f || d.y != 0.0f || d.z != 0.0f) || !(tmin <= tmax)) return false;
    RayShear sh = make_shear(d);
    T.sx = sh.sx;
    T.sy = sh.sy;
    T.sz = sh.sz;
    const float eps = 1e-12f;
    T.idir = f3(1.0f / (fabsf(d.x) > eps ? d.x : copysignf(eps, d.x)),
                1.0f / (fabsf(d.y) > eps ? d.y : copysignf(eps, d.y)),
                1.0f / (fabsf(d.z) > eps ? d.z : copysignf(eps, d.z)));
    uint32_t oct = (d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u);
    T.axes = (uint32_t)sh.kx | ((uint32_t)sh.ky << 2) | ((uint32_t)sh.kz << 4) | (oct << 8);
    T.g = make_uint2(0u, (1u << (24 + (0u ^ (oct ^ 7u)))) | 1u);
    return true;
}

// Pooled triangle tests, called by all 32 lanes of a warp
// at once: the triangles pending at the lanes' last node visits (T.tg of the
// lanes with `live` set) are numbered across the warp by a prefix sum and
// dealt out one per lane per round, so a round tests up to 32 triangles
// whatever lanes they belong to (idle lanes work too), instead of each lane
// looping over its own with the others waiting.  The owners list a round's
// tasks in `tasks` (32 words of shared memory per warp); a lane fetches its
// task's ray from the owner (shuffles) and tests it with the same tri_test; the
// owner then reads the hits of its tasks (consecutive lanes of a ballot) and
// keeps the lexicographic minimum of (t, id).  The closest hit does not depend
// on the order of the tests, so results are unchanged; any-hit rays stop at
// their first hit (T.best != MISS afterwards).  Leaves T.tg empty.
// Looping over its own triangles kept 4.45 of 32 lanes busy on bounce 1 of
// config 2; with pooled tests in both forms and 8 blocks per SM (lists instead
// of a search and an __fns per task, hits read from the ballot instead of a
// segmented minimum): closest hits 3.13 -> 2.99 ms and shadow rays 1.83 -> 1.79
// ms per config-2 frame, Cornell 640x480 0.68 -> 0.68 and 0.41 -> 0.40, a seeded
// scene of 812k triangles 0.97 -> 0.94 and 0.52 -> 0.53, caustic slab 1.30 -> 1.34
// and 0.77 -> 0.76 (its nodes hold few triangles; testing one per lane directly
// where no lane has more: 1.35).
// MULTI: the lanes trace rays of different scenes (the batched renderer's
// persistent launch), so a task reads the triangles of its owner's scene.
template <bool ANY, bool MULTI = false>
SRT_DEV void pool_tris(const DevScene& S, TravState& T, bool live, uint32_t* tasks, uint32_t& n_tris) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t bits = live ? T.tg.y : 0u;
    if (!__any_sync(FULL, bits != 0u)) return;
    const uint32_t cnt = (uint32_t)__popc(bits);
    uint32_t incl = cnt;
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += v;
    }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    const uint32_t excl = incl - cnt;
    uint32_t pos = excl;
    for (uint32_t base = 0; base < total; base += 32u) {
        while (bits != 0u && pos < base + 32u) {
            tasks[pos - base] = lane | ((uint32_t)(__ffs(bits) - 1) << 8);
            bits &= bits - 1u;
            ++pos;
        }
        __syncwarp();
        const bool have = base + lane < total;
        const uint32_t task = have ? tasks[lane] : lane;
        __syncwarp();  // the next round's tasks go into the same words
        const int o = (int)(task & 31u);
        const uint32_t gx = __shfl_sync(FULL, T.tg.x, o);
        const float ox = __shfl_sync(FULL, T.o.x, o), oy = __shfl_sync(FULL, T.o.y, o), oz = __shfl_sync(FULL, T.o.z, o);
        const float sx = __shfl_sync(FULL, T.sx, o), sy = __shfl_sync(FULL, T.sy, o), sz = __shfl_sync(FULL, T.sz, o);
        const float tmin = __shfl_sync(FULL, T.tmin, o), tmax = __shfl_sync(FULL, T.tbest, o);
        const uint32_t axes = __shfl_sync(FULL, T.axes, o);
        const TriSlot* tris = S.tris;
        if (MULTI)
            tris = reinterpret_cast<const TriSlot*>(
                __shfl_sync(FULL, reinterpret_cast<unsigned long long>(S.tris), o));
        bool hit = false;
        float t = 0.f, u = 0.f, v = 0.f;
        uint32_t id = 0u;
        if (have) {
            const TriSlot* ts = tris + gx + (task >> 8);
            const float4 a0 = __ldg(&ts->v0), a1 = __ldg(&ts->v1), a2 = __ldg(&ts->v2);
            ++n_tris;
            id = __float_as_uint(a0.w);
            hit = tri_test(xyz(a0), xyz(a1), xyz(a2), f3(ox, oy, oz), axes & 3u, (axes >> 2) & 3u, (axes >> 4) & 3u, sx,
                           sy, sz, tmin, tmax, t, u, v);
        }
        // the hits of this lane's tasks: lanes [lo, hi) of the round
        uint32_t hits = __ballot_sync(FULL, hit);
        if (hits == 0u) continue;
        const uint32_t lo = max(excl, base) - base, hi = min(incl, base + 32u) - base;
        if (cnt == 0u || incl <= base || excl >= base + 32u) hits = 0u;
        else hits &= (hi - lo >= 32u ? FULL : ((1u << (hi - lo)) - 1u)) << lo;
        if (ANY) {
            if (hits != 0u) T.best = 0u;
            continue;
        }
        while (__any_sync(FULL, hits != 0u)) {
            const int src = hits != 0u ? __ffs(hits) - 1 : (int)lane;
            const float ht = __shfl_sync(FULL, t, src), hu = __shfl_sync(FULL, u, src), hv = __shfl_sync(FULL, v, src);
            const uint32_t hid = __shfl_sync(FULL, id, src);
            if (hits != 0u && (ht < T.tbest || (ht == T.tbest && hid < T.best))) {
                T.tbest = ht;
                T.best = hid;
                T.bu = hu;
                T.bv = hv;
            }
            hits &= hits - 1u;
        }
    }
    if (live) T.tg.y = 0u;
}

// One node visit of this lane's ray, after pool_tris; true when the ray is
// finished.
template <int STACK>
SRT_DEV bool trav_step(const DevScene& S, TravState& T, uint2* stack, int stride, uint32_t* err, uint32_t& n_nodes) {
    const uint32_t oct = (T.axes >> 8) & 7u;
    if ((T.g.y & 0xFF000000u) == 0u) {
        if (T.sp == 0) return true;
        --T.sp;
        T.g = stack[T.sp * stride];
    }
    const int bit = 31 - __clz(T.g.y & 0xFF000000u);
    T.g.y &= ~(1u << bit);
    const uint32_t slot = (uint32_t)(bit - 24) ^ (oct ^ 7u);
    const uint32_t idx = T.g.x + __popc(T.g.y & ((1u << slot) - 1u) & 0xFFu);
    if (T.g.y & 0xFF000000u) {
        if (T.sp >= STACK) {
            atomicOr(err, ERR_STACK_OVERFLOW);
            return true;
        }
        stack[T.sp * stride] = T.g;
        ++T.sp;
    }
    if (idx >= S.n_nodes) {
        atomicOr(err, ERR_BAD_INDEX);
        return true;
    }
    const uint4* np = reinterpret_cast<const uint4*>(S.nodes + idx);
    const uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    ++n_nodes;
    node_children(w0, w1, w2, w3, w4, T.o, T.idir, oct, T.tmin, T.tbest, T.g, T.tg);
    return false;
}

// ------------------------------------------------------------------ one ray on eight lanes
// The same traversal with a ray on a group of 8 lanes (4 rays per warp): lane
// c of the group tests child c of a node and the triangles of that child's
// leaf, so a node visit is one slab test deep instead of eight and a node's
// leaves are tested at once.  Per ray it issues about as many warp
// instructions as the one-lane form at its usual occupancy of lanes, but the
// chain of a single ray is several times shorter, and rays of a warp do not
// diverge (the groups step together).  It serves the launches that last as
// long as their longest rays: few rays (k_trace_pt) and the tail.
// Every function here is called by all 32 lanes of a warp at once.
constexpr uint32_t GROUP = 8;
constexpr uint32_t GROUP_LEADERS = 0x01010101u;  // lane 0 of each group

template <int STACK>
struct GroupTrav {
    float3 o, idir;
    float tmin, tbest;  // tbest: the group's closest t so far
    float sx, sy, sz;
    uint32_t axes;      // kx | ky << 2 | kz << 4 | oct << 8
    uint2 g;
    uint2 st[STACK / 8];  // the group's stack: entry e in slot e / 8 of lane e % 8
    int sp;
    float t, u, v;      // this lane's closest hit
    uint32_t id;        // MISS: none
};

// Returns false when the ray cannot hit anything.  The same values in all
// lanes of a group.
template <int STACK>
SRT_DEV bool group_init(GroupTrav<STACK>& T, const DevScene& S, float3 o, float3 d, float tmin, float tmax) {
    T.id = MISS;
    T.t = __int_as_float(0x7F800000);
    T.u = T.v = 0.f;
    T.tbest = tmax;
    T.tmin = tmin;
    T.sp = 0;
    T.o = o;
    T.g = make_uint2(0u, 0u);
    if (S.n_nodes == 0u || !(d.x != 0.0f || d.y != 0.0f || d.z != 0.0f) || !(tmin <= tmax)) return false;
    const RayShear sh = make_shear(d);
    T.sx = sh.sx;
    T.sy = sh.sy;
    T.sz = sh.sz;
    const float eps = 1e-12f;
    T.idir = f3(1.0f / (fabsf(d.x) > eps ? d.x : copysignf(eps, d.x)),
                1.0f / (fabsf(d.y) > eps ? d.y : copysignf(eps, d.y)),
                1.0f / (fabsf(d.z) > eps ? d.z : copysignf(eps, d.z)));
    const uint32_t oct = (d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u);
    T.axes = (uint32_t)sh.kx | ((uint32_t)sh.ky << 2) | ((uint32_t)sh.kz << 4) | (oct << 8);
    T.g = make_uint2(0u, (1u << (24 + (0u ^ (oct ^ 7u)))) | 1u);
    return true;
}

// One node visit and its triangles for the groups with `active` set; true
// when the group's ray is finished (`any`, the same in the warp: at its first hit).
template <int STACK>
SRT_DEV bool group_step(const DevScene& S, GroupTrav<STACK>& T, bool active, bool any, uint32_t* err, uint32_t& n_nodes,
                        uint32_t& n_tris) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, c = lane & 7u, shift = lane & 24u;
    const uint32_t oct = (T.axes >> 8) & 7u;
    bool fin = false;
    const bool empty = active && (T.g.y & 0xFF000000u) == 0u;
    if (__any_sync(FULL, empty)) {
        const int top = T.sp - 1;
        uint2 e = T.st[0];
#pragma unroll
        for (int k = 1; k < STACK / 8; ++k)
            if ((top >> 3) == k) e = T.st[k];
        const uint32_t px = __shfl_sync(FULL, e.x, (int)(shift | ((uint32_t)top & 7u)));
        const uint32_t py = __shfl_sync(FULL, e.y, (int)(shift | ((uint32_t)top & 7u)));
        if (empty) {
            if (top < 0) fin = true;
            else {
                T.g = make_uint2(px, py);
                T.sp = top;
            }
        }
    }
    bool go = active && !fin;
    bool hit = false;
    uint32_t cnt = 0u, first = 0u, imask = 0u, child = 0u;
    if (go) {
        const int bit = 31 - __clz(T.g.y & 0xFF000000u);
        T.g.y &= ~(1u << bit);
        const uint32_t slot = (uint32_t)(bit - 24) ^ (oct ^ 7u);
        const uint32_t idx = T.g.x + __popc(T.g.y & ((1u << slot) - 1u) & 0xFFu);
        if (T.g.y & 0xFF000000u) {
            if (T.sp >= STACK) {
                atomicOr(err, ERR_STACK_OVERFLOW);
                go = false;
            } else {
#pragma unroll
                for (int k = 0; k < STACK / 8; ++k)
                    if (T.sp == (int)(8u * k + c)) T.st[k] = T.g;
                ++T.sp;
            }
        }
        if (go && idx >= S.n_nodes) {
            atomicOr(err, ERR_BAD_INDEX);
            go = false;
        }
        if (go) {
            // header by every lane (one broadcast), child c's bytes by lane c
            const uint8_t* nb = reinterpret_cast<const uint8_t*>(S.nodes + idx);
            const uint4 w0 = __ldg(reinterpret_cast<const uint4*>(nb));
            const uint2 w1 = __ldg(reinterpret_cast<const uint2*>(nb + 16));
            const uint32_t m = __ldg(nb + 24 + c);
            const uint32_t lx = __ldg(nb + 32 + c), ly = __ldg(nb + 40 + c), lz = __ldg(nb + 48 + c);
            const uint32_t hx = __ldg(nb + 56 + c), hy = __ldg(nb + 64 + c), hz = __ldg(nb + 72 + c);
            if (c == 0u) ++n_nodes;
            const float ax = __uint_as_float((w0.w & 0xFFu) << 23) * T.idir.x,
                        ay = __uint_as_float(((w0.w >> 8) & 0xFFu) << 23) * T.idir.y,
                        az = __uint_as_float(((w0.w >> 16) & 0xFFu) << 23) * T.idir.z;
            const float bx = unbias(ax, (__uint_as_float(w0.x) - T.o.x) * T.idir.x),
                        by = unbias(ay, (__uint_as_float(w0.y) - T.o.y) * T.idir.y),
                        bz = unbias(az, (__uint_as_float(w0.z) - T.o.z) * T.idir.z);
            // the slab test of node_hits for one child: 2^23 + byte as a float
            const uint32_t B = 0x4B000000u;
            const float nx = fmaf(__uint_as_float(B | ((oct & 1u) ? hx : lx)), ax, bx),
                        fx = fmaf(__uint_as_float(B | ((oct & 1u) ? lx : hx)), ax, bx),
                        ny = fmaf(__uint_as_float(B | ((oct & 2u) ? hy : ly)), ay, by),
                        fy = fmaf(__uint_as_float(B | ((oct & 2u) ? ly : hy)), ay, by),
                        nz = fmaf(__uint_as_float(B | ((oct & 4u) ? hz : lz)), az, bz),
                        fz = fmaf(__uint_as_float(B | ((oct & 4u) ? lz : hz)), az, bz);
            const float tn = fmaxf(fmaxf(nx, ny), fmaxf(nz, T.tmin));
            const float tf = fminf(fminf(fx, fy), fminf(fz, T.tbest)) * 1.0000004f;
            hit = m != 0u && tn <= tf;
            imask = w0.w >> 24;
            child = w1.x;
            if (hit && !((imask >> c) & 1u)) {
                cnt = m >> 5;
                first = w1.y + (m & 31u);
            }
        } else {
            fin = true;
        }
    }
    uint32_t ib = ((__ballot_sync(FULL, hit) >> shift) & 0xFFu) & imask;
    if (go) {
        const uint32_t x = oct ^ 7u;
        ib = (x & 1u) ? (((ib & 0x55u) << 1) | ((ib >> 1) & 0x55u)) : ib;
        ib = (x & 2u) ? (((ib & 0x33u) << 2) | ((ib >> 2) & 0x33u)) : ib;
        ib = (x & 4u) ? (((ib & 0x0Fu) << 4) | ((ib >> 4) & 0x0Fu)) : ib;
        T.g = make_uint2(child, (ib << 24) | imask);
    }
    if (!__any_sync(FULL, cnt != 0u)) return fin;
    // the hit leaves' triangles, each lane its own leaf's
    for (uint32_t k = 0; __any_sync(FULL, k < cnt); ++k) {
        if (k < cnt) {
            const TriSlot* ts = S.tris + first + k;
            const float4 a0 = __ldg(&ts->v0), a1 = __ldg(&ts->v1), a2 = __ldg(&ts->v2);
            ++n_tris;
            float t, u, v;
            if (tri_test(xyz(a0), xyz(a1), xyz(a2), T.o, T.axes & 3u, (T.axes >> 2) & 3u, (T.axes >> 4) & 3u, T.sx, T.sy,
                         T.sz, T.tmin, T.tbest, t, u, v)) {
                const uint32_t id = __float_as_uint(a0.w);
                if (t < T.t || (t == T.t && id < T.id)) {
                    T.t = t;
                    T.id = id;
                    T.u = u;
                    T.v = v;
                }
            }
        }
    }
    if (any) {
        if ((__ballot_sync(FULL, active && T.id != MISS) >> shift) & 0xFFu) fin = true;
    } else {
        float t = fminf(T.t, T.tbest);
        t = fminf(t, __shfl_xor_sync(FULL, t, 1));
        t = fminf(t, __shfl_xor_sync(FULL, t, 2));
        t = fminf(t, __shfl_xor_sync(FULL, t, 4));
        if (active) T.tbest = t;
    }
    return fin;
}

// The closest hit of each group's finished ray, in all its lanes: the
// lexicographic minimum of (t, id) over the lanes; prim MISS without a hit.
template <int STACK>
SRT_DEV void group_closest(const GroupTrav<STACK>& T, float& t, uint32_t& prim, float& u, float& v) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    t = T.t;
    prim = T.id;
    uint32_t own = threadIdx.x & 31u;
#pragma unroll
    for (uint32_t d = 1; d < GROUP; d <<= 1) {
        const float ot = __shfl_xor_sync(FULL, t, d);
        const uint32_t oi = __shfl_xor_sync(FULL, prim, d), oo = __shfl_xor_sync(FULL, own, d);
        if (ot < t || (ot == t && oi < prim)) {
            t = ot;
            prim = oi;
            own = oo;
        }
    }
    u = __shfl_sync(FULL, T.u, (int)own);
    v = __shfl_sync(FULL, T.v, (int)own);
}
// Whether an any-hit ray's group found a hit.
template <int STACK>
SRT_DEV bool group_occluded(const GroupTrav<STACK>& T) {
    return ((__ballot_sync(0xFFFFFFFFu, T.id != MISS) >> (threadIdx.x & 24u)) & 0xFFu) != 0u;
}

// ------------------------------------------------------------------ surface data at a hit
struct Surface {
    uint32_t inst, mat;
    float3 wn;     // normalised world shading normal (not face-forwarded)
    bool front;
};

// get_interpolated_normal (shader.wgsl:530-545), the world transform
// (:573-576) and the ray query's front_face: counter-clockwise as seen from
// the ray in object space.
SRT_DEV Surface surface_at(const DevScene& S, uint32_t prim, float u, float v, float3 dir_world) {
    Surface sf;
    uint32_t ii = __ldg(&S.tri_inst[prim]);
    const InstDev& in = S.inst[ii];
    const uint32_t vo = __float_as_uint(in.w2o0.w), io = __float_as_uint(in.w2o1.w) + prim * 3u;
    uint32_t i0 = __ldg(&S.indices[io]) + vo, i1 = __ldg(&S.indices[io + 1]) + vo, i2 = __ldg(&S.indices[io + 2]) + vo;
    float4 p0 = __ldg(&S.vtx[2 * i0]), n0 = __ldg(&S.vtx[2 * i0 + 1]);
    float4 p1 = __ldg(&S.vtx[2 * i1]), n1 = __ldg(&S.vtx[2 * i1 + 1]);
    float4 p2 = __ldg(&S.vtx[2 * i2]), n2 = __ldg(&S.vtx[2 * i2 + 1]);
    float w = 1.0f - u - v;
    float3 ln = normalize(xyz(n0) * w + xyz(n1) * u + xyz(n2) * v);
    float4 r0 = in.w2o0, r1 = in.w2o1, r2 = in.w2o2;
    // local_normal * mat3x3(w2o columns) = transpose(W2O) * n
    float3 wn = f3(ln.x * r0.x + ln.y * r1.x + ln.z * r2.x, ln.x * r0.y + ln.y * r1.y + ln.z * r2.y,
                   ln.x * r0.z + ln.y * r1.z + ln.z * r2.z);
    sf.wn = normalize(wn);
    float3 dobj = f3(dot(xyz(r0), dir_world), dot(xyz(r1), dir_world), dot(xyz(r2), dir_world));
    float3 gn = cross(xyz(p1) - xyz(p0), xyz(p2) - xyz(p0));
    sf.front = dot(dobj, gn) < 0.0f;
    sf.inst = ii;
    sf.mat = in.mat_id;
    return sf;
}

}  // namespace srt
