// vg_device.cuh — device functions of the meshlet cull shared by the single-view
// kernels (vg_cull.cu) and the persistent multi-view kernel (batch.cu).
#pragma once

#include "common.cuh"
#include "vg.h"

namespace helio {

// 32 bytes in one load (sm_100); p is 32-byte aligned. (Not of the read-only path: see ld_weak.)
__device__ __forceinline__ void ld_pair(const float4* p, float4& a, float4& b) {
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// The frustum test's share of an instance: model holds xyz of each column (the w of columns 0 and 1
// carry max_scale and the flags, those of 2 and 3 the start of the normal matrix).
struct InstanceView {
    Mat4 model;
    __device__ float max_scale() const { return model.c0.w; }
    __device__ bool valid() const { return (__float_as_uint(model.c1.w) & 1u) != 0u; }
    __device__ bool cone() const { return (__float_as_uint(model.c1.w) & 2u) != 0u; }
};

__device__ __forceinline__ InstanceView load_instance(const VgSceneDev& S, uint32_t i) {
    const float4* p = S.xform + 6u * (size_t)i;
    InstanceView v;
    ld_pair(p, v.model.c0, v.model.c1);
    ld_pair(p + 2, v.model.c2, v.model.c3);
    return v;
}

// The rest of the normal matrix of instance i.
__device__ __forceinline__ void load_normal(const VgSceneDev& S, uint32_t i, float4& na, float4& nb) {
    ld_pair(S.xform + 6u * (size_t)i + 4u, na, nb);
}

// mat3(normal matrix) * axis, in the order of mat3_vec.
__device__ __forceinline__ F3 normal_vec(const InstanceView& v, float4 na, float4 nb, float4 axis) {
    return mat3_vec(make_float4(v.model.c2.w, v.model.c3.w, na.x, 0.0f), make_float4(na.y, na.z, na.w, 0.0f), nb,
                    f3(axis.x, axis.y, axis.z));
}

__device__ __forceinline__ ObjectWorld load_world(const VgSceneDev& S, uint32_t o) {
    const uint4 a = __ldca(S.world + 2u * (size_t)o), b = __ldca(S.world + 2u * (size_t)o + 1u);
    ObjectWorld w;
    w.sphere = make_float4(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w));
    w.max_scale = __uint_as_float(b.x);
    w.lod_count = b.y;
    w.instance = b.z;
    w.pad = 0u;
    return w;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The cone test's decision dot(cta / |cta|, a / |a|) >= cutoff (vg_cull.wgsl:172-180),
// bit-for-bit. The reference value E normalises both vectors with a correctly rounded
// square root and three divisions each, then takes the dot product; it lies within
// about 10 ulp(1) of the real cosine R (both vectors are unit length after
// normalisation, so every term is at most 1). D = fma-dot(cta, a) * rsqrt.approx(|cta|^2)
// * rsqrt.approx(|a|^2) lies within about 16 ulp(1) of R: 3 roundings in the dot
// (relative to sum |cta_i a_i| <= |cta||a|), at most 2^-22.9 relative error in each
// rsqrt.approx (PTX ISA) plus the squared norms' own rounding, and two products. So
// |D - E| < 2^-19, and D outside cutoff +- 2^-16 decides the comparison; everything
// else (and squared norms outside [1e-30, 1e30], non-finite values) takes the
// reference's own sequence.
__device__ __forceinline__ bool cone_rejects(F3 a, F3 cta, float ads, float cutoff) {
    const float da = dot3(a, a);
    if (da >= 1.0e-30f && da <= 1.0e30f && ads <= 1.0e30f) {
        const float t = fmaf(cta.z, a.z, fmaf(cta.y, a.y, cta.x * a.x));
        const float d = t * rsqrt_approx(ads) * rsqrt_approx(da);
        if (isfinite(d)) {
            if (d >= cutoff + 0x1p-16f) return true;
            if (d < cutoff - 0x1p-16f) return false;
        }
    }
    const F3 axis_ws = divs3(a, fsqrt(da));
    return dot3(divs3(cta, fsqrt(ads)), axis_ws) >= cutoff;
}

// cull_meshlet, first part (vg_cull.wgsl:143-182): the frustum and normal-cone
// tests. True = the meshlet is still a candidate and the Hi-Z test decides it;
// (c, wr) is its world-space sphere (:150-152). kLazyCone: the cone's other inputs (axis, the rest of
// the normal matrix) are loaded only for meshlets whose sphere passes the frustum: fewer registers
// live at a time, for kernels that run more warps per SM instead of more loads per warp. Otherwise
// everything is loaded in one go (one memory round trip instead of one per test).
template <bool kLazyCone>
__device__ __forceinline__ bool meshlet_frustum_cone(const CullView& C, const VgSceneDev& S, uint32_t mi,
                                                     uint32_t instance, F3& c, float& wr) {
    const InstanceView in = load_instance(S, instance);
    float4 b, cone, axis, na, nb;
    ld_pair(S.m_bounds + 2u * (size_t)mi, b, cone);
    if (!kLazyCone) {
        axis = __ldca(S.m_axis + mi);
        load_normal(S, instance, na, nb);
    }
    if (!in.valid()) return false;
    c = mat4_point3(in.model, f3(b.x, b.y, b.z));
    wr = fmaxf(fmul(b.w, in.max_scale()), 0.0f);
    if (!sphere_visible_vg(C.planes, c, wr)) return false;
    // Perspective normal-cone test (:159-182).
    if (in.cone()) {
        const F3 cam = f3(C.pos_near.x, C.pos_near.y, C.pos_near.z);
        const F3 ctc = sub3(c, cam);
        const float cam_dist_sq = dot3(ctc, ctc);
        const float guard = fmul(wr, 1.5f);
        if (cam_dist_sq > fmul(guard, guard) && cone.w <= 1.0f) {
            if (kLazyCone) {
                axis = __ldca(S.m_axis + mi);
                load_normal(S, instance, na, nb);
            }
            const F3 a = normal_vec(in, na, nb, axis);
            const F3 apex = mat4_point3(in.model, f3(cone.x, cone.y, cone.z));
            const F3 cta = sub3(apex, cam);
            const float ads = dot3(cta, cta);
            if (ads > 1.0e-12f && cone_rejects(a, cta, ads, cone.w)) return false;
        }
    }
    return true;
}

// cull_meshlet, second part (vg_cull.wgsl:184-240): the conservative Hi-Z test of
// the sphere (c, wr). True = visible. kCoherentHiz: the pyramid was written
// earlier in the same launch.
template <bool kCoherentHiz = false>
__device__ __forceinline__ bool meshlet_hiz_visible(const CullView& C, F3 c, float wr) {
    const HizView& hz = C.hiz;
    const F3 ctc = sub3(c, f3(C.pos_near.x, C.pos_near.y, C.pos_near.z));
    const float4 clip = mat4_point4(C.vp, c);
    if (clip.w > 0.0f) {
        const float ndc_x = fdiv(clip.x, clip.w), ndc_y = fdiv(clip.y, clip.w);
        const float uv_x = fadd(fmul(ndc_x, 0.5f), 0.5f), uv_y = fadd(fmul(ndc_y, -0.5f), 0.5f);
        const float nvd = fsub(clip.w, wr);
        if (nvd > C.pos_near.w) {
            const float ndc_r = fmaxf(fabsf(fdiv(fmul(wr, C.p00), nvd)), fabsf(fdiv(fmul(wr, C.p11), nvd)));
            const float uvr = fmul(ndc_r, 0.5f);
            const float u0 = fsub(uv_x, uvr), v0 = fsub(uv_y, uvr), u1 = fadd(uv_x, uvr), v1 = fadd(uv_y, uvr);
            if (u0 >= 0.0f && v0 >= 0.0f && u1 <= 1.0f && v1 <= 1.0f) {
                // The four texel loads first: the sphere's nearest depth below is computed
                // while they are in flight (neither depends on the other).
                const float half_h = fmul((float)C.screen_height, 0.5f);
                const float dpx = fmaxf(fmul(fmul(ndc_r, half_h), 2.0f), 1.0f);
                const uint32_t mip = min(ceil_log2_exact(dpx), C.hiz_mip_count - 1u);
                const float h00 = hiz_sample<kCoherentHiz>(hz, u0, v0, mip);
                const float h01 = hiz_sample<kCoherentHiz>(hz, u1, v0, mip);
                const float h10 = hiz_sample<kCoherentHiz>(hz, u0, v1, mip);
                const float h11 = hiz_sample<kCoherentHiz>(hz, u1, v1, mip);
                const float dist_sq = dot3(ctc, ctc);
                float near_z = 0.0f;
                if (dist_sq > fmul(wr, wr)) {
                    const F3 dir = divs3(ctc, fsqrt(dist_sq));
                    const F3 nws = sub3(c, muls3(dir, wr));
                    const float4 nc = mat4_point4(C.vp, nws);
                    if (nc.w > 0.0f) near_z = clampf(fdiv(nc.z, nc.w), 0.0f, 1.0f);
                }
                const float hzv = fmaxf(fmaxf(h00, h01), fmaxf(h10, h11));
                if (near_z > fadd(hzv, 1.0f / 65536.0f)) return false;
            }
        }
    }
    return true;
}

// cull_meshlet decision part (vg_cull.wgsl:143-240): true = emit a draw.
template <bool kCoherentHiz = false, bool kLazyCone = false>
__device__ __forceinline__ bool meshlet_visible(const VgSceneDev& S, const CullView& C, uint32_t mi,
                                                uint32_t instance) {
    F3 c;
    float wr;
    if (!meshlet_frustum_cone<kLazyCone>(C, S, mi, instance, c, wr)) return false;
    return meshlet_hiz_visible<kCoherentHiz>(C, c, wr);
}

// Largest lane j whose exclusive offset is <= s (for s below the warp total this
// is the item that owns window slot s; empty items are skipped because they share
// their offset with the next item).
__device__ __forceinline__ int owner_lane(uint32_t off, uint32_t s) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const uint32_t o = __shfl_sync(0xffffffffu, off, lo + step);
        if (o <= s) lo += step;
    }
    return lo;
}

// Bits [off, off + n) (n <= 64) of a little-endian bit array of 32-bit words; the
// two words after the field's first word must be readable.
__device__ __forceinline__ uint2 bit_field64(const uint32_t* words, uint32_t off, uint32_t n) {
    if (n == 0) return make_uint2(0u, 0u);
    const uint32_t w0 = off >> 5, sh = off & 31u;
    const unsigned long long a = (unsigned long long)words[w0] | ((unsigned long long)words[w0 + 1] << 32);
    const unsigned long long c = words[w0 + 2];
    unsigned long long field = sh ? ((a >> sh) | (c << (64 - sh))) : a;
    if (n < 64) field &= (1ull << n) - 1ull;
    return make_uint2((uint32_t)field, (uint32_t)(field >> 32));
}

}  // namespace helio
