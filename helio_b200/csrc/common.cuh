// common.cuh — device-side arithmetic in the reference WGSL operation order.
//
// Every float operation goes through a correctly-rounded intrinsic (__fadd_rn,
// __fmul_rn, __fdiv_rn, __fsqrt_rn), so no FMA contraction or approximate
// division can change a visibility / LOD / mip decision, whatever the compiler
// flags. The rules (identical on every path of this library):
//   dot(a, b)      = (a.x*b.x + a.y*b.y) + a.z*b.z
//   M * vec4(p,1)  = ((M[0]*p.x + M[1]*p.y) + M[2]*p.z) + M[3]      (column sums)
//   mat3 * v       = (N[0]*v.x + N[1]*v.y) + N[2]*v.z
//   length(v)      = sqrt(dot(v, v)),  normalize(v) = v / length(v)
//   max / min      = fmaxf / fminf,  clamp(x, lo, hi) = fminf(fmaxf(x, lo), hi)
//   u32(ceil(log2(d))) for d >= 1 is exact, from the binary32 exponent/mantissa
//   textureSampleLevel (nearest, clamp-to-edge):
//       level = min(mip, mip_count - 1); i = clamp(floor(u * W_level), 0, W_level - 1)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/helio_cull.h"

namespace helio {

struct F3 {
    float x, y, z;
};

__device__ __forceinline__ F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fsqrt(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ F3 sub3(F3 a, F3 b) { return f3(fsub(a.x, b.x), fsub(a.y, b.y), fsub(a.z, b.z)); }
__device__ __forceinline__ F3 muls3(F3 a, float s) { return f3(fmul(a.x, s), fmul(a.y, s), fmul(a.z, s)); }
__device__ __forceinline__ F3 divs3(F3 a, float s) { return f3(fdiv(a.x, s), fdiv(a.y, s), fdiv(a.z, s)); }
__device__ __forceinline__ float dot3(F3 a, F3 b) {
    return fadd(fadd(fmul(a.x, b.x), fmul(a.y, b.y)), fmul(a.z, b.z));
}
__device__ __forceinline__ float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// ── Exact `a / b <= thr` without the correctly rounded division in clear cases ──
// r = rcp.approx.f32(b) has at most 1 ulp of error (PTX ISA), so q = RN(a * r)
// lies within 2^-22 (relative) of a / b. With margins of |thr| * 2^-18 on either
// side of thr, q below the lower margin proves RN(a / b) <= thr and q above the
// upper margin proves RN(a / b) > thr; everything in between (and NaN) takes the
// correctly rounded division. The margins are -inf / +inf (always exact) unless
// 2^-60 <= |thr| <= 2^60, and r is NaN (always exact) unless 2^-64 <= b <= 2^64,
// which keeps q clear of underflow relative to thr.
struct QuotientBound {
    float thr, lo, hi;
};

__device__ __forceinline__ QuotientBound quotient_bound(float thr) {
    const float at = fabsf(thr);
    if (at >= 0x1p-60f && at <= 0x1p60f) {
        const float m = fmul(at, 0x1p-18f);
        return QuotientBound{thr, fsub(thr, m), fadd(thr, m)};
    }
    return QuotientBound{thr, -__int_as_float(0x7f800000), __int_as_float(0x7f800000)};
}

__device__ __forceinline__ float quotient_rcp(float b) {
    if (!(b >= 0x1p-64f && b <= 0x1p64f)) return __int_as_float(0x7fffffff);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
}

// RN(a / b) <= q.thr, bit-for-bit; r = quotient_rcp(b).
__device__ __forceinline__ bool quotient_le(float a, float b, float r, const QuotientBound& q) {
    const float approx = fmul(a, r);
    if (approx < q.lo) return true;
    if (approx > q.hi) return false;
    return fdiv(a, b) <= q.thr;
}

// A load of what an earlier kernel of the stream, or its caller's, may have written. An ordinary one: the
// read-only path (ld.global.nc, __ldg) promises that nothing is written while the kernel runs, which
// a kernel launched as a dependent cannot, since it may be resident before the one that writes has
// ended; and no fence or clobber keeps a load of that kind behind pdl_wait.
template <typename T>
__device__ __forceinline__ T ld_weak(const T* p) {
    return *p;
}
// (The cull kernels use __ldca, the same load as a function of its own, which the compiler keeps where
// the code has it: as ordinary loads of structures' pointers they cost the frame kernel 276 bytes of
// spills, and frames of 100,000 objects 43.7 instead of 37.7 us.)
// x, known to the compiler only behind the wait before it (volatile statements keep their order).
__device__ __forceinline__ uint32_t after_wait(uint32_t x) {
    asm volatile("" : "+r"(x));
    return x;
}

// Column-major 4x4 matrix held as four columns.
struct Mat4 {
    float4 c0, c1, c2, c3;
};

__device__ __forceinline__ Mat4 load_mat4(const float* m) {
    const float4* p = reinterpret_cast<const float4*>(m);
    return Mat4{p[0], p[1], p[2], p[3]};
}
__device__ __forceinline__ Mat4 ld_mat4(const float* m) {
    const float4* p = reinterpret_cast<const float4*>(m);
    return Mat4{ld_weak(p), ld_weak(p + 1), ld_weak(p + 2), ld_weak(p + 3)};
}

// (M * vec4(p, 1)).xyz
__device__ __forceinline__ F3 mat4_point3(const Mat4& m, F3 p) {
    return f3(fadd(fadd(fadd(fmul(m.c0.x, p.x), fmul(m.c1.x, p.y)), fmul(m.c2.x, p.z)), m.c3.x),
              fadd(fadd(fadd(fmul(m.c0.y, p.x), fmul(m.c1.y, p.y)), fmul(m.c2.y, p.z)), m.c3.y),
              fadd(fadd(fadd(fmul(m.c0.z, p.x), fmul(m.c1.z, p.y)), fmul(m.c2.z, p.z)), m.c3.z));
}
// M * vec4(p, 1), all four components.
__device__ __forceinline__ float4 mat4_point4(const Mat4& m, F3 p) {
    F3 xyz = mat4_point3(m, p);
    float w = fadd(fadd(fadd(fmul(m.c0.w, p.x), fmul(m.c1.w, p.y)), fmul(m.c2.w, p.z)), m.c3.w);
    return make_float4(xyz.x, xyz.y, xyz.z, w);
}
// mat3(n0.xyz, n1.xyz, n2.xyz) * v
__device__ __forceinline__ F3 mat3_vec(float4 n0, float4 n1, float4 n2, F3 v) {
    return f3(fadd(fadd(fmul(n0.x, v.x), fmul(n1.x, v.y)), fmul(n2.x, v.z)),
              fadd(fadd(fmul(n0.y, v.x), fmul(n1.y, v.y)), fmul(n2.y, v.z)),
              fadd(fadd(fmul(n0.z, v.x), fmul(n1.z, v.y)), fmul(n2.z, v.z)));
}

// Exact u32(ceil(log2(d))) for d >= 1; values >= 2^32 (and +inf) give 0xFFFFFFFF.
__device__ __forceinline__ uint32_t ceil_log2_exact(float d) {
    if (!(d >= 1.0f)) return 0u;
    if (d >= 4294967296.0f) return 0xFFFFFFFFu;
    uint32_t bits = __float_as_uint(d);
    uint32_t e = ((bits >> 23) & 0xFFu) - 127u;
    return (bits & 0x7FFFFFu) ? e + 1u : e;
}

// Hi-Z pyramid as passed to kernels (a copy of helio_hiz_pyramid in param space). What a sample needs
// of its level but the pitch is one 16-byte word: lanes sample levels of their own.
struct HizLevel {
    const float* texels;
    uint32_t width, height;
};
static_assert(sizeof(HizLevel) == 16, "one load");
struct alignas(16) HizView {
    HizLevel level[HELIO_HIZ_MAX_MIPS];
    uint32_t pitch[HELIO_HIZ_MAX_MIPS];
    uint32_t mip_count;
    uint32_t pad[3];
};

__device__ __forceinline__ HizLevel hiz_level(const HizView& hz, uint32_t l) {
    const uint4 q = *reinterpret_cast<const uint4*>(&hz.level[l]);
    HizLevel r;
    r.texels = reinterpret_cast<const float*>(((uint64_t)q.y << 32) | q.x);
    r.width = q.z;
    r.height = q.w;
    return r;
}

// kCoherent: the pyramid was written earlier in the same launch, so it is read
// through L2 (ld.global.cg) instead of the read-only path.
template <bool kCoherent = false>
__device__ __forceinline__ float hiz_sample(const HizView& hz, float u, float v, uint32_t mip) {
    const uint32_t l = min(mip, hz.mip_count - 1u);
    const HizLevel lv = hiz_level(hz, l);
    const uint32_t w = lv.width, h = lv.height;
    // u, v lie in [0, 1] at every call site, so the products lie in [0, w] / [0, h].
    int ix = (int)floorf(fmul(u, (float)w));
    int iy = (int)floorf(fmul(v, (float)h));
    ix = min(max(ix, 0), (int)w - 1);
    iy = min(max(iy, 0), (int)h - 1);
    const float* p = lv.texels + (size_t)iy * hz.pitch[l] + ix;
    return kCoherent ? __ldcg(p) : __ldca(p);
}

// Frustum planes as published by vg_cull.wgsl:266-280 (GPU form, no length guard).
struct Planes {
    float4 p[6];
};

// p / length(p.xyz) for the six Gribb–Hartmann rows of view_proj (column-major).
__device__ __forceinline__ Planes publish_planes(const float* vp) {
    auto e = [&](int c, int r) { return vp[c * 4 + r]; };
    float p[6][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        p[0][c] = fadd(e(c, 3), e(c, 0));
        p[1][c] = fsub(e(c, 3), e(c, 0));
        p[2][c] = fadd(e(c, 3), e(c, 1));
        p[3][c] = fsub(e(c, 3), e(c, 1));
        p[4][c] = e(c, 2);
        p[5][c] = fsub(e(c, 3), e(c, 2));
    }
    Planes out;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        float len = fsqrt(dot3(f3(p[i][0], p[i][1], p[i][2]), f3(p[i][0], p[i][1], p[i][2])));
        out.p[i] = make_float4(fdiv(p[i][0], len), fdiv(p[i][1], len), fdiv(p[i][2], len), fdiv(p[i][3], len));
    }
    return out;
}

// The same planes computed by lanes 0..5 of one warp in parallel (lane i builds
// plane i); every lane of the warp must call it. Writes `out` (shared memory).
__device__ __forceinline__ void publish_planes_warp(const float* vp, Planes& out) {
    const int lane = threadIdx.x & 31;
    if (lane < 6) {
        float p[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float r3 = ld_weak(vp + c * 4 + 3);
            const float rr = ld_weak(vp + c * 4 + (lane >> 1));  // rows 0,0,1,1,2,2
            if (lane == 4) p[c] = ld_weak(vp + c * 4 + 2);
            else if (lane == 5) p[c] = fsub(r3, ld_weak(vp + c * 4 + 2));
            else if (lane & 1) p[c] = fsub(r3, rr);
            else p[c] = fadd(r3, rr);
        }
        const float len = fsqrt(dot3(f3(p[0], p[1], p[2]), f3(p[0], p[1], p[2])));
        out.p[lane] = make_float4(fdiv(p[0], len), fdiv(p[1], len), fdiv(p[2], len), fdiv(p[3], len));
    }
    __syncwarp();
}

// sphere_visible, vg_cull.wgsl:126-133: every plane satisfies dot(n, c) + d >= -r.
__device__ __forceinline__ bool sphere_visible_vg(const Planes& pl, F3 c, float r) {
    float nr = -r;
    bool v = true;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        float d = fadd(dot3(f3(pl.p[i].x, pl.p[i].y, pl.p[i].z), c), pl.p[i].w);
        v = v && (d >= nr);
    }
    return v;
}

// Programmatic dependent launch. A kernel launched with programmatic stream serialization
// is scheduled as the CTAs of the stream's previous kernel end; pdl_wait returns once that
// kernel has completed and its writes are visible (at once in a kernel launched normally), so
// it goes before the first read of anything the previous kernel wrote. No kernel here signals
// its dependents early (griddepcontrol.launch_dependents): their waiting CTAs then took slots and
// issue cycles from the running one (Hi-Z of 1367x769 back to back 6.5 us, 9.4 with the signal;
// frames 16.6, 26.8 and 43.7 us, 18.6, 31.0 and 46.4 with it).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Device error word values.
enum : uint32_t { kDevOk = 0u, kDevTimeout = 1u };

constexpr uint32_t kSpinLimit = 1u << 22;  // polls before a bounded wait gives up (~1 s with backoff)

}  // namespace helio

// Host-side launch accounting (helio_kernel_launch_count) and the optional
// event profiler (helio_profiler_*): every launch is bracketed by these two calls.
void helio_launch_begin(const char* kernel, cudaStream_t stream);
void helio_launch_end(cudaStream_t stream);
// Counts one more launch inside an open begin/end bracket (a step of several kernels).
void helio_launch_note(void);
// Records `message` as the calling thread's helio_last_error() and returns `code`.
int32_t helio_report_error(int32_t code, const char* message);
