// vg_cull.cu — virtual-geometry object select and meshlet cull (VirtualGeometryPass).
//
// References (crates/helio-pass-virtual-geometry/):
//   shaders/vg_cull.wgsl:282-352   cs_select_objects  -> select_object
//   shaders/vg_cull.wgsl:135-264   cull_meshlet       -> meshlet_visible + emission
//   shaders/vg_cull.wgsl:354-405   cs_cull_meshlets   -> vg_frame_kernel
//   src/lib.rs:132-167             InstanceCullData::from_instance -> instance_cull_data_kernel
//
// Layout and scheduling (B200 design, not a translation of the WGSL dispatches):
//   * meshlet descriptors are re-laid once per upload into three streams;
//   * one launch does the whole view. A tile CTA takes up to 512 consecutive work items, two
//     per thread, and selects their objects itself (an object's few items repeat its select,
//     from L2, which costs less than a launch and a round trip of records in between); it then
//     packs the items' active meshlets densely into 32-lane windows shared out over its warps,
//     so a work item whose LOD has 13 meshlets occupies 13 lanes and a warp whose items are all
//     visible does not run on alone;
//   * further CTAs run the select once per object for its outputs (objects[i].reserved, the
//     LOD histogram), in the shadow of the tiles;
//   * visible meshlets are compacted deterministically: tiles are handed out in order by a
//     ticket, each publishes its count and takes its first slot from the tiles before it
//     (decoupled look-back, bounded), so each draw lands at slot = (visible meshlets before it
//     in (work item, lane) order). The reference appends with atomicAdd (vg_cull.wgsl:247), so
//     its order is unspecified; this order is reproducible and first_instance = slot.

#include <algorithm>

#include "common.cuh"
#include "host_util.h"
#include "kernels.h"
#include "vg.h"
#include "vg_device.cuh"

namespace helio {

namespace {

// ── Scene preparation ─────────────────────────────────────────────────────────

// InstanceCullData::from_instance (lib.rs:132-167), Rust f32 evaluation order, of the
// column-major model matrix m.
__device__ __forceinline__ HelioInstanceCullData cull_data_of(const Mat4& mm) {
    const float m[16] = {mm.c0.x, mm.c0.y, mm.c0.z, mm.c0.w, mm.c1.x, mm.c1.y, mm.c1.z, mm.c1.w,
                         mm.c2.x, mm.c2.y, mm.c2.z, mm.c2.w, mm.c3.x, mm.c3.y, mm.c3.z, mm.c3.w};
    const float sx = fsqrt(fadd(fadd(fmul(m[0], m[0]), fmul(m[1], m[1])), fmul(m[2], m[2])));
    const float sy = fsqrt(fadd(fadd(fmul(m[4], m[4]), fmul(m[5], m[5])), fmul(m[6], m[6])));
    const float sz = fsqrt(fadd(fadd(fmul(m[8], m[8]), fmul(m[9], m[9])), fmul(m[10], m[10])));
    const float max_scale = fmaxf(fmaxf(sx, sy), sz);
    const float min_scale = fminf(fminf(sx, sy), sz);
    const float dot_xy = fadd(fadd(fmul(m[0], m[4]), fmul(m[1], m[5])), fmul(m[2], m[6]));
    const float dot_xz = fadd(fadd(fmul(m[0], m[8]), fmul(m[1], m[9])), fmul(m[2], m[10]));
    const float dot_yz = fadd(fadd(fmul(m[4], m[8]), fmul(m[5], m[9])), fmul(m[6], m[10]));
    const float det = fadd(fsub(fmul(m[0], fsub(fmul(m[5], m[10]), fmul(m[6], m[9]))),
                                fmul(m[4], fsub(fmul(m[1], m[10]), fmul(m[2], m[9])))),
                           fmul(m[8], fsub(fmul(m[1], m[6]), fmul(m[2], m[5]))));
    const bool affine = fabsf(m[3]) <= 1.0e-6f && fabsf(m[7]) <= 1.0e-6f && fabsf(m[11]) <= 1.0e-6f &&
                        fabsf(fsub(m[15], 1.0f)) <= 1.0e-4f;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 16; ++k) finite = finite && isfinite(m[k]);
    const bool valid = finite && isfinite(max_scale) && min_scale > 1.0e-8f && affine;
    const float ut = fmul(max_scale, 1.0e-4f);
    const float ot = fmul(fmul(max_scale, max_scale), 1.0e-4f);
    const bool ap = fsub(max_scale, min_scale) <= ut && fabsf(dot_xy) <= ot && fabsf(dot_xz) <= ot &&
                    fabsf(dot_yz) <= ot;
    const bool cone = valid && ap && det > 0.0f;
    HelioInstanceCullData r;
    r.max_scale = valid ? max_scale : 0.0f;
    r.min_scale = valid ? min_scale : 0.0f;
    r.cone_cull_enabled = cone ? 1u : 0u;
    r.valid_transform = valid ? 1u : 0u;
    return r;
}

__global__ void instance_cull_data_kernel(const HelioGpuInstanceData* __restrict__ inst, uint32_t n,
                                          HelioInstanceCullData* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = cull_data_of(ld_mat4(inst[i].model));
}

// launch_scene_update. CTAs come in three kinds: one per 256 rows and 256 objects (the same
// indices, since an object mostly names the instance of its own index, whose row is then in L1), one
// per 2048 work items, one per 512 meshlets. Copies have all their loads in flight before the
// first store. No kind waits for another's results: rows are read from their source, and an object
// recomputes its instance's scale. Bound by memory: 240 bytes per row, 256 per copied object.
// Bounds and sums meet in the block, so that a block costs at most five atomics (two per warp on
// the same two words took 37 us for 475,000 objects).
constexpr uint32_t kUpdateThreads = 256;
constexpr uint32_t kUpdateItems = 8 * kUpdateThreads;
constexpr uint32_t kUpdateMeshlets = 2 * kUpdateThreads;

// 32 bytes in one store (sm_100), a whole sector; p is 32-byte aligned.
__device__ __forceinline__ void st_pair(float4* p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}

// Copies n 16-byte words (at most kEach per thread) from src to dst, loads first.
template <int kEach>
__device__ __forceinline__ void copy_words(uint4* dst, const uint4* src, uint32_t n) {
    uint4 x[kEach];
#pragma unroll
    for (int k = 0; k < kEach; ++k)
        if (k * kUpdateThreads + threadIdx.x < n) x[k] = ld_weak(src + k * kUpdateThreads + threadIdx.x);
#pragma unroll
    for (int k = 0; k < kEach; ++k)
        if (k * kUpdateThreads + threadIdx.x < n) dst[k * kUpdateThreads + threadIdx.x] = x[k];
}

__device__ __forceinline__ void update_items(const SceneUpdate& U, uint32_t block) {
    const uint2* src = reinterpret_cast<const uint2*>(U.src_items);
    uint2* dst = reinterpret_cast<uint2*>(U.items);
    uint2 x[8];
    const uint64_t i0 = (uint64_t)block * kUpdateItems + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (i0 + k * kUpdateThreads < U.item_count) x[k] = ld_weak(src + i0 + k * kUpdateThreads);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (i0 + k * kUpdateThreads < U.item_count) dst[i0 + k * kUpdateThreads] = x[k];
}

// Meshlets into the three streams.
__device__ __forceinline__ void update_meshlets(const SceneUpdate& U, uint32_t block) {
    const uint4* src = reinterpret_cast<const uint4*>(U.src_meshlets);
    uint4* streams[4] = {reinterpret_cast<uint4*>(U.m_bounds), reinterpret_cast<uint4*>(U.m_bounds) + 1,
                         reinterpret_cast<uint4*>(U.m_axis), U.m_draw};
    const uint64_t m0 = (uint64_t)block * kUpdateMeshlets;
    uint4 x[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint64_t m = m0 + (uint32_t)r * kUpdateThreads + threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (m < U.meshlet_count) x[r][k] = __ldcs(src + 4u * m + k);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint64_t m = m0 + (uint32_t)r * kUpdateThreads + threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (m < U.meshlet_count) streams[k][k < 2 ? 2u * m : m] = x[r][k];
    }
}

// The InstanceXform of instance first + k from its row.
__device__ __forceinline__ void put_xform(const SceneUpdate& U, uint32_t k) {
    const float4* row = reinterpret_cast<const float4*>(U.rows + k);
    const Mat4 m{ld_weak(row), ld_weak(row + 1), ld_weak(row + 2), ld_weak(row + 3)};
    const float4 n0 = ld_weak(row + 4), n1 = ld_weak(row + 5), n2 = ld_weak(row + 6);
    const HelioInstanceCullData cd = cull_data_of(m);
    const uint32_t flags = (cd.valid_transform ? 1u : 0u) | (cd.cone_cull_enabled ? 2u : 0u);
    float4* x = U.xform + 6u * (size_t)(U.first + k);
    st_pair(x, make_float4(m.c0.x, m.c0.y, m.c0.z, cd.max_scale),
            make_float4(m.c1.x, m.c1.y, m.c1.z, __uint_as_float(flags)));
    st_pair(x + 2, make_float4(m.c2.x, m.c2.y, m.c2.z, n0.x), make_float4(m.c3.x, m.c3.y, m.c3.z, n0.y));
    st_pair(x + 4, make_float4(n0.z, n1.x, n1.y, n1.z), make_float4(n2.x, n2.y, n2.z, 0.0f));
}

// The ObjectWorld of object i, of `lods` LODs and the local sphere lb, which names row k. Returns the
// LODs of the record (0: the object is never visible) and its world sphere.
__device__ __forceinline__ uint32_t put_world(const SceneUpdate& U, uint32_t i, uint32_t k, uint32_t lods, float4 lb,
                                              float4& sphere) {
    const Mat4 model = ld_mat4(U.rows[k].model);
    const HelioInstanceCullData cd = cull_data_of(model);
    uint32_t live = 0;
    if (lods && cd.valid_transform) {
        const F3 c = mat4_point3(model, f3(lb.x, lb.y, lb.z));
        sphere = make_float4(c.x, c.y, c.z, fmaxf(fmul(lb.w, cd.max_scale), 0.0f));
        live = lods;
    }
    U.world[2u * (size_t)i] = make_uint4(__float_as_uint(sphere.x), __float_as_uint(sphere.y),
                                         __float_as_uint(sphere.z), __float_as_uint(sphere.w));
    U.world[2u * (size_t)i + 1u] = make_uint4(__float_as_uint(cd.max_scale), live, U.first + k, 0u);
    return live;
}

template <bool kTotals>
__global__ void __launch_bounds__(kUpdateThreads, 4)
    scene_update_kernel(const __grid_constant__ SceneUpdate U, uint32_t object_blocks, uint32_t item_blocks) {
    const VgSceneDev& S = U.scene;
    pdl_wait();
    if (blockIdx.x >= object_blocks) {
        const uint32_t b = blockIdx.x - object_blocks;
        if (b < item_blocks) update_items(U, b);
        else update_meshlets(U, b - item_blocks);
        return;
    }
    const uint32_t i0 = blockIdx.x * kUpdateThreads, i = after_wait(i0 + threadIdx.x);
    if (U.src_objects && i0 < S.object_count)
        copy_words<8>(reinterpret_cast<uint4*>(S.objects + i0), reinterpret_cast<const uint4*>(U.src_objects + i0),
                      min(kUpdateThreads, S.object_count - i0) * (uint32_t)(sizeof(HelioGpuVgObject) / 16));
    // The object's fields are on their way while the instance's record is made.
    const HelioGpuVgObject* obj = (U.src_objects ? U.src_objects : S.objects) + i;
    uint2 head = make_uint2(0u, 0u);  // instance_index, lod_count
    float4 lb = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < S.object_count) {
        head = ld_weak(reinterpret_cast<const uint2*>(obj));
        lb = ld_weak(reinterpret_cast<const float4*>(obj->local_bounds));
    }
    if (i < U.count) put_xform(U, i);
    uint32_t rad = 0u, far1 = 0u;  // bits of the largest radius and centre (non-negative floats order like their bits)
    unsigned long long lod0 = 0, spans = 0, draws = 0;
    if (i < S.object_count) {
        const uint32_t lods = min(head.y, 8u);
        if (kTotals) {
            const uint4 c0 = ld_weak(reinterpret_cast<const uint4*>(obj->lod_meshlet_counts));
            const uint4 c1 = ld_weak(reinterpret_cast<const uint4*>(obj->lod_meshlet_counts + 4));
            const uint32_t c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            uint32_t mx = 0;
#pragma unroll
            for (uint32_t l = 0; l < 8; ++l) mx = l < lods ? max(mx, c[l]) : mx;
            lod0 = c[0];
            spans = (mx + 63u) / 64u;
            draws = mx;
        }
        float4 sphere = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t live = 0;
        const bool named = head.x < S.instance_count;
        if (U.names) U.names[i] = head.x;
        if (named && head.x - U.first < U.count) {
            live = put_world(U, i, head.x - U.first, lods, lb, sphere);
        } else if (!named) {
            U.world[2u * (size_t)i] = U.world[2u * (size_t)i + 1u] = make_uint4(0u, 0u, 0u, 0u);
        } else if (U.bounds) {
            const ObjectWorld w = load_world(S, i);
            sphere = w.sphere;
            live = w.lod_count;
        }
        if (live) {
            rad = __float_as_uint(sphere.w);  // (NaN above +inf)
            // Rounding up is not needed: the reject boxes leave 2^-20 of slack.
            far1 = __float_as_uint(fabsf(sphere.x) + fabsf(sphere.y) + fabsf(sphere.z));
        }
    }
    if (!U.bounds && !kTotals) return;
    __shared__ uint32_t s_max[2];
    __shared__ unsigned long long s_sum[3];
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0ull;
    __syncthreads();
    rad = __reduce_max_sync(0xffffffffu, rad);
    far1 = __reduce_max_sync(0xffffffffu, far1);
    if (kTotals) {
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) {
            lod0 += __shfl_xor_sync(0xffffffffu, lod0, k);
            spans += __shfl_xor_sync(0xffffffffu, spans, k);
            draws += __shfl_xor_sync(0xffffffffu, draws, k);
        }
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicMax(s_max, rad);
        atomicMax(s_max + 1, far1);
        if (kTotals) {
            atomicAdd(s_sum, lod0);
            atomicAdd(s_sum + 1, spans);
            atomicAdd(s_sum + 2, draws);
        }
    }
    __syncthreads();
    if (U.bounds && threadIdx.x < 2 && s_max[threadIdx.x]) atomicMax(U.bounds + threadIdx.x, s_max[threadIdx.x]);
    if (kTotals && threadIdx.x < 3 && s_sum[threadIdx.x]) atomicAdd(U.totals + threadIdx.x, s_sum[threadIdx.x]);
}

// A patch: a thread per row, and the objects' names over the grid, four loads in flight per thread; the
// objects that name a row in the range are derived again. Reading every object's head and bounds for
// that made a patch of one row as slow as the scene is large (a million objects: 19.4 us, 5.1 with
// the names).
__global__ void __launch_bounds__(kUpdateThreads) scene_patch_kernel(const __grid_constant__ SceneUpdate U) {
    const VgSceneDev& S = U.scene;
    pdl_wait();
    const uint32_t i = blockIdx.x * kUpdateThreads + threadIdx.x, step = gridDim.x * kUpdateThreads;
    if (i < U.count) put_xform(U, i);  // (a thread per row at the least)
    for (uint64_t o0 = i; o0 < S.object_count; o0 += 4ull * step) {
        uint32_t k[4];  // the row that object o0 + j * step names
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            k[j] = o0 + (uint64_t)j * step < S.object_count ? U.names[o0 + (uint64_t)j * step] - U.first : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            if (k[j] >= U.count) continue;
            const uint32_t o = (uint32_t)(o0 + (uint64_t)j * step);
            const uint32_t lods = min(ld_weak(&S.objects[o].lod_count), 8u);
            const float4 lb = ld_weak(reinterpret_cast<const float4*>(S.objects[o].local_bounds));
            float4 sphere = make_float4(0.f, 0.f, 0.f, 0.f);
            put_world(U, o, k[j], lods, lb, sphere);
        }
    }
}

// ── View constants ────────────────────────────────────────────────────────────

// The view constants of P's camera into v (shared memory), by one warp (every lane of
// the warp calls it; lanes 0..5 build the planes, lane 0 the camera's fields, all of them copy
// the pyramid descriptor).
__device__ __forceinline__ void view_setup_warp(const ViewSetupParams& P, CullView& v) {
    const uint32_t lane = threadIdx.x & 31u;
    publish_planes_warp(P.camera->view_proj, v.planes);
    static_assert(sizeof(HizView) % 4 == 0, "copied word by word");
    for (uint32_t k = lane; k < sizeof(HizView) / 4; k += 32u)
        reinterpret_cast<uint32_t*>(&v.hiz)[k] = reinterpret_cast<const uint32_t*>(&P.hiz)[k];
    if (lane == 0) {
        const HelioGpuCameraUniforms* cam = P.camera;
        v.vp = ld_mat4(cam->view_proj);
        v.pos_near = ld_weak(reinterpret_cast<const float4*>(cam->position_near));
        v.p00 = ld_weak(&cam->proj[0]);
        v.p11 = ld_weak(&cam->proj[5]);
        v.focal = fmul(fmul(fabsf(v.p11), (float)P.screen_height), 0.5f);
        v.lod_threshold_px = P.lod_threshold_px;
        v.screen_height = P.screen_height;
        v.hiz_mip_count = P.hiz_mip_count;
        v.first_span = v.pad = 0u;
    }
    __syncwarp();
}

// ── Object select: cs_select_objects (vg_cull.wgsl:282-352) ───────────────────

struct Selected {
    uint32_t sel;  // LOD + 1, 0 = culled
    uint32_t lod_count, instance;
};

__device__ __forceinline__ Selected select_object(const VgSceneDev& S, const CullView& view, uint32_t i) {
    const ObjectWorld w = load_world(S, i);
    Selected r{0u, w.lod_count, w.instance};
    const F3 c = f3(w.sphere.x, w.sphere.y, w.sphere.z);
    const float wr = w.sphere.w;
    if (w.lod_count == 0u || !sphere_visible_vg(view.planes, c, wr)) return r;
    const HelioGpuVgObject* o = S.objects + i;
    const float4 e0 = __ldca(reinterpret_cast<const float4*>(o->lod_errors));
    const float4 e1 = __ldca(reinterpret_cast<const float4*>(o->lod_errors + 4));
    const float4 pn = view.pos_near;
    const F3 d = sub3(c, f3(pn.x, pn.y, pn.z));
    const float dist = fsqrt(dot3(d, d));
    const float closest = fmaxf(fsub(dist, wr), fmaxf(pn.w, 1.0e-4f));
    const float focal = view.focal;
    const QuotientBound qb = quotient_bound(view.lod_threshold_px);
    const float rc = quotient_rcp(closest);
    const float err[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
    uint32_t lod = 0;
#pragma unroll
    for (uint32_t level = 1; level < 8; ++level) {
        if (level >= r.lod_count) break;
        // px = err * max_scale * focal / closest; px <= threshold keeps the level.
        if (quotient_le(fmul(fmul(err[level], w.max_scale), focal), closest, rc, qb)) lod = level;
        else break;
    }
    r.sel = lod + 1u;
    return r;
}

// Object CTA: the select's outputs of kObjectBlock objects. The CTA that finishes last (an atomic
// count) publishes the histogram and leaves the accumulators at zero for the next launch.
constexpr uint32_t kObjectRounds = 4;
constexpr uint32_t kObjectBlock = kObjectRounds * kCullWarps * 32u;

__device__ void object_block(const VgFrameParams& P, const CullView& view, uint32_t block, uint32_t blocks,
                             uint32_t* s_hist, uint32_t* s_flag) {
    const VgSceneDev& S = P.scene;
    const uint32_t i0 = after_wait(block * kObjectBlock + threadIdx.x), lane = threadIdx.x & 31u;
    if (threadIdx.x < 9) s_hist[threadIdx.x] = 0u;
    Selected r[kObjectRounds];
#pragma unroll
    for (uint32_t k = 0; k < kObjectRounds; ++k) {
        const uint32_t i = i0 + k * kCullWarps * 32u;
        r[k] = Selected{0u, 0u, 0u};
        if (i < S.object_count) {
            r[k] = select_object(S, view, i);
            S.objects[i].reserved = r[k].sel;
        }
    }
    if (P.counter_count < 11u) return;  // uniform over the grid
    __syncthreads();
    uint32_t mx = 0;
#pragma unroll
    for (uint32_t k = 0; k < kObjectRounds; ++k) {
        mx = max(mx, r[k].sel ? r[k].lod_count - 1u : 0u);
        if (!__any_sync(0xffffffffu, r[k].sel != 0u)) continue;
#pragma unroll
        for (uint32_t l = 0; l < 8; ++l) {
            const uint32_t n = __popc(__ballot_sync(0xffffffffu, r[k].sel == l + 1u));
            if (lane == 0 && n) atomicAdd(s_hist + l, n);
        }
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(s_hist + 8, mx);
    __syncthreads();
    uint32_t* hist = P.state + kVgHist;
    if (threadIdx.x < 8 && s_hist[threadIdx.x]) atomicAdd(hist + threadIdx.x, s_hist[threadIdx.x]);
    if (threadIdx.x == 8 && s_hist[8]) atomicMax(hist + 8, s_hist[8]);
    __threadfence();  // this CTA's sums before its count
    __syncthreads();
    if (threadIdx.x == 0) *s_flag = atomicAdd(P.state + kVgDone, 1u) + 1u == blocks;
    __syncthreads();
    if (!*s_flag) return;
    __threadfence();
    if (threadIdx.x < 9) {
        P.counters[2 + threadIdx.x] = __ldcg(hist + threadIdx.x);
        hist[threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) P.state[kVgDone] = 0u;
}

// ── Meshlet cull ──────────────────────────────────────────────────────────────

constexpr uint32_t kThreads = kCullWarps * 32u;
constexpr uint32_t kMaxWindows = kMaxTileItems * HELIO_VG_MESHLETS_PER_WORK_ITEM / 32u;  // of a tile
constexpr uint32_t kItemRounds = kMaxTileItems / kThreads;  // items per thread
constexpr uint32_t kThreadWindows = kMaxWindows / kThreads;  // windows per thread, counted after the tests
static_assert(kItemRounds == 2u && kThreadWindows * kThreads == kMaxWindows, "the tile's rounds");
// A packed position and a rank share a word (rank << 16 | position).
static_assert(kMaxTileItems * HELIO_VG_MESHLETS_PER_WORK_ITEM < (1u << 16) && kMaxTileItems < (1u << 16), "packed scan");

// Exclusive scan over the CTA; `total` gets the CTA's sum. s: kCullWarps words.
__device__ __forceinline__ uint32_t tile_scan(uint32_t x, uint32_t* s, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = x;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    __syncthreads();
    if (lane == 31u) s[warp] = inc;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kCullWarps; ++w) {
        const uint32_t t = s[w];
        if (w < warp) before += t;
        total += t;
    }
    return before + inc - x;
}

// The active items of a tile in item order (rank = position among the active ones).
struct TileItems {
    uint32_t off[kMaxTileItems];    // packed position of the item's first meshlet
    uint32_t first[kMaxTileItems];  // its first meshlet
    uint32_t inst[kMaxTileItems];
    uint8_t lod[kMaxTileItems];
    uint32_t heads[kMaxWindows];    // bit p of word w: an item starts at position 32 w + p
    uint16_t owner[kMaxWindows];    // rank of the item that holds position 32 w
};

// Rank of the item that holds position 32 w + lane.
__device__ __forceinline__ uint32_t item_at(const TileItems& t, uint32_t w) {
    const uint32_t le = 0xffffffffu >> (31u - (threadIdx.x & 31u));
    return t.owner[w] + __popc(t.heads[w] & le & ~1u);
}

// A status holds the tile's count, or all up to it; or the tile's wait gave up.
enum : uint32_t { kTileSum = 1u, kTilePrefix = 2u, kTileLost = 3u };

__device__ __forceinline__ unsigned long long tile_status(uint32_t epoch, uint32_t kind, uint32_t value) {
    return ((unsigned long long)(epoch & 0x3FFFFFFFu) << 34) | ((unsigned long long)kind << 32) | value;
}
// Relaxed GPU-scope accesses: a status carries its whole message.
__device__ __forceinline__ unsigned long long ld_status(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_status(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Visible meshlets of the tiles before `tile`, by the whole CTA: thread t waits (bounded) for
// the status of tile hi - 1 - t; the nearest one that holds a prefix ends the walk, the counts
// nearer than it are added. Every earlier ticket is held by a CTA that runs and publishes its
// count without waiting, so the waits end. Returns false, uniformly, when one gave up, here or in
// a tile before this one.
__device__ bool tile_look_back(const VgFrameParams& P, uint32_t tile, uint32_t epoch, uint32_t* s_red,
                               uint32_t& prefix) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    prefix = 0;
    for (uint32_t hi = tile; hi > 0;) {
        const bool mine = threadIdx.x < hi;
        unsigned long long st = 0;
        int lost = 0;
        if (mine) {
            const unsigned long long* p = P.status + (hi - 1u - threadIdx.x);
            uint32_t polls = 0;
            while (st = ld_status(p), (uint32_t)(st >> 34) != (epoch & 0x3FFFFFFFu)) {
                if (++polls > P.spin_limit) {
                    lost = 1;
                    break;
                }
                if (polls > 32u) __nanosleep(polls < 512u ? 32 : 256);
            }
            if (((uint32_t)(st >> 32) & 3u) == kTileLost) lost = 1;
        }
        if (__syncthreads_or(lost)) return false;
        // The nearest prefix: the lowest thread that saw one.
        const bool is_prefix = mine && ((uint32_t)(st >> 32) & 3u) == kTilePrefix;
        const uint32_t bal = __ballot_sync(0xffffffffu, is_prefix);
        if (lane == 0) s_red[warp] = bal ? warp * 32u + (uint32_t)__ffs(bal) - 1u : 0xFFFFFFFFu;
        __syncthreads();
        uint32_t near = 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t w = 0; w < kCullWarps; ++w) near = min(near, s_red[w]);
        uint32_t sum = mine && threadIdx.x <= near ? (uint32_t)st : 0u;
        sum = __reduce_add_sync(0xffffffffu, sum);
        __syncthreads();
        if (lane == 0) s_red[warp] = sum;
        __syncthreads();
#pragma unroll
        for (uint32_t w = 0; w < kCullWarps; ++w) prefix += s_red[w];
        if (near != 0xFFFFFFFFu) break;
        hi = hi > kThreads ? hi - kThreads : 0u;
        __syncthreads();
    }
    return true;
}

// A wait that gave up must leave no draw count behind that covers draws nobody wrote: the draw side
// reads the count on the device. The tile that gave up stores a count of zero, marked with the launch
// in the word behind it; the last tile stores the count. Both exchange the two words as one, so that
// either the last tile gets the mark back (and then stores zeros), or the zero is stored after its
// count. No fence, and the exchange is on its way during the emission. (A fence between the count and
// a look for the mark: frames of 4,096 objects 17.3 us, 16.9 with the exchange, 16.7 without either.)
__device__ __forceinline__ unsigned long long swap_count(const VgFrameParams& P, uint32_t count, uint32_t rejected) {
    return atomicExch(reinterpret_cast<unsigned long long*>(P.counters), ((unsigned long long)rejected << 32) | count);
}
// Never the words of a finished launch, where a count of zero has nothing rejected, nor another launch's.
__device__ __forceinline__ uint32_t lost_mark(uint32_t epoch) { return 0x80000000u | epoch; }

__device__ __forceinline__ void give_up(const VgFrameParams& P, uint32_t tile, uint32_t epoch) {
    atomicOr(P.state + kVgError, (uint32_t)kDevTimeout);
    swap_count(P, 0u, lost_mark(epoch));
    st_status(P.status + tile, tile_status(epoch, kTileLost, 0u));  // the tiles after it give up too
}

// kWide: the form for large scenes, whose launch has more CTAs than fit at four per SM: they
// gain more from a fifth resident CTA than they lose to loading the cone inputs after the
// frustum test. In smaller scenes each warp's latency dominates, and the loads stay together.
//
// Bound by the latency of its dependent loads (item, object, instance, meshlet, pyramid texel)
// and by the launch. In place of a select, a test and an emission launch with the counters cleared
// before them, it took a frame (Hi-Z build included) from 29.3 to 21.7 us with 4,096 instances x 64
// meshlets at 1024x1024, from 42.1 to 31.8 with 10,000 x 100 (500 of them moved) at 1920x1080, and
// from 60.3 to 54.3 with 100,000 x 100 at 3840x2160; with the objects' world records, tiles of up
// to 512 items, the instances' records and the bounds' pairs these frames now take 16.9, 21.5 and
// 38 us.
template <bool kWide>
__global__ void __launch_bounds__(kThreads, kWide ? 5 : 4) vg_frame_kernel(const __grid_constant__ VgFrameParams P) {
    __shared__ CullView s_view;
    __shared__ TileItems s_it;
    __shared__ uint32_t s_bits[kMaxWindows + 2];  // window ballots (+2 so bit-field reads stay in bounds)
    __shared__ uint32_t s_pre[kMaxWindows];       // visible meshlets of the tile before each window
    __shared__ uint32_t s_tmp[kCullWarps + 1];
    __shared__ uint32_t s_tile, s_epoch;

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const VgSceneDev& S = P.scene;
    for (uint32_t k = tid; k < kMaxWindows + 2; k += kThreads) s_bits[k] = 0u;
    for (uint32_t k = tid; k < kMaxWindows; k += kThreads) s_it.heads[k] = 0u;
    pdl_wait();  // the kernel before may be the Hi-Z build, or the previous launch of this one
    // The object CTAs come first: they are short, and the tiles beyond the first wave start behind them.
    const uint32_t object_ctas = gridDim.x - P.num_tiles;
    const bool object_cta = blockIdx.x < object_ctas;
    if (warp == 1) view_setup_warp(P.setup, s_view);
    if (tid == 0 && !object_cta) {
        uint32_t epoch, ticket;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(epoch) : "l"(P.state + kVgEpoch) : "memory");
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(P.state + kVgTicket) : "memory");
        if (ticket == P.num_tiles - 1u) {  // the last one: every tile CTA has read the epoch
            P.state[kVgTicket] = 0u;
            P.state[kVgEpoch] = epoch + 1u;
        }
        s_tile = ticket;
        s_epoch = epoch + 1u;  // never the zeros of a fresh status
    }
    __syncthreads();
    if (object_cta) {
        object_block(P, s_view, blockIdx.x, object_ctas, s_it.off, s_tmp);
        return;
    }
    const uint32_t tile = s_tile, epoch = s_epoch;
    if (tile >= P.num_tiles) {  // uniform; only if launches of one pass ran at the same time, which they must not
        if (tid == 0) atomicOr(P.state + kVgError, (uint32_t)kDevTimeout);
        return;
    }

    // The tile's items, in rounds of one per thread: the object's selected LOD and the item's share
    // of it.
    const uint32_t w0 = tile * P.tile_items + tid;
    uint32_t n[kItemRounds], first[kItemRounds], inst[kItemRounds], lod[kItemRounds], off[kItemRounds];
#pragma unroll
    for (uint32_t r = 0; r < kItemRounds; ++r) {
        n[r] = first[r] = inst[r] = lod[r] = 0u;
        if (r * kThreads + tid >= P.tile_items || w0 + r * kThreads >= S.work_item_count) continue;
        const uint2 it = __ldca(reinterpret_cast<const uint2*>(S.items + w0 + r * kThreads));  // object, local meshlet base
        if (it.x >= S.object_count) continue;
        const HelioGpuVgObject* o = S.objects + it.x;
        const Selected sel = select_object(S, s_view, it.x);
        if (!sel.sel) continue;
        const uint32_t count = __ldca(&o->lod_meshlet_counts[sel.sel - 1u]);
        if (it.y >= count) continue;
        n[r] = min(64u, count - it.y);
        first[r] = __ldca(&o->lod_first_meshlets[sel.sel - 1u]) + it.y;
        inst[r] = sel.instance;
        lod[r] = sel.sel - 1u;
    }
    // Packed positions and ranks, a scan per round.
    uint32_t total = 0, ranks = 0;
#pragma unroll
    for (uint32_t r = 0; r < kItemRounds; ++r) {
        if (r * kThreads >= P.tile_items) break;  // uniform
        uint32_t sums;
        const uint32_t ex = tile_scan(n[r] ? (1u << 16) | n[r] : 0u, s_tmp, sums);
        off[r] = total + (ex & 0xFFFFu);
        if (n[r]) {
            const uint32_t rank = ranks + (ex >> 16);
            s_it.off[rank] = off[r];
            s_it.first[rank] = first[r];
            s_it.inst[rank] = inst[r];
            s_it.lod[rank] = (uint8_t)lod[r];
            atomicOr(s_it.heads + (off[r] >> 5), 1u << (off[r] & 31u));
            for (uint32_t w = (off[r] + 31u) >> 5; 32u * w < off[r] + n[r]; ++w) s_it.owner[w] = (uint16_t)rank;
        }
        total += sums & 0xFFFFu;
        ranks += sums >> 16;
    }
    const uint32_t windows = (total + 31u) >> 5;
    __syncthreads();

    for (uint32_t w = warp; w < windows; w += kCullWarps) {
        const uint32_t s = w * 32u + lane;
        bool vis = false;
        if (s < total) {
            const uint32_t k = item_at(s_it, w);
            const uint32_t mi = s_it.first[k] + (s - s_it.off[k]);
            if (mi < S.meshlet_count) {
                vis = meshlet_visible<false, kWide>(S, s_view, mi, s_it.inst[k]);
            }
        }
        const uint32_t bits = __ballot_sync(0xffffffffu, vis);
        if (lane == 0) s_bits[w] = bits;
    }
    __syncthreads();

    // Visible meshlets before each window, and of the tile.
    uint32_t count;
    {
        uint32_t c[kThreadWindows], sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < kThreadWindows; ++k) {
            c[k] = __popc(s_bits[kThreadWindows * tid + k]);
            sum += c[k];
        }
        uint32_t before = tile_scan(sum, s_tmp, count);
#pragma unroll
        for (uint32_t k = 0; k < kThreadWindows; ++k) {
            s_pre[kThreadWindows * tid + k] = before;
            before += c[k];
        }
    }
    if (tid == 0 && tile != P.withheld_tile)
        st_status(P.status + tile, tile_status(epoch, tile == 0u ? kTilePrefix : kTileSum, count));
    // Per-work-item visibility words: bits [off, off + n) of the tile's window bits.
#pragma unroll
    for (uint32_t r = 0; r < kItemRounds; ++r)
        if (r * kThreads + tid < P.tile_items && w0 + r * kThreads < S.work_item_count)
            reinterpret_cast<uint2*>(P.visibility)[w0 + r * kThreads] = bit_field64(s_bits, off[r], n[r]);
    const bool last = tile == P.num_tiles - 1u;
    if (count == 0u && !last) return;  // uniform: nothing to place

    uint32_t base;
    if (!tile_look_back(P, tile, epoch, s_tmp, base)) {
        if (tid == 0) give_up(P, tile, epoch);
        return;
    }
    if (tid == 0 && tile != 0u && tile != P.withheld_tile)
        st_status(P.status + tile, tile_status(epoch, kTilePrefix, base + count));
    const uint32_t all = base + count;
    unsigned long long held = 0;
    if (last && tid == 0) held = swap_count(P, all, all > P.capacity ? all - P.capacity : 0u);
    // Emission, four windows at a time per warp: their draw records are loaded before any is
    // written. (tile_look_back ended with s_pre visible to every thread.)
    __syncthreads();
    for (uint32_t wb = warp; wb < windows; wb += 4u * kCullWarps) {
        uint4 d[4];
        uint32_t b[4], mi[4], k[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t w = wb + (uint32_t)q * kCullWarps;
            b[q] = w < windows ? s_bits[w] : 0u;
            if ((b[q] >> lane) & 1u) {
                k[q] = item_at(s_it, w);
                mi[q] = s_it.first[k[q]] + (w * 32u + lane - s_it.off[k[q]]);
                d[q] = __ldca(S.m_draw + mi[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!((b[q] >> lane) & 1u)) continue;
            const uint32_t w = wb + (uint32_t)q * kCullWarps;
            const uint32_t slot = base + s_pre[w] + __popc(b[q] & ((1u << lane) - 1u));
            if (slot >= P.capacity) continue;
            uint32_t* o = reinterpret_cast<uint32_t*>(P.indirect + slot);
            o[0] = d[q].y;  // index_count
            o[1] = 1u;
            o[2] = d[q].x;  // first_index
            o[3] = d[q].z;  // vertex_offset
            o[4] = slot;    // first_instance
            reinterpret_cast<uint4*>(P.draws)[slot] = make_uint4(s_it.inst[k[q]], mi[q], s_it.lod[k[q]], 0u);
        }
    }
    if (last && tid == 0 && held == (unsigned long long)lost_mark(epoch) << 32) swap_count(P, 0u, 0u);
}

}  // namespace

void launch_instance_cull_data(const HelioGpuInstanceData* inst, uint32_t n, HelioInstanceCullData* out,
                               cudaStream_t stream) {
    if (!n) return;
    const uint32_t blocks = std::min((n + 255u) / 256u, device_sms() * 16u);
    helio_launch_begin("instance_cull_data", stream);
    instance_cull_data_kernel<<<blocks, 256, 0, stream>>>(inst, n, out);
    helio_launch_end(stream);
}

cudaError_t launch_scene_update(const SceneUpdate& u, cudaStream_t stream) {
    auto blocks = [](uint64_t n, uint32_t per) { return (uint32_t)((n + per - 1) / per); };
    const uint32_t objects = blocks(std::max(u.count, u.scene.object_count), kUpdateThreads);
    const uint32_t items = u.src_items ? blocks(u.item_count, kUpdateItems) : 0u;
    const uint32_t meshlets = u.src_meshlets ? blocks(u.meshlet_count, kUpdateMeshlets) : 0u;
    if (objects + items + meshlets == 0u) return cudaSuccess;
    helio_launch_begin("scene_update", stream);
    if (u.patch && u.names) {
        // A thread per row, and for the names at most one wave.
        const uint32_t grid = std::max(blocks(u.count, kUpdateThreads),
                                       std::min(blocks(u.scene.object_count, kUpdateThreads), 8u * device_sms()));
        const cudaError_t e = launch_after(scene_patch_kernel, grid, kUpdateThreads, 0, stream, u);
        helio_launch_end(stream);
        return e;
    }
    const cudaError_t e = launch_after(u.totals ? scene_update_kernel<true> : scene_update_kernel<false>,
                                       objects + items + meshlets, kUpdateThreads, 0, stream, u, objects, items);
    helio_launch_end(stream);
    return e;
}

cudaError_t launch_scene_update_from(SceneUpdate u, const HelioGpuInstanceData* src, uint32_t memory,
                                     const RowStaging& staging, cudaStream_t stream) {
    u.rows = src;
    const bool device = memory == HELIO_MEM_DEVICE;
    if (u.count == 0 || (device && caller_array(reads_directly, src, 16))) return launch_scene_update(u, stream);
    auto rows_in = [](const DevBuf& b) { return (uint32_t)std::min<size_t>(b.bytes / sizeof(HelioGpuInstanceData), 0xFFFFFFFFu); };
    const DevBuf* buf = &staging.kept;
    const uint32_t wanted = std::min(u.scene.object_count, kPatchStagingRows);
    if (staging.patch && u.count > rows_in(*buf) && wanted > rows_in(*buf)) {
        // Not under capture: nothing may be allocated there, and a graph must not hold a buffer that a
        // later patch may replace.
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        const cudaError_t e = cudaStreamIsCapturing(stream, &capture);
        if (e != cudaSuccess) return e;
        if (capture == cudaStreamCaptureStatusNone) {
            const cudaError_t grown = staging.patch->ensure(wanted * sizeof(HelioGpuInstanceData));
            if (grown != cudaSuccess) return grown;
            buf = staging.patch;
        }
    }
    const bool own = staging.upload_rows > rows_in(*buf);
    HelioGpuInstanceData* rows = own ? staging.upload : buf->as<HelioGpuInstanceData>();
    const uint32_t room = own ? staging.upload_rows : rows_in(*buf);
    if (!room) return cudaErrorInvalidValue;  // (a scene of at least one object has room for a row)
    const uint32_t first = u.first, count = u.count;
    uint32_t* const bounds = u.bounds;
    unsigned long long* const totals = u.totals;
    u.rows = rows;
    for (uint32_t done = 0; done < count;) {
        u.first = first + done;
        u.count = std::min(room, count - done);
        cudaError_t e = cudaMemcpyAsync(rows, src + done, (size_t)u.count * sizeof(HelioGpuInstanceData),
                                        device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, stream);
        if (e != cudaSuccess) return e;
        done += u.count;
        u.bounds = done == count ? bounds : nullptr;
        u.totals = done == count ? totals : nullptr;
        if ((e = launch_scene_update(u, stream)) != cudaSuccess) return e;
        // The first piece has copied the rest of the scene, and written the names.
        u.patch = !bounds && !totals;
        u.src_objects = nullptr;
        u.src_items = nullptr;
        u.src_meshlets = nullptr;
    }
    return cudaSuccess;
}

cudaError_t launch_vg_frame(const VgFrameParams& p, cudaStream_t stream) {
    if (!p.num_tiles) return cudaSuccess;
    const uint32_t grid = p.num_tiles + (uint32_t)(((uint64_t)p.scene.object_count + kObjectBlock - 1) / kObjectBlock);
    const bool wide = grid > 4u * device_sms();
    helio_launch_begin("vg_frame", stream);
    const cudaError_t e = launch_after(wide ? vg_frame_kernel<true> : vg_frame_kernel<false>, grid, kThreads, 0, stream, p);
    helio_launch_end(stream);
    return e;
}

}  // namespace helio
