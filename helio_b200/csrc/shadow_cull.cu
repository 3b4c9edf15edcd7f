// shadow_cull.cu — the per-face shadow frustum cull (ShadowCullPass,
// crates/helio-pass-shadow-cull/src/lib.rs:246-328, shaders/shadow_cull.wgsl:49-96).
//
// Per movable draw and per dirty shadow face (at most 256): the draw's instance sphere
// against the face's six planes, built from the columns of its matrix (c3 + c0,
// c3 - c0, c3 + c1, c3 - c1, c2, c3 - c2), each divided by the length of its normal
// when that exceeds 1e-10; the draw is culled when some plane gives
// (dot(n, c) + w) + r < 0, and skipped when r <= 0. The reference appends the visible
// draws of a face with an atomic counter, so their order within the face is not
// defined; here it is the draw order, and face_counts[f] counts all of them as the
// reference's counter does (only the first 4096 are stored).
//
// Stages and layout: shadow_device.cuh. Up to 2,048 draws one launch does everything, a cluster
// of 8 CTAs per chunk of 32 dirty faces; beyond that a test and a place launch, with a scan
// between them from 1,024 blocks of 256 draws on. Against three launches in every case: 2,000
// draws x 10 dirty faces 16.4 -> 6.3 us a pass, 4,188 x 19 18.4 -> 8.7, 100,000 x 44 35.5 -> 21.7.

#include <algorithm>
#include <new>

#include <cooperative_groups.h>

#include "common.cuh"
#include "host_util.h"
#include "shadow_device.cuh"
#include "shadow_host.h"

namespace helio {
namespace {

constexpr uint32_t kThreads = kShadowThreads;
constexpr uint32_t kWarps = kShadowWarps;
constexpr uint32_t kFaces = kShadowFaces;
constexpr uint32_t kChunks = kShadowChunks;

// Small draw lists in one launch: cluster y is chunk y, its CTA x takes the draws [256 x, ...), one
// per thread, and learns the counts of the CTAs before it through distributed shared memory, so
// that nothing but the results touches global memory. Bound by latency: the dirty list, the draws'
// instances and spheres, the planes and one cluster barrier. Up to 2,048 draws it takes 5.6 to 8.6
// us on the device (10 to 60 dirty faces), the two launches below 6.9 to 10.0; with several draws
// per thread it fell behind them (3,000 draws x 19 faces: 12.5 against 8.9 us).
constexpr uint32_t kClusterCtas = 8;
constexpr uint32_t kClusterDraws = kClusterCtas * kThreads;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kThreads)
    shadow_cluster_kernel(const __grid_constant__ ShadowDev D) {
    namespace cg = cooperative_groups;
    __shared__ ShadowSmem s;
    __shared__ uint32_t s_cnt[kWarps][kShadowChunk];  // visible draws per (warp, face)
    __shared__ uint32_t s_total[kShadowChunk];        // this CTA's visible draws per face
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, x = blockIdx.x, c = blockIdx.y;
    pdl_wait();
    const uint32_t d = x * kThreads + threadIdx.x;
    bool live;  // loaded while the dirty faces are listed
    const float4 sphere = shadow_draw_sphere(D, d, live);
    HelioDrawIndexedIndirectArgs draw{};
    if (d < D.draw_count) draw = D.src[d];
    const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
    const uint32_t n_active = shadow_list_dirty(D.face_dirty, s);
    if (x == 0 && c == 0) shadow_clear_clean(D);
    if (c * kShadowChunk >= n_active) return;  // uniform over the cluster
    const uint32_t nf = min(kShadowChunk, n_active - c * kShadowChunk), width = shadow_width(nf);
    shadow_put_sphere(s.sphere[warp], sphere);
    const ShadowPlanes p = shadow_chunk_planes(D, c * kShadowChunk, nf, width, s);
    uint32_t word = 0u;
    if (live_mask) word = shadow_test_word(p, s.sphere[warp], width) & live_mask;  // uniform over the warp
    if (lane >= nf) word = 0u;
    s_cnt[warp][lane] = __popc(word);
    __syncthreads();
    uint32_t at = 0;
    for (uint32_t w = 0; w < warp; ++w) at += s_cnt[w][lane];
    if (warp == kWarps - 1) s_total[lane] = at + __popc(word);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    uint32_t all = 0;
    for (uint32_t r = 0; r < kClusterCtas; ++r) {
        const uint32_t t = *cluster.map_shared_rank(s_total + lane, r);
        if (r < x) at += t;
        all += t;
    }
    cluster.sync();  // no CTA leaves while another reads its totals
    const uint32_t face = lane < nf ? s.active[c * kShadowChunk + lane] : 0u;
    if (x == 0 && warp == 0 && lane < nf) D.face_counts[face] = all;
    shadow_place_words(D, draw, word, at, face);
}

// Larger lists: test and place over (block of 256 draws) x (chunks y, y + gridDim.y, ...).
__global__ void __launch_bounds__(kThreads) shadow_test_kernel(const __grid_constant__ ShadowDev D) {
    __shared__ ShadowSmem s;
    pdl_wait();
    shadow_test_block(D, blockIdx.x, blockIdx.y, gridDim.y, s);
}

// A CTA per chunk, as wide as it can be: a warp's run of blocks is a chain of round trips (a million
// draws x 1 face through all three launches 86 us with 8 warps and 8 rows in flight, 59 with 32 and 16).
constexpr uint32_t kScanWarps = 32;

__global__ void __launch_bounds__(kScanWarps * 32) shadow_scan_kernel(const __grid_constant__ ShadowDev D) {
    __shared__ ShadowSmem s;
    __shared__ uint32_t s_sums[kScanWarps][kShadowChunk];
    pdl_wait();
    shadow_scan_chunk<kScanWarps>(D, blockIdx.x, s, s_sums);
}

template <bool kScanned>
__global__ void __launch_bounds__(kThreads) shadow_place_kernel(const __grid_constant__ ShadowDev D) {
    __shared__ ShadowSmem s;
    pdl_wait();
    if (blockIdx.x == 0 && blockIdx.y == 0) shadow_clear_clean(D);
    shadow_place_block<kScanned>(D, blockIdx.x, blockIdx.y, gridDim.y, s);
}

// Blocks up to which each place block sums the counts before it (128 bytes per block and chunk):
// about 1,000 such sums cost less than the scan's launch; the work grows with the square.
constexpr uint32_t kSumBlocks = 1024;

cudaError_t launch_shadow(const ShadowDev& D, cudaStream_t s) {
    if (D.draw_count <= kClusterDraws) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterCtas, kChunks);
        cfg.blockDim = dim3(kThreads);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, shadow_cluster_kernel, D);
    }
    // One CTA takes all chunks of its draws when the blocks alone fill the device; below that the
    // chunks are shared out, so that a CTA's chain of loads and planes is not repeated per chunk.
    const dim3 grid(D.blocks, std::max(1u, std::min(kChunks, device_sms() * 6u / D.blocks)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, shadow_test_kernel, D);
    if (e != cudaSuccess) return e;
    helio_launch_note();
    if (D.blocks > kSumBlocks) {
        cfg.gridDim = dim3(kChunks);
        cfg.blockDim = dim3(kScanWarps * 32);
        e = cudaLaunchKernelEx(&cfg, shadow_scan_kernel, D);
        if (e != cudaSuccess) return e;
        helio_launch_note();
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kThreads);
        return cudaLaunchKernelEx(&cfg, shadow_place_kernel<true>, D);
    }
    return cudaLaunchKernelEx(&cfg, shadow_place_kernel<false>, D);
}

}  // namespace
}  // namespace helio

using helio::DevBuf;

struct helio_shadow_cull_pass {
    DevBuf dst, counts, bits, block_counts;
    helio_shadow_cull_inputs in{};
    uint32_t blocks = 0, words = 0;
    bool prepared = false;
};

bool helio::shadow_dev(const helio_shadow_cull_pass* p, ShadowDev* out) {
    if (!p || !p->prepared || p->in.face_count == 0 || p->in.draw_count == 0) return false;
    ShadowDev D{};
    D.matrices = p->in.shadow_matrices;
    D.instances = p->in.instances;
    D.src = p->in.src_indirect;
    D.face_dirty = p->in.face_dirty;
    D.instance_count = p->in.instance_count;
    D.draw_count = p->in.draw_count;
    D.blocks = p->blocks;
    D.words = p->words;
    D.bits = p->bits.as<uint32_t>();
    D.counts = p->block_counts.as<uint32_t>();
    D.dst = p->dst.as<HelioDrawIndexedIndirectArgs>();
    D.face_counts = p->counts.as<uint32_t>();
    *out = D;
    return true;
}

extern "C" {

int32_t helio_shadow_cull_create(helio_shadow_cull_pass** out) {
    HELIO_ARG(out, "null pointer");
    *out = nullptr;
    helio_shadow_cull_pass* p = new (std::nothrow) helio_shadow_cull_pass();
    if (!p) return helio_fail(HELIO_ERR_RESOURCE, "out of host memory");
    // lib.rs:104-117: 256 faces x 4096 draws of 20 bytes, and 256 counts.
    constexpr size_t F = HELIO_SHADOW_MAX_FACES;
    cudaError_t e = p->dst.ensure(F * HELIO_SHADOW_MAX_DRAWS_PER_FACE * sizeof(HelioDrawIndexedIndirectArgs));
    if (e == cudaSuccess) e = p->counts.ensure(F * 4);
    if (e == cudaSuccess) e = cudaMemset(p->counts.ptr, 0, F * 4);
    if (e != cudaSuccess) {
        delete p;
        return helio_fail(HELIO_ERR_CUDA, "shadow cull buffers: %s", cudaGetErrorString(e));
    }
    *out = p;
    return HELIO_OK;
}

int32_t helio_shadow_cull_prepare(helio_shadow_cull_pass* p, const helio_shadow_cull_inputs* in) {
    HELIO_ARG(p && in, "null pointer");
    HELIO_ARG(in->face_count == 0 || in->draw_count == 0 || (in->shadow_matrices && in->face_dirty),
              "shadow matrices and face dirty words missing");
    HELIO_ARG(in->draw_count == 0 || (in->src_indirect && (in->instances || in->instance_count == 0)),
              "draws or instances missing");
    HELIO_ARG((reinterpret_cast<uintptr_t>(in->shadow_matrices) & 15u) == 0 &&
                  (reinterpret_cast<uintptr_t>(in->instances) & 15u) == 0,
              "shadow_matrices and instances must be 16-byte aligned");
    const uint32_t blocks = (uint32_t)(((uint64_t)in->draw_count + helio::kThreads - 1) / helio::kThreads);
    const uint32_t words = blocks * helio::kWarps;
    constexpr size_t F = HELIO_SHADOW_MAX_FACES;
    HELIO_CK(p->bits.ensure(F * words * 4));
    HELIO_CK(p->block_counts.ensure(F * blocks * 4));
    p->in = *in;
    p->blocks = blocks;
    p->words = words;
    p->prepared = true;
    return HELIO_OK;
}

int32_t helio_shadow_cull_execute(helio_shadow_cull_pass* p, void* stream) {
    HELIO_ARG(p, "null pointer");
    HELIO_ARG(p->prepared, "pass not prepared");
    if (p->in.face_count == 0 || p->in.draw_count == 0) return HELIO_OK;  // lib.rs:261-263
    cudaStream_t s = helio::as_stream(stream);
    helio::ShadowDev D{};
    helio::shadow_dev(p, &D);
    helio_launch_begin("shadow_cull", s);
    const cudaError_t e = helio::launch_shadow(D, s);
    helio_launch_end(s);
    HELIO_CK(e);
    HELIO_CK(cudaGetLastError());
    return HELIO_OK;
}

int32_t helio_shadow_cull_publish(const helio_shadow_cull_pass* p, helio_shadow_cull_outputs* out) {
    HELIO_ARG(p && out, "null pointer");
    out->face_indirect = p->dst.as<HelioDrawIndexedIndirectArgs>();
    out->face_counts = p->counts.as<uint32_t>();
    out->max_faces = HELIO_SHADOW_MAX_FACES;
    out->max_draws_per_face = HELIO_SHADOW_MAX_DRAWS_PER_FACE;
    return HELIO_OK;
}

void helio_shadow_cull_destroy(helio_shadow_cull_pass* p) { delete p; }

}  // extern "C"
