// shadow_device.cuh — the stages of the per-face shadow frustum cull (ShadowCullPass,
// crates/helio-pass-shadow-cull/src/lib.rs:246-328, shaders/shadow_cull.wgsl:49-96) as
// block-level device functions, shared by the standalone launches (shadow_cull.cu) and the
// batched kernel (batch.cu), which runs them as units of its own phases.
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
// The dirty faces, in ascending order, are taken 32 at a time (a chunk): lane j of every warp
// is the chunk's j-th face and holds its planes in registers, and the warp walks its 32 draws,
// whose spheres it broadcasts from shared memory. A lane thus collects its face's 32-draw
// word by itself (no ballots, one shared load per 32 tests instead of six), and two draws go
// through each packed multiply or add. A last chunk of at most 16 faces repeats them in the
// warp's other lanes, which take every second (fourth, ...) pair of draws. The test is bound by
// instruction issue (100,000 draws x 44 faces: 6.5M warp instructions, 20M with a lane per draw
// and the planes read from shared memory). Stages (no atomics on the data path):
//   test   block of 256 draws: per chunk and warp the lanes' words, per chunk the block's
//          counts, both stored lane by lane;
//   scan   per chunk: the counts become exclusive prefixes over the blocks, in place, and the
//          face totals (only where the place stage does not sum the counts itself);
//   place  block of 256 draws: each visible draw stored at the face's draws before the block +
//          before the warp + rank in the word.
#pragma once

#include "common.cuh"

namespace helio {

constexpr uint32_t kShadowFaces = HELIO_SHADOW_MAX_FACES;
constexpr uint32_t kShadowMaxPerFace = HELIO_SHADOW_MAX_DRAWS_PER_FACE;
constexpr uint32_t kShadowThreads = 256;  // draws per block; threads of every stage's block
constexpr uint32_t kShadowWarps = kShadowThreads / 32;
constexpr uint32_t kShadowChunk = 32;     // dirty faces taken at once, one per lane
constexpr uint32_t kShadowChunks = kShadowFaces / kShadowChunk;
static_assert(kShadowThreads == kShadowFaces, "one thread per face when a block lists the dirty faces");
static_assert(kShadowChunk * 6 <= kShadowThreads, "one thread per plane of a chunk");

struct ShadowDev {
    const float* matrices;  // [256][16], column-major
    const HelioGpuInstanceData* instances;
    const HelioDrawIndexedIndirectArgs* src;
    const uint32_t* face_dirty;  // [256]
    uint32_t instance_count, draw_count, blocks, words;
    uint32_t* bits;    // [kShadowChunks][words][32]: lane j = the chunk's j-th face
    uint32_t* counts;  // [kShadowChunks][blocks][32]
    HelioDrawIndexedIndirectArgs* dst;  // [256][4096]
    uint32_t* face_counts;              // [256]
};

// Shared memory of one block running a stage.
struct ShadowSmem {
    union {
        float4 pl[kShadowChunk][6];                 // test: the chunk's planes
        uint32_t word[kShadowWarps][kShadowChunk];  // test: the warps' visible counts; place: the same, or sums
    };
    float4 sphere[kShadowWarps][32];  // test: the draws' spheres, pair k in 2k: {x x y y}, 2k + 1: {z z r r}
    uint8_t active[kShadowFaces];     // the dirty faces in ascending order
    uint32_t warp[kShadowWarps];
};

// Two binary32 operations in one instruction, each correctly rounded (sm_100 packed arithmetic).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// A product of its own, as a multiply-add of a -0 that the compiler does not know: the assembler joins a
// packed multiply (also one whose -0 is a constant) and the packed addition that takes it into one
// operation with one rounding, in spite of .rn and of its switch for that, and then spheres within a
// rounding of a plane changed sides (1 of 24.8 million draw-face decisions). In constant memory, since
// the batched kernel has no register for it (as a parameter it cost that kernel 40 bytes of spills and
// 2% of its time).
static __constant__ float2 c_minus_zero = {-0.0f, -0.0f};

__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(pack2(c_minus_zero.x, c_minus_zero.y)));
    return r;
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// normalize_plane (shadow_cull.wgsl:49-55).
__device__ __forceinline__ float4 shadow_normalize(float4 p) {
    const float len = fsqrt(fadd(fadd(fmul(p.x, p.x), fmul(p.y, p.y)), fmul(p.z, p.z)));
    if (len > 1e-10f) return make_float4(fdiv(p.x, len), fdiv(p.y, len), fdiv(p.z, len), fdiv(p.w, len));
    return p;
}

// The dirty faces in ascending order into s.active; returns their number. Every thread
// of the block, of kWarps >= kShadowWarps warps, calls it.
template <uint32_t kWarps = kShadowWarps>
__device__ __forceinline__ uint32_t shadow_list_dirty(const uint32_t* face_dirty, ShadowSmem& s) {
    const uint32_t f = threadIdx.x, lane = f & 31u, warp = f >> 5;
    const bool dirty = (kWarps == kShadowWarps || f < kShadowFaces) && ld_weak(face_dirty + f) != 0u;
    const uint32_t bal = __ballot_sync(0xffffffffu, dirty);
    __syncthreads();  // the block's previous use of s is over
    if (lane == 0 && (kWarps == kShadowWarps || warp < kShadowWarps)) s.warp[warp] = __popc(bal);
    __syncthreads();
    uint32_t before = 0, n = 0;
    for (uint32_t w = 0; w < kShadowWarps; ++w) {
        if (w < warp) before += s.warp[w];
        n += s.warp[w];
    }
    if (dirty) s.active[before + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)f;
    __syncthreads();
    return n;
}

// Plane i of sphere_in_frustum (shadow_cull.wgsl:58-68) for the column-major matrix m:
// c3 + c0, c3 - c0, c3 + c1, c3 - c1, c2, c3 - c2, normalised.
__device__ __forceinline__ float4 shadow_face_plane(const float* m, uint32_t i) {
    const float4* c = reinterpret_cast<const float4*>(m);
    const float4 c3 = c[3];
    float4 p;
    if (i == 4) {
        p = c[2];
    } else {
        const float4 a = c[i == 5 ? 2 : i >> 1];
        p = (i & 1u) || i == 5 ? make_float4(fsub(c3.x, a.x), fsub(c3.y, a.y), fsub(c3.z, a.z), fsub(c3.w, a.w))
                               : make_float4(fadd(c3.x, a.x), fadd(c3.y, a.y), fadd(c3.z, a.z), fadd(c3.w, a.w));
    }
    return shadow_normalize(p);
}

// The draw's sphere; not live when the draw is skipped (outside the draw list, an
// instance index past the instance array, or r <= 0; a NaN radius goes on, as in the
// reference's `radius <= 0.0` test).
__device__ __forceinline__ float4 shadow_draw_sphere(const ShadowDev& D, uint32_t d, bool& live) {
    live = false;
    if (d >= D.draw_count) return make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t fi = ld_weak(&D.src[d].first_instance);
    if (fi >= D.instance_count) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 b = ld_weak(reinterpret_cast<const float4*>(D.instances[fi].bounds));
    live = !(b.w <= 0.0f);
    return b;
}

// The planes of a face, each component twice in a register pair.
struct ShadowPlanes {
    uint64_t x[6], y[6], z[6], w[6];
};

// Stores a draw's sphere as half of its pair.
__device__ __forceinline__ void shadow_put_sphere(float4* spheres, float4 c) {
    const uint32_t lane = threadIdx.x & 31u;
    float* p = reinterpret_cast<float*>(spheres + (lane & ~1u)) + (lane & 1u);
    p[0] = c.x;
    p[2] = c.y;
    p[4] = c.z;
    p[6] = c.w;
}

// The planes of this lane's face of the chunk [g0, g0 + nf), computed by the block (one thread
// per plane; every thread calls it).
__device__ __forceinline__ ShadowPlanes shadow_chunk_planes(const ShadowDev& D, uint32_t g0, uint32_t nf,
                                                            uint32_t width, ShadowSmem& s) {
    __syncthreads();  // the previous chunk's planes and counts are read
    if (threadIdx.x < nf * 6) {
        const uint32_t j = threadIdx.x / 6, i = threadIdx.x - j * 6;
        s.pl[j][i] = shadow_face_plane(D.matrices + 16 * s.active[g0 + j], i);
    }
    __syncthreads();
    const uint32_t j = min(threadIdx.x & (width - 1u), nf - 1u);  // lanes past the chunk repeat its last face
    ShadowPlanes p;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const float4 a = s.pl[j][k];
        p.x[k] = pack2(a.x, a.x);
        p.y[k] = pack2(a.y, a.y);
        p.z[k] = pack2(a.z, a.z);
        p.w[k] = pack2(a.w, a.w);
    }
    return p;
}

// Lanes that one face takes in a chunk of nf faces: nf rounded up to a power of two.
__device__ __forceinline__ uint32_t shadow_width(uint32_t nf) { return nf > 1u ? 1u << (32 - __clz(nf - 1u)) : 1u; }

// Bit i of the result: draw i of the warp's 32 spheres is in this lane's face: every plane
// gives !((((n.x c.x + n.y c.y) + n.z c.z) + w) + r < 0), in that order. A live draw's r is
// positive or NaN, so a distance is never -0 and a NaN distance is the canonical one, whose sign
// bit is clear: the sign bits decide. Lane j of each group of `width` lanes tests the pairs
// g, g + 32 / width, ... of its group g; the groups' bits are brought together at the end.
__device__ __forceinline__ uint32_t shadow_test_word(const ShadowPlanes& p, const float4* spheres, uint32_t width) {
    const uint32_t lane = threadIdx.x & 31u, groups = 32u / width, g = lane / width;
    uint32_t in = 0;
#pragma unroll 2
    for (uint32_t k = g; k < 16u; k += groups) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(spheres + 2u * k);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(spheres + 2u * k + 1u);
        uint32_t n0 = 0, n1 = 0;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float d0, d1;
            const uint64_t x = fmul2(p.x[i], a.x), y = fmul2(p.y[i], a.y), z = fmul2(p.z[i], b.x);
            unpack2(fadd2(fadd2(fadd2(fadd2(x, y), z), p.w[i]), b.y), d0, d1);
            n0 |= __float_as_uint(d0);
            n1 |= __float_as_uint(d1);
        }
        in |= (3u ^ ((n0 >> 31) | (n1 >> 31 << 1))) << (2u * k);
    }
    for (uint32_t d = width; d < 32u; d <<= 1) in |= __shfl_xor_sync(0xffffffffu, in, d);
    return in;
}

// Test stage of draw block `block` against the chunks c_begin, c_begin + c_step, ... Every
// thread of the block calls it.
static __device__ __noinline__ void shadow_test_block(const ShadowDev& D, uint32_t block, uint32_t c_begin,
                                                      uint32_t c_step, ShadowSmem& s) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    bool live;  // loaded while the dirty faces are listed
    const float4 sphere = shadow_draw_sphere(D, block * kShadowThreads + threadIdx.x, live);
    const uint32_t n_active = shadow_list_dirty(D.face_dirty, s);
    if (c_begin * kShadowChunk >= n_active) return;  // uniform over the block
    shadow_put_sphere(s.sphere[warp], sphere);
    const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
    for (uint32_t c = c_begin; c * kShadowChunk < n_active; c += c_step) {
        const uint32_t nf = min(kShadowChunk, n_active - c * kShadowChunk);
        const uint32_t width = shadow_width(nf);
        const ShadowPlanes p = shadow_chunk_planes(D, c * kShadowChunk, nf, width, s);
        const uint32_t all = shadow_test_word(p, s.sphere[warp], width) & live_mask;
        const uint32_t word = lane < nf ? all : 0u;
        D.bits[((size_t)c * D.words + block * kShadowWarps + warp) * 32u + lane] = word;
        __syncthreads();  // the planes are read: their region takes the counts
        s.word[warp][lane] = __popc(word);
        __syncthreads();
        if (warp == 0) {
            uint32_t n = 0;
#pragma unroll
            for (uint32_t w = 0; w < kShadowWarps; ++w) n += s.word[w][lane];
            D.counts[((size_t)c * D.blocks + block) * 32u + lane] = n;
        }
    }
}

// Counts of chunk c summed over the blocks before `block`, per face into s.word[0..7] partial
// sums (one row per warp); every thread of the block calls it. A warp reads the rows of four
// blocks with one load (a quarter-warp per row, four faces per lane), eight loads in flight.
__device__ __forceinline__ void shadow_sum_before(const ShadowDev& D, uint32_t c, uint32_t block, ShadowSmem& s) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint4* in = reinterpret_cast<const uint4*>(D.counts + (size_t)c * D.blocks * 32u) + (lane & 7u);
    uint4 n = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 8
    for (uint32_t b = warp * 4u + (lane >> 3); b < block; b += kShadowWarps * 4u) {
        const uint4 t = __ldcg(in + (size_t)b * 8u);
        n.x += t.x;
        n.y += t.y;
        n.z += t.z;
        n.w += t.w;
    }
#pragma unroll
    for (int k = 8; k < 32; k <<= 1) {
        n.x += __shfl_xor_sync(0xffffffffu, n.x, k);
        n.y += __shfl_xor_sync(0xffffffffu, n.y, k);
        n.z += __shfl_xor_sync(0xffffffffu, n.z, k);
        n.w += __shfl_xor_sync(0xffffffffu, n.w, k);
    }
    if (lane < 8u) *reinterpret_cast<uint4*>(&s.word[warp][4u * lane]) = n;
}

// Scan stage of chunk c (nothing when it holds no dirty face): counts become the draws of each
// face before each block, and the faces' totals are written. Every thread of the block of kWarps
// warps calls it; sums: a row per warp.
template <uint32_t kWarps>
static __device__ __noinline__ void shadow_scan_chunk(const ShadowDev& D, uint32_t c, ShadowSmem& s,
                                                      uint32_t (*sums)[kShadowChunk]) {
    const uint32_t n_active = shadow_list_dirty<kWarps>(D.face_dirty, s);
    if (c * kShadowChunk >= n_active) return;  // uniform over the block
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // Each warp takes a run of blocks: its sum, then its prefixes.
    const uint32_t run = (D.blocks + kWarps - 1) / kWarps;
    const uint32_t b0 = min(D.blocks, warp * run), b1 = min(D.blocks, b0 + run);
    __syncthreads();
    {
        const uint32_t* in = D.counts + (size_t)c * D.blocks * 32u + lane;
        uint32_t n = 0;
#pragma unroll 16
        for (uint32_t b = b0; b < b1; ++b) n += __ldcg(in + (size_t)b * 32u);
        sums[warp][lane] = n;
    }
    __syncthreads();
    uint32_t at = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) {
        if (w < warp) at += sums[w][lane];
        total += sums[w][lane];
    }
    uint32_t* counts = D.counts + (size_t)c * D.blocks * 32u + lane;
    uint32_t b = b0;
    for (; b + 16u <= b1; b += 16u) {
        uint32_t n[16];
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k) n[k] = __ldcg(counts + (size_t)(b + k) * 32u);
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k) {
            counts[(size_t)(b + k) * 32u] = at;
            at += n[k];
        }
    }
    for (; b < b1; ++b) {
        const uint32_t n = __ldcg(counts + (size_t)b * 32u);
        counts[(size_t)b * 32u] = at;
        at += n;
    }
    if (warp == 0 && c * kShadowChunk + lane < n_active) D.face_counts[s.active[c * kShadowChunk + lane]] = total;
}

// The counts of the clean faces are cleared (lib.rs:266-270); one block calls it.
__device__ __forceinline__ void shadow_clear_clean(const ShadowDev& D) {
    if (ld_weak(D.face_dirty + threadIdx.x) == 0u) D.face_counts[threadIdx.x] = 0u;
}

// Stores the warp's visible draws (bit i of lane j's word: draw i in face j) at lane j's `at` +
// rank, as far as the face has room. `draw` is this lane's draw, `face` lane j's face. Every lane
// calls it.
__device__ __forceinline__ void shadow_place_words(const ShadowDev& D, const HelioDrawIndexedIndirectArgs& draw,
                                                   uint32_t word, uint32_t at, uint32_t face) {
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t room = at < kShadowMaxPerFace ? kShadowMaxPerFace - at : 0u;
    uint32_t over = __popc(word);
    over = over > room ? over - room : 0u;
    for (; over; --over) word &= ~(0x80000000u >> __clz(word));  // the last draws do not fit
    const uint32_t base = face * kShadowMaxPerFace + at;
    for (uint32_t left = __ballot_sync(0xffffffffu, word != 0u); left; left &= left - 1u) {
        const int j = __ffs(left) - 1;
        const uint32_t wj = __shfl_sync(0xffffffffu, word, j), bj = __shfl_sync(0xffffffffu, base, j);
        if ((wj >> lane) & 1u) D.dst[bj + __popc(wj & lt)] = draw;
    }
}

// Place stage of draw block `block` for the chunks c_begin, c_begin + c_step, ... kScanned: the
// counts are prefixes already (shadow_scan_chunk); otherwise the block sums those before it, and
// the last block writes the faces' totals. Every thread of the block calls it.
template <bool kScanned>
static __device__ __noinline__ void shadow_place_block(const ShadowDev& D, uint32_t block, uint32_t c_begin,
                                                       uint32_t c_step, ShadowSmem& s) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t d = block * kShadowThreads + threadIdx.x;
    HelioDrawIndexedIndirectArgs draw{};
    if (d < D.draw_count) draw = D.src[d];  // loaded while the dirty faces are listed
    const uint32_t n_active = shadow_list_dirty(D.face_dirty, s);
    if (c_begin * kShadowChunk >= n_active) return;  // uniform over the block
    for (uint32_t c = c_begin; c * kShadowChunk < n_active; c += c_step) {
        const uint32_t word = __ldcg(D.bits + ((size_t)c * D.words + block * kShadowWarps + warp) * 32u + lane);
        const uint32_t before = kScanned ? __ldcg(D.counts + ((size_t)c * D.blocks + block) * 32u + lane) : 0u;
        const uint32_t face = c * kShadowChunk + lane < n_active ? s.active[c * kShadowChunk + lane] : 0u;
        // at = draws of the face before this block, then those of the block's earlier warps.
        uint32_t at = before;
        if (!kScanned) {
            __syncthreads();  // the previous chunk's table is read
            shadow_sum_before(D, c, block, s);
            __syncthreads();
#pragma unroll
            for (uint32_t w = 0; w < kShadowWarps; ++w) at += s.word[w][lane];
        }
        __syncthreads();
        s.word[warp][lane] = __popc(word);
        __syncthreads();
        const uint32_t block_at = at;
        for (uint32_t w = 0; w < warp; ++w) at += s.word[w][lane];
        if (!kScanned && block == D.blocks - 1u && warp == 0 && c * kShadowChunk + lane < n_active) {
            uint32_t total = block_at;
            for (uint32_t w = 0; w < kShadowWarps; ++w) total += s.word[w][lane];
            D.face_counts[face] = total;
        }
        shadow_place_words(D, draw, word, at, face);
    }
}

}  // namespace helio
