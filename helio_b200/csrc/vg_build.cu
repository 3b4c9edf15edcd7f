// vg_build.cu — the VG input producer: the reference's rebuild_vg_buffers
// (crates/helio/src/scene/virtual_geometry/rebuild.rs:18-58, 98-172) on the device.
//
// The reference walks the dense object slots on the host. A slot is used when its
// mesh exists and has descriptors and LODs (rebuild.rs:29-33, 121-129). Each used
// mesh's descriptors are appended once, at its first reference (rebuild.rs:25-40);
// each used slot appends one object, whose LOD ranges are offset by the mesh's base
// (rebuild.rs:135-152), one instance, ceil(max_meshlet_count / 64) work items
// (rebuild.rs:45-58) and max_meshlet_count draws of capacity (rebuild.rs:158-161).
//
// Here every append position is an exclusive prefix sum over the slots, so all
// slots are placed in parallel with the reference's order:
//   1. first_ref[m] = the smallest used slot of mesh m (atomics), and per block of 1024 slots
//      the sums that do not need it (used slots, work items, draws); the block that finishes
//      last folds the tables and adds each mesh's descriptors and first reference to the sums
//      of its first slot's block;
//   2. each block sums the blocks before it (all of them, for the totals) and places its
//      slots with one block scan: it writes its work items, and a first reference writes its
//      mesh's base and rank;
//   3. per used slot its instance and object record (the LOD offsets need its mesh's base),
//      and beside them one CTA per used mesh copies its descriptors to its base.
// Larger scenes scan the block sums in a launch of their own between 1 and 2, and larger
// libraries add the first references in one, where a single block would take too long.
// Counts, draws and LOD offsets are checked against u32 where the reference's
// checked arithmetic panics; the call then fails with HELIO_ERR_INVALID_ARG.

#include <algorithm>
#include <cstring>
#include <new>

#include "common.cuh"
#include "host_util.h"

namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kVals = 5;  // used, descriptors, work items, first references, draws
constexpr uint32_t kSub = 4;   // 256-slot sub-blocks per scan block
constexpr uint32_t kScanBlock = kSub * kThreads;  // slots per block of the slot scan
constexpr uint32_t kErrPool = 1u;    // a used mesh's descriptors leave the pool
constexpr uint32_t kErrOffset = 2u;  // an LOD descriptor offset exceeds u32

// Mesh records are read as 16-byte words (the API requires them 16-byte aligned): a
// warp's lanes usually name different meshes, so every load instruction touches up to
// 32 lines, and wide loads keep the number of such instructions down.
// (Not of the read-only path, see ld_weak; as ordinary loads they waited for the stores before them: 2M slots
// 259 -> 271 us.)
__device__ __forceinline__ uint4 mesh_word(const HelioVgMeshRecord* meshes, uint32_t m, int k) {
    return __ldca(reinterpret_cast<const uint4*>(meshes + m) + k);
}

// Word 0 of the record: first_meshlet, meshlet_count, lod_count, max_meshlet_count.
__device__ __forceinline__ bool head_used(uint4 h) { return h.y > 0u && h.z > 0u; }

__device__ __forceinline__ bool mesh_used(const HelioVgMeshRecord* meshes, uint32_t mesh_count, uint32_t m) {
    return m < mesh_count && head_used(mesh_word(meshes, m, 0));
}

__device__ __forceinline__ uint32_t item_count(uint4 h) {
    return (uint32_t)(((uint64_t)h.w + HELIO_VG_MESHLETS_PER_WORK_ITEM - 1u) / HELIO_VG_MESHLETS_PER_WORK_ITEM);
}

constexpr uint32_t kSharedMeshes = 8192;   // libraries up to this size take the shared table
constexpr uint32_t kTableWords = 8192;     // their global copies hold about this many words together
constexpr uint32_t kFoldMeshes = 4096;     // libraries up to this size are folded by the last block
constexpr uint32_t kSumBlocks = 1024;      // scenes up to this many blocks sum the blocks before each block

// Copies of the global table: several for a small library, so that the grid's atomics do not pile
// onto a few L2 lines; one for a large one, which spreads them by itself.
inline uint32_t table_copies(uint32_t mesh_count) {
    return mesh_count == 0 || mesh_count > kSharedMeshes ? 1u : std::min(32u, std::max(1u, kTableWords / mesh_count));
}

// Working storage, zero before the run.
struct BuildWork {
    uint32_t* first_ref;  // [copies][mesh_count]: ~(smallest used slot) as a running maximum, 0 = none
    uint64_t* first_sums; // [blocks][2]: descriptors and first references of the meshes first used in the block
    uint32_t* error;      // kErr* bits
    uint32_t* done;       // blocks of first_ref_kernel that have finished
    uint64_t* slot_sums;  // [blocks][3]: used slots, work items, draws (written, not zeroed)
    uint32_t copies;
    uint32_t blocks;
};

// Mesh m's first slot from the copies (folded into copy 0), and its share of the sums of that
// slot's block.
__device__ __forceinline__ void fold_mesh(const helio_vg_build_inputs& in, const BuildWork& w, uint32_t m) {
    uint32_t f = __ldcg(w.first_ref + m);
#pragma unroll 16
    for (uint32_t c = 1; c < w.copies; ++c) f = max(f, __ldcg(w.first_ref + (size_t)c * in.mesh_count + m));
    if (f == 0u) return;
    w.first_ref[m] = f;
    unsigned long long* sums = reinterpret_cast<unsigned long long*>(w.first_sums) + 2u * (size_t)(~f / kScanBlock);
    atomicAdd(sums, (unsigned long long)mesh_word(in.meshes, m, 0).y);
    atomicAdd(sums + 1, 1ull);
}

// Step 1. A block of kScanBlock slots: the smallest slot per mesh in a shared table (libraries of
// at most kSharedMeshes), pushed to copy b % copies of the global one; a global atomic is skipped
// when the table already holds an earlier slot. kFold: the last block to finish folds the copies.
template <bool kFold>
__global__ void __launch_bounds__(kThreads) first_ref_kernel(const __grid_constant__ helio_vg_build_inputs in,
                                                             const __grid_constant__ BuildWork w) {
    extern __shared__ uint32_t s_first[];
    __shared__ unsigned long long s_sum[3];
    __shared__ uint32_t s_last;
    const bool local = in.mesh_count <= kSharedMeshes;
    if (local)
        for (uint32_t k = threadIdx.x; k < in.mesh_count; k += kThreads) s_first[k] = 0u;
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0ull;
    helio::pdl_wait();
    uint32_t m[kSub];
    uint4 h[kSub];
    const uint32_t o0 = blockIdx.x * kScanBlock + threadIdx.x;
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) {
        const uint64_t o = (uint64_t)o0 + j * kThreads;
        m[j] = o < in.slot_count ? in.slot_mesh[o] : HELIO_VG_NO_MESH;
    }
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) h[j] = m[j] < in.mesh_count ? mesh_word(in.meshes, m[j], 0) : make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    uint32_t used = 0;
    unsigned long long items = 0, draws = 0;
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) {
        if (!head_used(h[j])) continue;
        if ((uint64_t)h[j].x + h[j].y > in.pool_count) atomicOr(w.error, kErrPool);
        const uint32_t key = ~(o0 + j * kThreads);
        if (local) atomicMax(s_first + m[j], key);
        else if (__ldcg(w.first_ref + m[j]) < key) atomicMax(w.first_ref + m[j], key);
        used += 1u;
        items += item_count(h[j]);
        draws += h[j].w;
    }
    used = __reduce_add_sync(0xffffffffu, used);
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
        items += __shfl_xor_sync(0xffffffffu, items, k);
        draws += __shfl_xor_sync(0xffffffffu, draws, k);
    }
    if ((threadIdx.x & 31u) == 0 && used) {
        atomicAdd(s_sum, (unsigned long long)used);
        atomicAdd(s_sum + 1, items);
        atomicAdd(s_sum + 2, draws);
    }
    __syncthreads();
    if (threadIdx.x < 3) w.slot_sums[3u * (size_t)blockIdx.x + threadIdx.x] = s_sum[threadIdx.x];
    if (local) {
        uint32_t* copy = w.first_ref + (size_t)(blockIdx.x % w.copies) * in.mesh_count;
        for (uint32_t k = threadIdx.x; k < in.mesh_count; k += kThreads) {
            const uint32_t f = s_first[k];
            if (f && __ldcg(copy + k) < f) atomicMax(copy + k, f);
        }
    }
    if (!kFold) return;
    __threadfence();  // this block's table entries before its count
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(w.done, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t k = threadIdx.x; k < in.mesh_count; k += kThreads) fold_mesh(in, w, k);
}

__global__ void __launch_bounds__(kThreads) fold_kernel(const __grid_constant__ helio_vg_build_inputs in,
                                                        const __grid_constant__ BuildWork w) {
    helio::pdl_wait();
    const uint32_t m = helio::after_wait(blockIdx.x * kThreads + threadIdx.x);
    if (m < in.mesh_count) fold_mesh(in, w, m);
}

// Position of the r-th (0-based) set bit of x; x has more than r set bits, so the
// result is in 0..31.
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t x, uint32_t r) {
    uint32_t p = 0;
#pragma unroll
    for (uint32_t w = 16; w; w >>= 1) {
        const uint32_t c = __popc(x & ((1u << w) - 1u));
        if (r >= c) {
            r -= c;
            x >>= w;
            p += w;
        }
    }
    return p;
}

// Inclusive scans of the kVals values x[k] over a block of T threads at once (one
// exchange through shared memory s[kVals][T / 32]); total[k] gets the block sums.
template <uint32_t T>
__device__ void block_scan5(uint64_t (&x)[kVals], uint64_t (*s)[T / 32], uint64_t (&total)[kVals]) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1)
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) {
            const uint64_t t = __shfl_up_sync(0xffffffffu, x[k], d);
            if (lane >= d) x[k] += t;
        }
    if (lane == 31u)
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) s[k][warp] = x[k];
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kVals; ++k) {
        uint64_t before = 0, sum = 0;
        for (uint32_t w = 0; w < T / 32u; ++w) {
            const uint64_t t = s[k][w];
            if (w < warp) before += t;
            sum += t;
        }
        x[k] += before;
        total[k] = sum;
    }
    __syncthreads();
}

// The five sums of block b: used slots, descriptors, work items, first references, draws.
__device__ __forceinline__ void block_sums(const BuildWork& w, uint32_t b, uint64_t (&x)[kVals]) {
    const uint64_t* slot = w.slot_sums + 3u * (size_t)b;
    const uint64_t* first = w.first_sums + 2u * (size_t)b;
    x[0] = __ldcg(slot);
    x[1] = __ldcg(first);
    x[2] = __ldcg(slot + 1);
    x[3] = __ldcg(first + 1);
    x[4] = __ldcg(slot + 2);
}

// One block: exclusive scan of the block sums of every value; totals[k] = the sums.
// Round r scans blocks [r T, (r + 1) T) (consecutive threads read consecutive blocks)
// and carries its sums into the next round.
constexpr uint32_t kScanThreads = 512;

__global__ void __launch_bounds__(kScanThreads) scan_blocks_kernel(const __grid_constant__ BuildWork w,
                                                                   uint64_t* block_base, uint64_t* totals) {
    __shared__ uint64_t s[kVals][kScanThreads / 32];
    helio::pdl_wait();
    uint64_t carry[kVals] = {0, 0, 0, 0, 0};
    for (uint32_t b0 = 0; b0 < w.blocks; b0 += kScanThreads) {
        const uint32_t b = b0 + threadIdx.x;
        uint64_t x[kVals] = {0, 0, 0, 0, 0}, own[kVals], total[kVals];
        if (b < w.blocks) block_sums(w, b, x);
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) own[k] = x[k];
        block_scan5<kScanThreads>(x, s, total);
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) {
            if (b < w.blocks) block_base[(size_t)b * kVals + k] = carry[k] + x[k] - own[k];
            carry[k] += total[k];
        }
    }
    if (threadIdx.x == 0)
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) totals[k] = carry[k];
}

struct BuildOut {
    HelioGpuMeshletEntry* meshlets;
    HelioGpuVgObject* objects;
    HelioGpuInstanceData* instances;
    HelioGpuVgWorkItem* items;
    uint32_t* obj_of_slot;  // [slot_count]: object index of a used slot
    uint32_t* mesh_base;    // [mesh_count]: first descriptor of a used mesh in the output
    uint32_t* mesh_order;   // [used meshes]: mesh of each first reference, in slot order
    uint64_t* totals;        // the kVals totals
    const uint32_t* error;
    uint64_t cap_objects, cap_meshlets, cap_items;  // records the output buffers hold
};

// The output passes are launched before the host has read the scan's totals, with the
// buffers the builder holds. They write only when the totals fit those buffers and the
// reference would not have stopped (a used mesh's descriptors leave the pool, or a count
// exceeds u32); otherwise every thread leaves at once and the host, after reading the
// totals, grows the buffers and runs the passes again (or reports the error).
__device__ __forceinline__ bool outputs_fit(const BuildOut& o, uint64_t objects, uint64_t descs, uint64_t items,
                                            uint64_t draws) {
    return (__ldcg(o.error) & kErrPool) == 0u && descs <= 0xFFFFFFFFull && items <= 0xFFFFFFFFull &&
           draws <= 0xFFFFFFFFull && objects <= o.cap_objects && descs <= o.cap_meshlets && items <= o.cap_items;
}

// Step 2: a block of kScanBlock slots, in four rounds of 256 so that the writes of a warp's slots
// are contiguous. Its first positions are the sums of the blocks before it (kScanned: from
// scan_blocks_kernel); the warp sums of all rounds meet behind one barrier and give every slot its
// own. Bound by latency: the sums, the slots' mesh indices, the mesh heads.
template <bool kScanned>
__global__ void __launch_bounds__(kThreads, 4) place_kernel(const __grid_constant__ helio_vg_build_inputs in,
                                                         const __grid_constant__ BuildWork w,
                                                         const uint64_t* block_base,
                                                         const __grid_constant__ BuildOut out) {
    __shared__ uint64_t s_sums[2 * kVals][kThreads / 32];
    __shared__ uint32_t s_scan[4][kSub * kThreads / 32];  // per (value, round and warp)
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    helio::pdl_wait();
    // The slots' meshes are on their way while the sums are taken.
    const uint64_t o0 = (uint64_t)blockIdx.x * kScanBlock + threadIdx.x;
    uint32_t m[kSub];
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) {
        const uint64_t o = o0 + j * kThreads;
        m[j] = o < in.slot_count ? in.slot_mesh[o] : HELIO_VG_NO_MESH;
    }
    uint64_t base[kVals], total[kVals];
    if (kScanned) {
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) {
            base[k] = __ldcg(block_base + (size_t)blockIdx.x * kVals + k);
            total[k] = __ldcg(out.totals + k);
        }
    } else {
        uint64_t before[kVals] = {0, 0, 0, 0, 0}, all[kVals] = {0, 0, 0, 0, 0};
        for (uint32_t b = threadIdx.x; b < w.blocks; b += kThreads) {
            uint64_t x[kVals];
            block_sums(w, b, x);
#pragma unroll
            for (uint32_t k = 0; k < kVals; ++k) {
                all[k] += x[k];
                if (b < blockIdx.x) before[k] += x[k];
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                before[k] += __shfl_xor_sync(0xffffffffu, before[k], d);
                all[k] += __shfl_xor_sync(0xffffffffu, all[k], d);
            }
            if (lane == 0) {
                s_sums[k][warp] = before[k];
                s_sums[kVals + k][warp] = all[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kVals; ++k) {
            base[k] = total[k] = 0;
            for (uint32_t i = 0; i < kThreads / 32; ++i) {
                base[k] += s_sums[k][i];
                total[k] += s_sums[kVals + k][i];
            }
        }
        if (blockIdx.x == 0 && threadIdx.x == 0)
#pragma unroll
            for (uint32_t k = 0; k < kVals; ++k) out.totals[k] = total[k];
    }
    if (!outputs_fit(out, total[0], total[1], total[2], total[4])) return;  // uniform over the grid
    // From here on every position fits in u32. Counts of a slot: used, descriptors and first
    // reference (if it is its mesh's first), work items.
    uint4 h[kSub];
    uint32_t fr[kSub];
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) {
        const bool ok = m[j] < in.mesh_count;
        h[j] = ok ? mesh_word(in.meshes, m[j], 0) : make_uint4(0u, 0u, 0u, 0u);
        // Through L1: past it, a small library's table is a few L2 lines that every slot asks for.
        fr[j] = ok ? __ldca(w.first_ref + m[j]) : 0u;
    }
    uint32_t ex[kSub][4];  // exclusive within the warp and round
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) {
        const bool used = head_used(h[j]), first = used && fr[j] == ~(uint32_t)(o0 + j * kThreads);
        const uint32_t v[4] = {used ? 1u : 0u, first ? h[j].y : 0u, used ? item_count(h[j]) : 0u, first ? 1u : 0u};
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            uint32_t inc = v[k];
#pragma unroll
            for (uint32_t d = 1; d < 32u; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += t;
            }
            if (lane == 31u) s_scan[k][j * (kThreads / 32) + warp] = inc;
            ex[j][k] = inc - v[k];
        }
    }
    __syncthreads();
    // Sums of the (round, warp) runs before this warp's in each round: lane i scans run i.
    static_assert(kSub * kThreads / 32 == 32, "one run per lane");
    uint32_t run[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t own = s_scan[k][lane];
        uint32_t inc = own;
#pragma unroll
        for (uint32_t d = 1; d < 32u; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += t;
        }
        run[k] = (uint32_t)base[k] + inc - own;
    }
#pragma unroll
    for (uint32_t j = 0; j < kSub; ++j) {
        uint32_t at[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) at[k] = ex[j][k] + __shfl_sync(0xffffffffu, run[k], j * (kThreads / 32) + warp);
        if (!head_used(h[j])) continue;
        const uint32_t o = (uint32_t)(o0 + j * kThreads), items = item_count(h[j]);
        out.obj_of_slot[o] = at[0];
        for (uint32_t i = 0; i < items; ++i)
            out.items[at[2] + i] = HelioGpuVgWorkItem{at[0], i * HELIO_VG_MESHLETS_PER_WORK_ITEM};
        if (fr[j] == ~o) {
            out.mesh_base[m[j]] = at[1];
            out.mesh_order[at[3]] = m[j];
        }
    }
}

// Step 3, slot CTAs: one thread per slot. A warp's used slots have consecutive object indices, so
// the warp copies their instances and writes their records as contiguous runs of 16-byte words,
// all loads of a run in flight before its first store. For the records, lane t of round r
// takes word w = t % 8 of the warp's k-th used slot (k = (32 r + t) / 8), reads that
// word of its mesh record (four whole records per load instruction) and stores it in
// place. The object record is the mesh record with word 0 replaced (object index,
// lod_count, max_meshlet_count, 0) and the LOD firsts (words 4, 5) offset by the
// mesh's base.
__device__ __forceinline__ void write_objects(const helio_vg_build_inputs& in, const BuildOut& out, uint32_t block,
                                              uint32_t* error) {
    static_assert(sizeof(HelioGpuVgObject) == 128 && sizeof(HelioVgMeshRecord) == 128, "record layouts");
    const uint64_t o = (uint64_t)block * kThreads + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t m = o < in.slot_count ? in.slot_mesh[o] : HELIO_VG_NO_MESH;
    const uint32_t obj = o < in.slot_count ? out.obj_of_slot[o] : 0u;  // undefined for unused slots
    const bool used = o < in.slot_count && mesh_used(in.meshes, in.mesh_count, m);
    const uint32_t used_mask = __ballot_sync(0xffffffffu, used);
    if (!used_mask) return;
    const uint32_t obj0 = __shfl_sync(0xffffffffu, obj, __ffs(used_mask) - 1);
    const uint32_t n_used = __popc(used_mask);
    // Lane k holds the k-th used lane: found once, then read by shuffles.
    const uint32_t nth = nth_set_bit(used_mask, min(lane, n_used - 1u));
    {
        constexpr uint32_t kW = sizeof(HelioGpuInstanceData) / 16;  // 9 words per instance
        const uint4* src = reinterpret_cast<const uint4*>(in.slot_instances) + (o - lane) * kW;
        uint4* dst = reinterpret_cast<uint4*>(out.instances + obj0);
        const uint32_t words = n_used * kW;
        uint4 x[kW];
#pragma unroll
        for (uint32_t r = 0; r < kW; ++r) {
            const uint32_t w = r * 32u + lane, k = w / kW;  // k-th used lane of the warp
            const uint32_t from = __shfl_sync(0xffffffffu, nth, k);
            if (w < words) x[r] = __ldcs(src + from * kW + (w - k * kW));
        }
#pragma unroll
        for (uint32_t r = 0; r < kW; ++r)
            if (r * 32u + lane < words) dst[r * 32u + lane] = x[r];
    }
    uint4* dst = reinterpret_cast<uint4*>(out.objects + obj0);
    const uint32_t w = lane & 7u;  // the word of the record, the same in every round
    uint4 x[8];
    uint32_t base[8];
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) {
        const uint32_t k = 4u * r + (lane >> 3);
        const uint32_t mk = __shfl_sync(0xffffffffu, m, __shfl_sync(0xffffffffu, nth, k));
        if (k >= n_used) continue;
        x[r] = mesh_word(in.meshes, mk, (int)w);
        base[r] = w == 4u || w == 5u ? __ldca(out.mesh_base + mk) : 0u;
    }
    bool over = false;
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) {
        const uint32_t k = 4u * r + (lane >> 3);
        if (k >= n_used) continue;
        uint4 q = x[r];
        if (w == 0u) {
            q = make_uint4(obj0 + k, q.z, q.w, 0u);
        } else if (w == 4u || w == 5u) {
            const uint64_t a = (uint64_t)base[r] + q.x, b = (uint64_t)base[r] + q.y, c = (uint64_t)base[r] + q.z,
                           d = (uint64_t)base[r] + q.w;
            over |= (a | b | c | d) > 0xFFFFFFFFull;
            q = make_uint4((uint32_t)a, (uint32_t)b, (uint32_t)c, (uint32_t)d);
        }
        dst[32u * r + lane] = q;
    }
    if (over) atomicOr(error, kErrOffset);
}

// Step 3, mesh CTAs: the descriptors of the used meshes in first-reference order, 4 x 16 bytes
// each, four loads per thread in flight.
__device__ __forceinline__ void copy_descriptors(const helio_vg_build_inputs& in, const BuildOut& out, uint32_t first,
                                                 uint32_t step) {
    const uint32_t used_meshes = (uint32_t)__ldcg(out.totals + 3);
    for (uint32_t r = first; r < used_meshes; r += step) {
        const uint32_t m = out.mesh_order[r];
        const uint4 h = mesh_word(in.meshes, m, 0);
        const uint4* src = reinterpret_cast<const uint4*>(in.pool + h.x);
        uint4* dst = reinterpret_cast<uint4*>(out.meshlets + out.mesh_base[m]);
        const uint64_t words = (uint64_t)h.y * 4u;
        for (uint64_t i0 = threadIdx.x; i0 < words; i0 += 4u * kThreads) {
            uint4 x[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (i0 + k * kThreads < words) x[k] = __ldca(src + i0 + k * kThreads);
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (i0 + k * kThreads < words) dst[i0 + k * kThreads] = x[k];
        }
    }
}

// The same, `group` meshes at a time: the first warp looks them up together and lays their words end
// to end, so that a library of more meshes than CTAs does not pay the chain of three look-ups once per
// mesh and CTA (200,000 slots: 50,000 meshes of 64 descriptors 228 -> 175 us, 100,000 of 2 231 -> 134;
// finding each word's mesh costs 100 meshes of 20,000 138 -> 161, so that those stay above).
constexpr uint32_t kMeshGroup = 16;  // at most

__device__ __forceinline__ void copy_descriptor_groups(const helio_vg_build_inputs& in, const BuildOut& out,
                                                       uint32_t first, uint32_t step, uint32_t group) {
    __shared__ uint64_t s_end[kMeshGroup];    // words of the group's meshes up to and with this one
    __shared__ const uint4* s_src[kMeshGroup];  // the mesh's descriptors, less the words before it
    __shared__ uint4* s_dst[kMeshGroup];
    const uint32_t used_meshes = (uint32_t)__ldcg(out.totals + 3);
    for (uint64_t r0 = (uint64_t)first * group; r0 < used_meshes; r0 += (uint64_t)step * group) {
        const uint32_t n = (uint32_t)min((uint64_t)group, used_meshes - r0);
        __syncthreads();  // the previous group's table is read
        if (threadIdx.x < 32u) {
            const uint32_t lane = threadIdx.x;
            uint4 h = make_uint4(0u, 0u, 0u, 0u);
            uint32_t base = 0;
            if (lane < n) {
                const uint32_t m = out.mesh_order[r0 + lane];
                h = mesh_word(in.meshes, m, 0);
                base = out.mesh_base[m];
            }
            const uint64_t words = 4ull * h.y;
            uint64_t end = words;
#pragma unroll
            for (uint32_t d = 1; d < kMeshGroup; d <<= 1) {
                const uint64_t t = __shfl_up_sync(0xffffffffu, end, d);
                if (lane >= d) end += t;
            }
            if (lane < n) {
                s_end[lane] = end;
                s_src[lane] = reinterpret_cast<const uint4*>(in.pool) + 4ull * h.x - (end - words);
                s_dst[lane] = reinterpret_cast<uint4*>(out.meshlets) + 4ull * base - (end - words);
            }
        }
        __syncthreads();
        const uint64_t total = s_end[n - 1u];
        for (uint64_t i0 = threadIdx.x; i0 < total; i0 += 4u * kThreads) {
            uint4 x[4];
            uint4* dst[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint64_t i = i0 + k * kThreads;
                if (i >= total) continue;
                uint32_t j = 0;  // the mesh that holds word i
                while (s_end[j] <= i) ++j;
                x[k] = __ldca(s_src[j] + i);
                dst[k] = s_dst[j] + i;
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (i0 + k * kThreads < total) *dst[k] = x[k];
        }
    }
}

// The mesh CTAs come first: a mesh may have far more descriptors than a block has slots.
template <bool kGroups>
__global__ void __launch_bounds__(kThreads) outputs_kernel(const __grid_constant__ helio_vg_build_inputs in,
                                                           const __grid_constant__ BuildOut out, uint32_t mesh_ctas,
                                                           uint32_t mesh_group, uint32_t* error) {
    helio::pdl_wait();
    if (!outputs_fit(out, __ldcg(out.totals), __ldcg(out.totals + 1), __ldcg(out.totals + 2), __ldcg(out.totals + 4)))
        return;  // uniform over the grid
    if (blockIdx.x >= mesh_ctas) write_objects(in, out, blockIdx.x - mesh_ctas, error);
    else if (kGroups) copy_descriptor_groups(in, out, blockIdx.x, mesh_ctas, mesh_group);
    else copy_descriptors(in, out, blockIdx.x, mesh_ctas);
}

}  // namespace

using helio::DevBuf;

struct helio_vg_builder {
    DevBuf work, slot_sums, block_base, obj_of_slot, mesh_base, mesh_order;
    DevBuf meshlets, objects, instances, items;
    uint32_t meshlet_count = 0, object_count = 0, item_count = 0, max_draw_count = 0;
    uint64_t runs = 0;
    bool valid = false;
};

extern "C" {

int32_t helio_vg_builder_create(helio_vg_builder** out) {
    HELIO_ARG(out, "null pointer");
    *out = new (std::nothrow) helio_vg_builder();
    if (!*out) return helio_fail(HELIO_ERR_RESOURCE, "out of host memory");
    return HELIO_OK;
}

int32_t helio_vg_builder_run(helio_vg_builder* b, const helio_vg_build_inputs* in, void* stream) {
    HELIO_ARG(b && in, "null pointer");
    HELIO_ARG(in->slot_count == 0 || (in->slot_mesh && in->slot_instances), "slot arrays missing");
    HELIO_ARG(in->mesh_count == 0 || in->meshes, "mesh records missing");
    HELIO_ARG(in->pool_count == 0 || in->pool, "descriptor pool missing");
    HELIO_ARG((reinterpret_cast<uintptr_t>(in->pool) & 15u) == 0 &&
                  (reinterpret_cast<uintptr_t>(in->meshes) & 15u) == 0 &&
                  (reinterpret_cast<uintptr_t>(in->slot_instances) & 15u) == 0,
              "pool, meshes and slot_instances must be 16-byte aligned");
    cudaStream_t s = helio::as_stream(stream);
    b->valid = false;
    const uint32_t S = in->slot_count, M = in->mesh_count;
    const uint32_t blocks = S ? (uint32_t)(((uint64_t)S + kScanBlock - 1) / kScanBlock) : 1u;  // slot-scan blocks
    // Zeroed working storage: first-reference sums | totals, error word, finished blocks | tables.
    BuildWork w{};
    w.copies = std::min(table_copies(M), blocks);
    w.blocks = blocks;
    const size_t sums_bytes = (size_t)blocks * 2 * 8, table_bytes = (size_t)M * 4 * w.copies;
    HELIO_CK(b->work.ensure(sums_bytes + (kVals + 1) * 8 + table_bytes));
    HELIO_CK(b->slot_sums.ensure((size_t)blocks * 3 * 8));
    HELIO_CK(b->block_base.ensure((size_t)blocks * kVals * 8));
    HELIO_CK(b->obj_of_slot.ensure((size_t)S * 4));
    HELIO_CK(b->mesh_base.ensure((size_t)M * 4));
    HELIO_CK(b->mesh_order.ensure((size_t)M * 4));
    w.first_sums = b->work.as<uint64_t>();
    uint64_t* totals = w.first_sums + (size_t)blocks * 2;
    w.error = reinterpret_cast<uint32_t*>(totals + kVals);
    w.done = w.error + 1;
    w.first_ref = w.done + 1;
    w.slot_sums = b->slot_sums.as<uint64_t>();
    HELIO_CK(cudaMemsetAsync(b->work.ptr, 0, sums_bytes + (kVals + 1) * 8 + table_bytes, s));
    // Launch accounting and the event profiler see one "vg_build" entry per run with
    // slots: helio_launch_end counts the first kernel, helio_launch_note each later one.
    const bool any = S > 0, scanned = blocks > kSumBlocks;
    cudaError_t e = cudaSuccess;
    if (any) {
        helio_launch_begin("vg_build", s);
        const size_t smem = M <= kSharedMeshes ? (size_t)M * 4 : 0;
        const bool fold = M <= kFoldMeshes;
        e = helio::launch_after(fold ? first_ref_kernel<true> : first_ref_kernel<false>, blocks, kThreads, smem, s, *in, w);
        if (e == cudaSuccess && !fold) {
            e = helio::launch_after(fold_kernel, (M + kThreads - 1) / kThreads, kThreads, 0, s, *in, w);
            helio_launch_note();
        }
        if (e == cudaSuccess && scanned) {
            e = helio::launch_after(scan_blocks_kernel, 1, kScanThreads, 0, s, w, b->block_base.as<uint64_t>(),
                                    totals);
            helio_launch_note();
        }
    }
    // The output passes with the buffers held now (a first run, or a larger library, finds
    // them too small: the passes then leave at once and run again below, once sized).
    auto outputs = [&]() {
        BuildOut o{b->meshlets.as<HelioGpuMeshletEntry>(), b->objects.as<HelioGpuVgObject>(),
                   b->instances.as<HelioGpuInstanceData>(), b->items.as<HelioGpuVgWorkItem>(),
                   b->obj_of_slot.as<uint32_t>(), b->mesh_base.as<uint32_t>(), b->mesh_order.as<uint32_t>(),
                   totals, w.error, 0, 0, 0};
        o.cap_objects = std::min(b->objects.bytes / sizeof(HelioGpuVgObject),
                                 b->instances.bytes / sizeof(HelioGpuInstanceData));
        o.cap_meshlets = b->meshlets.bytes / sizeof(HelioGpuMeshletEntry);
        o.cap_items = b->items.bytes / sizeof(HelioGpuVgWorkItem);
        return o;
    };
    auto launch_outputs = [&](const BuildOut& o) -> cudaError_t {
        if (!S) return cudaSuccess;
        cudaError_t r = helio::launch_after(scanned ? place_kernel<true> : place_kernel<false>, blocks, kThreads, 0, s,
                                            *in, w, b->block_base.as<uint64_t>(), o);
        helio_launch_note();
        if (r != cudaSuccess) return r;
        const uint32_t mesh_ctas = std::min(M, helio::device_sms() * 8u);
        const uint32_t mesh_group = mesh_ctas ? std::min(std::max(M / mesh_ctas, 1u), kMeshGroup) : 1u;
        r = helio::launch_after(mesh_group > 1u ? outputs_kernel<true> : outputs_kernel<false>,
                                mesh_ctas + (uint32_t)(((uint64_t)S + kThreads - 1) / kThreads), kThreads,
                                0, s, *in, o, mesh_ctas, mesh_group, w.error);
        helio_launch_note();
        return r;
    };
    const BuildOut held = outputs();
    if (e == cudaSuccess) e = launch_outputs(held);
    // The bracket ends with the last launch, before the read-back (later launches of a run
    // that had to grow its outputs are counted, not timed).
    if (any) helio_launch_end(s);
    uint64_t tot[kVals + 1] = {0};  // the totals, then the error word (and the finished blocks)
    if (e == cudaSuccess) e = cudaMemcpyAsync(tot, totals, sizeof(tot), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    uint32_t err = 0;
    std::memcpy(&err, &tot[kVals], 4);
    const char* why = e != cudaSuccess         ? cudaGetErrorString(e)
                      : (err & kErrPool)       ? "a mesh's descriptor range leaves the pool"
                      : tot[1] > 0xFFFFFFFFull ? "virtual geometry exceeds the u32 descriptor address space"
                      : tot[2] > 0xFFFFFFFFull ? "virtual geometry exceeds the u32 work-item address space"
                      : tot[4] > 0xFFFFFFFFull ? "virtual geometry indirect draw capacity exceeds u32"
                                               : nullptr;
    if (why) return helio_fail(e != cudaSuccess ? HELIO_ERR_CUDA : HELIO_ERR_INVALID_ARG, "%s", why);
    const uint64_t objects = tot[0], descriptors = tot[1], items = tot[2];
    if (objects > held.cap_objects || descriptors > held.cap_meshlets || items > held.cap_items) {
        if ((e = b->meshlets.ensure(descriptors * sizeof(HelioGpuMeshletEntry))) == cudaSuccess &&
            (e = b->objects.ensure(objects * sizeof(HelioGpuVgObject))) == cudaSuccess &&
            (e = b->instances.ensure(objects * sizeof(HelioGpuInstanceData))) == cudaSuccess)
            e = b->items.ensure(items * sizeof(HelioGpuVgWorkItem));
        if (e != cudaSuccess) return helio_fail(HELIO_ERR_CUDA, "vg_build outputs: %s", cudaGetErrorString(e));
        HELIO_CK(launch_outputs(outputs()));
        HELIO_CK(cudaMemcpyAsync(&err, w.error, 4, cudaMemcpyDeviceToHost, s));
        HELIO_CK(cudaStreamSynchronize(s));
    }
    HELIO_ARG(!(err & kErrOffset), "virtual geometry descriptor offset overflow");
    b->object_count = (uint32_t)objects;
    b->meshlet_count = (uint32_t)descriptors;
    b->item_count = (uint32_t)items;
    b->max_draw_count = (uint32_t)tot[4];
    b->runs += 1;
    b->valid = true;
    return HELIO_OK;
}

int32_t helio_vg_builder_frame_data(const helio_vg_builder* b, helio_vg_frame_data* out) {
    HELIO_ARG(b && out, "null pointer");
    HELIO_ARG(b->valid, "no successful run");
    std::memset(out, 0, sizeof(*out));
    out->meshlets = b->meshlets.as<HelioGpuMeshletEntry>();
    out->objects = b->objects.as<HelioGpuVgObject>();
    out->instances = b->instances.as<HelioGpuInstanceData>();
    out->work_items = b->items.as<HelioGpuVgWorkItem>();
    out->meshlet_count = b->meshlet_count;
    out->object_count = b->object_count;
    out->work_item_count = b->item_count;
    out->max_draw_count = b->max_draw_count;
    out->buffer_version = b->runs;
    out->instance_version = b->runs;
    out->memory = HELIO_MEM_DEVICE;
    return HELIO_OK;
}

void helio_vg_builder_destroy(helio_vg_builder* b) { delete b; }

}  // extern "C"
