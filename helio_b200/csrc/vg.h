// vg.h — launch parameters of the virtual-geometry kernels.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace helio {

// Device-resident scene in the layout the cull kernels read. Meshlet descriptors
// are split into three streams: bounds and cone side by side (one 32-byte load, the cone there when
// the frustum test has passed: batched meshlet tests 70.8 -> 65.6 us with 85 views, frames 39.9 ->
// 38.4 us with 100,000 objects, against two 16-byte streams), axis, draw arguments.
struct VgSceneDev {
    const float4* m_bounds;  // [2 * meshlet_count] center.xyz, radius | cone_apex.xyz, cone_cutoff
    const float4* m_axis;    // cone_axis.xyz, lod_error
    const uint4* m_draw;     // first_index, index_count, vertex_offset, instance_index
    HelioGpuVgObject* objects;
    const float4* xform;  // [6 * instance_count] InstanceXform
    const uint4* world;  // [2 * object_count] ObjectWorld, kept up to date by launch_scene_update
    const HelioGpuVgWorkItem* items;
    uint32_t meshlet_count;
    uint32_t object_count;
    uint32_t instance_count;
    uint32_t work_item_count;
};

// What the select reads of every object in every view: one 32-byte sector instead of 64 bytes
// of the object and, a round trip later, 80 of its instance. (100,000 objects in one view at
// 3840x2160: 54.3 -> 46.8 us a frame; 200,000 in 85 views: 254.8 -> 249.6 us a pass, packing
// included.)
struct ObjectWorld {
    float4 sphere;       // world centre, world radius (vg_cull.wgsl:315-318)
    float max_scale;     // of the instance
    uint32_t lod_count;  // min(lod_count, 8); 0 = never visible (no LOD, instance or valid transform)
    uint32_t instance;
    uint32_t pad;
};
static_assert(sizeof(ObjectWorld) == 32, "one sector");

// What the meshlet tests read of an instance: the affine rows of its model matrix, its
// InstanceCullData and its normal matrix in three 32-byte words, where the 144-byte
// GpuInstanceData and the cull data took eight 16-byte loads in two places. The frustum test reads
// the first two words, the cone test the third. (Meshlet tests of the batch: 73.0 -> 69.7 us with 85
// views over 200,000 objects, 94.5 -> 88.0 with 4 views over 475,000.)
struct InstanceXform {
    float4 c0;  // model column 0 (xyz), max_scale
    float4 c1;  // model column 1 (xyz), flags as bits: 1 = valid_transform, 2 = cone_cull_enabled
    float4 c2;  // model column 2 (xyz), normal column 0 x
    float4 c3;  // model column 3 (xyz), normal column 0 y
    float4 na;  // normal column 0 z, normal column 1 xyz
    float4 nb;  // normal column 2 xyz, unused
};
static_assert(sizeof(InstanceXform) == 96, "three 32-byte words");

// View constants of the select / cull stages (vg_cull.wgsl:266-280 planes; fields of
// GpuCameraUniforms) and the Hi-Z pyramid descriptor, held in shared memory.
struct CullView {
    Planes planes;
    Mat4 vp;
    float4 pos_near;
    float p00, p11;
    float focal;      // |proj[1][1]| * screen_height * 0.5 (vg_cull.wgsl:321-322)
    float lod_threshold_px;
    HizView hiz;
    uint32_t screen_height;
    uint32_t hiz_mip_count;
    uint32_t first_span;  // batches: the view's first span in the span list
    uint32_t pad;
};
static_assert(sizeof(CullView) % 16 == 0, "CullView is copied as 16-byte words");

// Inputs of a view's constants: read from the device camera.
struct ViewSetupParams {
    const HelioGpuCameraUniforms* camera;
    HizView hiz;
    uint32_t screen_height;
    uint32_t hiz_mip_count;
    float lod_threshold_px;
};

constexpr uint32_t kCullWarps = 8;        // warps per CTA
constexpr uint32_t kWindowsPerWarp = 64;  // 32 spans x 64 meshlets / 32 lanes (batch.cu)
constexpr uint32_t kMaxTileItems = 512;   // work items per CTA, at most (two per thread)

// Words of a pass's state, zero when its scene is uploaded, then kept by the kernel itself from
// launch to launch: no clearing launch precedes it.
enum : uint32_t {
    kVgTicket = 0,  // tiles handed out (zero between launches)
    kVgEpoch = 1,   // launches so far; a tile's status counts only with this launch's epoch
    kVgError = 2,   // kDevTimeout, sticky
    kVgDone = 3,    // object CTAs that have added their statistics (zero between launches)
    kVgHist = 4,    // 9 words: LOD histogram, largest lod_count (zero between launches)
    kVgStateWords = 16
};

struct VgFrameParams {
    VgSceneDev scene;
    ViewSetupParams setup;
    HelioDrawIndexedIndirectArgs* indirect;
    HelioGpuVgDraw* draws;
    uint32_t* counters;          // [counter_count], written whole by every launch; 8-byte aligned
    uint32_t* visibility;        // [2 * work_item_count]
    uint32_t* state;             // [kVgStateWords]
    unsigned long long* status;  // [num_tiles] epoch << 34 | kind << 32 | visible meshlets
    uint32_t capacity;
    uint32_t num_tiles;
    uint32_t tile_items;  // work items per tile: a power of two, 8 to kMaxTileItems
    uint32_t counter_count;
    uint32_t spin_limit;     // polls before a tile's wait gives up (kSpinLimit by default)
    uint32_t withheld_tile;  // a tile that publishes nothing (0xFFFFFFFF: none; tests only)
};

// Work items per tile: 512 for large scenes; halved for smaller ones until about one CTA
// per SM has a tile (down to 8), so that a small scene's windows spread over all SMs. The
// draw order is the item order for every choice. Measured, frames of 10,000 objects x 100 meshlets
// at 1920x1080 and of 100,000 x 100 at 3840x2160: 30.7, 26.9, 24.0 and 22.4 us with five, three, two
// and one tile per SM at the least (a tile pays its view constants, its ticket and its look-back
// once); 51.5, 44.0 and 40.2 us with at most 128, 256 and 512 items (782 tiles of 256 did not fit the
// device at once, 391 of 512 do).
constexpr uint32_t kTilesPerSm = 1;
inline uint32_t vg_tile_items(uint32_t work_items, uint32_t sms) {
    uint32_t n = kMaxTileItems;
    while (n > 8u && (uint64_t)work_items < (uint64_t)sms * kTilesPerSm * n) n >>= 1;
    return n;
}
inline uint32_t vg_tiles(uint32_t work_items, uint32_t tile_items) {
    return (uint32_t)(((uint64_t)work_items + tile_items - 1) / tile_items);
}

void launch_instance_cull_data(const HelioGpuInstanceData* inst, uint32_t n, HelioInstanceCullData* out,
                               cudaStream_t stream);

// Brings a device-resident scene up to date in one launch: copies what the caller gives in device
// memory, and derives from the instances [first, first + count) their InstanceXform and the
// ObjectWorld records of the objects that name them. A null source: the data is in the
// destination already (rows are never kept: everything reads what is derived from them).
// With `bounds` (u32[2], zero before the launch), bounds over all valid objects as float bits, for
// the batch's reject boxes: bounds[0] = largest world radius max(local_radius * max_scale, 0),
// bounds[1] = largest |c.x| + |c.y| + |c.z| of a world centre c. With `totals` (u64[3], zero before
// the launch), sums over all objects: totals[0] = lod_meshlet_counts[0], totals[1] = 64-meshlet
// spans and totals[2] = meshlets of the largest of the object's LODs.
// Objects above which a pass keeps their names: in smaller scenes the update kernel has the objects'
// fields on their way beside the rows instead of a round trip after the names.
constexpr uint32_t kPatchObjects = 65536;
struct SceneUpdate {
    VgSceneDev scene;  // object_count, instance_count, objects (written too, with src_objects) and world
    const HelioGpuInstanceData* rows;         // [count], 16-byte aligned
    const HelioGpuVgObject* src_objects;      // [object_count], 16-byte aligned
    const HelioGpuVgWorkItem* src_items;      // [item_count], 8-byte aligned
    const HelioGpuMeshletEntry* src_meshlets; // [meshlet_count], 16-byte aligned, packed into the three streams
    float4* xform;
    uint4* world;
    HelioGpuVgWorkItem* items;
    float4 *m_bounds, *m_axis;
    uint4* m_draw;
    uint32_t first, count, item_count, meshlet_count;
    // [object_count] each object's instance_index, written by an update that is no patch, or null. With it a
    // `patch` (rows only, no bounds or totals) looks for the objects to derive in 4 bytes per object
    // (kPatchObjects)
    uint32_t* names;
    bool patch;
    uint32_t* bounds;
    unsigned long long* totals;
};
cudaError_t launch_scene_update(const SceneUpdate& u, cudaStream_t stream);
// Instance rows that the update kernel does not read itself go through a staging buffer, in pieces of
// what it holds. Every piece costs a copy and a launch (4,000 rows as five pieces 75 us, 37 as one), but
// pieces of more than 4.7 MB copy no faster. A pass keeps that much from its upload on. A batch's
// scene, whose bytes count against a server's budget, keeps a fifth of its rows (with the records 285
// bytes per object, where rows and cull data took 288).
struct DevBuf;
struct RowStaging {
    DevBuf& kept;
    DevBuf* patch;  // for a patch of more rows in a small scene, allocated by the first one (null: none)
    HelioGpuInstanceData* upload;  // an upload's own, released after it, of kPatchStagingRows at most (null: none)
    uint32_t upload_rows;
};
constexpr uint32_t kMaxStagingRows = 32768;
inline uint32_t scene_staging_rows(uint32_t objects) { return std::min(std::max(objects / 5u, 1u), kMaxStagingRows); }
constexpr uint32_t kPatchStagingRows = 4096;
// The update `u` with its rows [u.first, u.first + u.count) in `src`, memory of the caller (HELIO_MEM_*),
// null if there are none. Rows of this device that 16-byte loads can read are read by the kernel.
// Others are copied to the staging piece by piece, each with an update of its own, the last with u's
// bounds and totals.
cudaError_t launch_scene_update_from(SceneUpdate u, const HelioGpuInstanceData* src, uint32_t memory,
                                     const RowStaging& staging, cudaStream_t stream);
// Object select, meshlet cull and emission of one view, in one launch.
cudaError_t launch_vg_frame(const VgFrameParams& p, cudaStream_t stream);

}  // namespace helio
