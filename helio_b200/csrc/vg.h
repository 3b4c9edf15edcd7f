// vg.h — launch parameters of the virtual-geometry kernels.
#pragma once

#include "common.cuh"

namespace helio {

// Device-resident scene in the layout the cull kernels read. Meshlet descriptors
// are split into four 16-byte streams so each warp load is one contiguous 512 B.
struct VgSceneDev {
    const float4* m_bounds;  // center.xyz, radius
    const float4* m_cone;    // cone_apex.xyz, cone_cutoff
    const float4* m_axis;    // cone_axis.xyz, lod_error
    const uint4* m_draw;     // first_index, index_count, vertex_offset, instance_index
    HelioGpuVgObject* objects;
    const HelioGpuInstanceData* instances;
    const HelioInstanceCullData* cull;
    const HelioGpuVgWorkItem* items;
    uint32_t meshlet_count;
    uint32_t object_count;
    uint32_t instance_count;
    uint32_t work_item_count;
};

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
    uint32_t pad[2];
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
constexpr uint32_t kMaxTileItems = 256;   // work items per CTA, at most (one per thread)

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
    uint32_t* counters;          // [counter_count], written whole by every launch
    uint32_t* visibility;        // [2 * work_item_count]
    uint32_t* state;             // [kVgStateWords]
    unsigned long long* status;  // [num_tiles] epoch << 34 | kind << 32 | visible meshlets
    uint32_t capacity;
    uint32_t num_tiles;
    uint32_t tile_items;  // work items per tile: a power of two, 8 to kMaxTileItems
    uint32_t counter_count;
};

// Work items per tile: 256 for large scenes; halved for smaller ones until about three CTAs
// per SM have a tile (down to 8), so that a small scene's windows spread over all SMs. The
// draw order is the item order for every choice.
inline uint32_t vg_tile_items(uint32_t work_items) {
    uint32_t n = kMaxTileItems;
    while (n > 8u && (uint64_t)work_items < 148ull * 3u * n) n >>= 1;
    return n;
}
inline uint32_t vg_tiles(uint32_t work_items, uint32_t tile_items) {
    return (uint32_t)(((uint64_t)work_items + tile_items - 1) / tile_items);
}

void launch_pack_meshlets(const HelioGpuMeshletEntry* aos, uint32_t n, float4* bounds, float4* cone, float4* axis,
                          uint4* draw, cudaStream_t stream);
void launch_instance_cull_data(const HelioGpuInstanceData* inst, uint32_t n, HelioInstanceCullData* out,
                               cudaStream_t stream);
// Object select, meshlet cull and emission of one view, in one launch.
cudaError_t launch_vg_frame(const VgFrameParams& p, cudaStream_t stream);

}  // namespace helio
