// hiz_tile.cuh — one 64x64 tile of the fused Hi-Z build (levels 0..6) and the
// per-view tail (levels 7..), shared by the standalone Hi-Z kernels and the
// persistent multi-view kernel.
//
// Reference: crates/helio-pass-hiz/shaders/hiz_depth_copy.wgsl:13-19 (level 0 copy)
// and hiz_build.wgsl:12-23 (dst = max(1, dim >> (m+1)); the +1 neighbours are
// clamped to src_size - 1, so odd sizes drop the last row / column).
//
//   * four warps own a 64x64 tile of level 0, one 32x32 quadrant each: registers and
//     shuffles give levels 1..5, the quadrants' level-5 texels level 6;
//   * levels 7.. come from level 6 in the same way (a warp reduces a 32x32 quadrant of
//     level 6 to level 11, the last one), once every tile of the view is done (an atomic
//     ticket, or the caller's barrier).
// Every level-l texel is exactly max() over a rectangle of level 0 (max is exact)
// and each 2x2 step applies the reference's clamp rule (a source dimension of 1
// reuses the same texel), so the result is bit-identical to the per-level chain.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace helio {

// One 2x2 step of hiz_build.wgsl: a=(2x,2y) b=(2x+1,2y) c=(2x,2y+1) d=(2x+1,2y+1);
// a source dimension of 1 clamps the +1 neighbour back onto the same texel.
__device__ __forceinline__ float hiz_red4(float a, float b, float c, float d, bool xc, bool yc) {
    if (xc) {
        b = a;
        d = c;
    }
    if (yc) {
        c = a;
        d = b;
    }
    return fmaxf(fmaxf(a, b), fmaxf(c, d));
}

// ── Warp per 32x32 quadrant ─────────────────────────────────────────────────
// Warp q (0..3; q = 2 * row + column) of a tile reduces quadrant q alone: lane l holds
// the 8-row x 4-column block at quadrant column 4 (l % 8), row 8 (l / 8); registers give
// levels 1 and 2, shuffles levels 3..5, and the four quadrants' level-5 texels give
// level 6 (hiz_quad_level6, one thread, after a barrier). Each 2x2 step takes its texels
// in the reference's order (top-left, top-right, bottom-left, bottom-right) through hiz_red4.

// Level 0 of the lane's 8x4 block of quadrant q of tile `tile` from global memory;
// outside the image the block reads 0 (those texels are never used).
__device__ __forceinline__ void hiz_quad_load(const HizJob& J, uint32_t tile, int q, float (&v)[8][4]) {
    const int lane = threadIdx.x & 31;
    const uint32_t tile_y = tile / J.tiles_x, tile_x = tile - tile_y * J.tiles_x;
    const uint32_t bx = tile_x * kHizTile + 32u * (q & 1) + 4u * (lane & 7);
    const uint32_t by = tile_y * kHizTile + 32u * (q >> 1) + 8u * (lane >> 3);
    const uint32_t W = J.lw[0], H = J.lh[0];
    const bool aligned = ((J.depth_pitch & 3u) == 0u) && ((reinterpret_cast<uintptr_t>(J.depth) & 15u) == 0u);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float* row = J.depth + (size_t)(by + r) * J.depth_pitch + bx;
        if (aligned && bx + 4 <= W && by + r < H) {
            const float4 x = __ldcs(reinterpret_cast<const float4*>(row));
            v[r][0] = x.x;
            v[r][1] = x.y;
            v[r][2] = x.z;
            v[r][3] = x.w;
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) v[r][c] = (bx + c < W && by + r < H) ? __ldcs(row + c) : 0.0f;
        }
    }
}

// Level 0 of the lane's 8x4 block of quadrant q of the tile at (X0, Y0) into the pyramid,
// when the job does not alias it.
__device__ __forceinline__ void hiz_quad_copy0(const HizJob& J, uint32_t X0, uint32_t Y0, int q,
                                               const float (&v)[8][4]) {
    if (!J.copy_mip0) return;
    const int lane = threadIdx.x & 31;
    const uint32_t bx = X0 + 32u * (q & 1) + 4u * (lane & 7), by = Y0 + 32u * (q >> 1) + 8u * (lane >> 3);
    const uint32_t W = J.lw[0], H = J.lh[0], p0 = J.lpitch[0];
    float* L0 = J.levels[0];
    const bool al0 = ((p0 & 3u) == 0u) && ((reinterpret_cast<uintptr_t>(L0) & 15u) == 0u);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        if (by + r >= H) break;
        float* row = L0 + (size_t)(by + r) * p0 + bx;
        if (al0 && bx + 4 <= W) {
            *reinterpret_cast<float4*>(row) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (bx + c < W) row[c] = v[r][c];
        }
    }
}

// Stores texel (x, y) of level l when it lies inside the level.
__device__ __forceinline__ void hiz_put(const HizJob& J, int l, uint32_t x, uint32_t y, float m) {
    if (x < J.lw[l] && y < J.lh[l]) J.levels[l][(size_t)y * J.lpitch[l] + x] = m;
}

// Levels kBase + 1 .. kBase + 5 of the 32x32 quadrant of level kBase whose first texel is
// (QX, QY) from the lane's 8x4 block v (lane = 8 * block row + block column); returns the
// quadrant's level kBase + 5 texel in lane 0. Every lane of the warp calls it.
template <int kBase>
__device__ __forceinline__ float hiz_quad_levels(const HizJob& J, uint32_t QX, uint32_t QY, const float (&v)[8][4]) {
    const int lane = threadIdx.x & 31, lx = lane & 7, ly = lane >> 3;
    // First level: 4 rows x 2 columns per lane.
    float m1[4][2];
    {
        const bool xc = J.lw[kBase] == 1u, yc = J.lh[kBase] == 1u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                m1[j][i] = hiz_red4(v[2 * j][2 * i], v[2 * j][2 * i + 1], v[2 * j + 1][2 * i],
                                    v[2 * j + 1][2 * i + 1], xc, yc);
        const uint32_t x1 = (QX >> 1) + 2u * lx, y1 = (QY >> 1) + 4u * ly;
        float* L1 = J.levels[kBase + 1];
        const uint32_t p1 = J.lpitch[kBase + 1];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (y1 + j >= J.lh[kBase + 1]) break;
            float* row = L1 + (size_t)(y1 + j) * p1 + x1;
            if (x1 + 2 <= J.lw[kBase + 1] && ((p1 & 1u) == 0u)) {
                *reinterpret_cast<float2*>(row) = make_float2(m1[j][0], m1[j][1]);
            } else {
                if (x1 < J.lw[kBase + 1]) row[0] = m1[j][0];
                if (x1 + 1 < J.lw[kBase + 1]) row[1] = m1[j][1];
            }
        }
    }
    if (J.mip_count <= kBase + 2) return 0.0f;
    // Second: 2 rows x 1 column per lane.
    float m2[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        m2[j] = hiz_red4(m1[2 * j][0], m1[2 * j][1], m1[2 * j + 1][0], m1[2 * j + 1][1], J.lw[kBase + 1] == 1u,
                         J.lh[kBase + 1] == 1u);
        hiz_put(J, kBase + 2, (QX >> 2) + lx, (QY >> 2) + 2u * ly + j, m2[j]);
    }
    if (J.mip_count <= kBase + 3) return 0.0f;
    // Third: the right neighbour is lane + 1 (lanes with an even block column).
    const float r0 = __shfl_xor_sync(0xffffffffu, m2[0], 1);
    const float r1 = __shfl_xor_sync(0xffffffffu, m2[1], 1);
    const float m3 = hiz_red4(m2[0], r0, m2[1], r1, J.lw[kBase + 2] == 1u, J.lh[kBase + 2] == 1u);
    if ((lx & 1) == 0) hiz_put(J, kBase + 3, (QX >> 3) + (lx >> 1), (QY >> 3) + ly, m3);
    if (J.mip_count <= kBase + 4) return 0.0f;
    // Fourth: right = lane + 2, below = lane + 8 (lanes with block column % 4 == 0 and an
    // even block row).
    const float b4 = __shfl_xor_sync(0xffffffffu, m3, 2);
    const float c4 = __shfl_xor_sync(0xffffffffu, m3, 8);
    const float d4 = __shfl_xor_sync(0xffffffffu, m3, 10);
    const float m4 = hiz_red4(m3, b4, c4, d4, J.lw[kBase + 3] == 1u, J.lh[kBase + 3] == 1u);
    if ((lx & 3) == 0 && (ly & 1) == 0) hiz_put(J, kBase + 4, (QX >> 4) + (lx >> 2), (QY >> 4) + (ly >> 1), m4);
    if (J.mip_count <= kBase + 5) return 0.0f;
    // Fifth: right = lane + 4, below = lane + 16 (lane 0).
    const float b5 = __shfl_xor_sync(0xffffffffu, m4, 4);
    const float c5 = __shfl_xor_sync(0xffffffffu, m4, 16);
    const float d5 = __shfl_xor_sync(0xffffffffu, m4, 20);
    const float m5 = hiz_red4(m4, b5, c5, d5, J.lw[kBase + 4] == 1u, J.lh[kBase + 4] == 1u);
    if (lane == 0) hiz_put(J, kBase + 5, QX >> 5, QY >> 5, m5);
    return m5;
}

// Levels 1..5 of quadrant q of the tile at (X0, Y0).
__device__ __forceinline__ float hiz_quad_levels(const HizJob& J, uint32_t X0, uint32_t Y0, int q,
                                                 const float (&v)[8][4]) {
    return hiz_quad_levels<0>(J, X0 + 32u * (uint32_t)(q & 1), Y0 + 32u * (uint32_t)(q >> 1), v);
}

// Level 6 of tile t from its four quadrants' level-5 texels (one thread).
__device__ __forceinline__ void hiz_quad_level6(const HizJob& J, uint32_t t, const float* l5) {
    const uint32_t ty = t / J.tiles_x, tx = t - ty * J.tiles_x;
    hiz_put(J, 6, tx, ty, hiz_red4(l5[0], l5[1], l5[2], l5[3], J.lw[5] == 1u, J.lh[5] == 1u));
}

// ── Levels 7.. ──────────────────────────────────────────────────────────────
// From level 6 by `warps` warps (this one is warp `w`; every lane calls it), a 32x32 quadrant
// of level 6 per warp and round: the quadrant's levels 7..11 need no other quadrant, so the
// warps do not wait for each other and a quadrant costs one round trip. (Level by level with a
// barrier in between, as before, each level cost 0.3 to 0.5 us however few its texels.) Level 6
// was written by other CTAs and is read through L2. mip_count > 7.
static_assert(HELIO_HIZ_MAX_MIPS <= 12, "a quadrant of level 6 ends at level 11");

static __device__ __forceinline__ void hiz_tail(const HizJob& J, uint32_t w, uint32_t warps) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t W = J.lw[6], H = J.lh[6], P = J.lpitch[6];
    const uint32_t qw = (W + 31u) / 32u, quads = qw * ((H + 31u) / 32u);
    for (uint32_t q = w; q < quads; q += warps) {
        const uint32_t qy = q / qw, QX = 32u * (q - qy * qw), QY = 32u * qy;
        const uint32_t bx = QX + 4u * (lane & 7u), by = QY + 8u * (lane >> 3);
        float v[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float* row = J.levels[6] + (size_t)(by + r) * P + bx;
            if (bx + 4 <= W && by + r < H) {  // rows of every level start 16-byte aligned
                const float4 x = __ldcg(reinterpret_cast<const float4*>(row));
                v[r][0] = x.x;
                v[r][1] = x.y;
                v[r][2] = x.z;
                v[r][3] = x.w;
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) v[r][c] = (bx + c < W && by + r < H) ? __ldcg(row + c) : 0.0f;
            }
        }
        hiz_quad_levels<6>(J, QX, QY, v);
    }
}

// The same as a call of its own (callers that keep few registers live across it).
static __device__ __noinline__ void hiz_tail_call(const HizJob& J, uint32_t w, uint32_t warps) {
    hiz_tail(J, w, warps);
}

// ── One tile per CTA of 4 warps ───────────────────────────────────────────────
constexpr uint32_t kHizBlockThreads = 128;

// Tile `tile` (flat index within job J) by the CTA's four warps; the CTA that takes the view's
// last ticket builds levels 7.. and leaves the ticket at zero. Thread 0 writes the tile's level-6
// texel, and its acquire-release add publishes it and, in the last CTA, sees every other one's.
// The level-0 copy follows the ticket, which therefore does not wait for those stores.
static __device__ __forceinline__ void hiz_tile_block(const HizJob& J, uint32_t tile, uint32_t* ticket) {
    __shared__ float s_l5[4];
    __shared__ uint32_t s_last;
    const int q = (int)(threadIdx.x >> 5);
    const uint32_t ty = tile / J.tiles_x, tx = tile - ty * J.tiles_x;
    const uint32_t X0 = tx * kHizTile, Y0 = ty * kHizTile;
    float v[8][4];
    hiz_quad_load(J, tile, q, v);
    if (J.mip_count > 1) {
        const float m5 = hiz_quad_levels(J, X0, Y0, q, v);
        if ((threadIdx.x & 31u) == 0u) s_l5[q] = m5;
    }
    if (J.mip_count > 6) {
        __syncthreads();
        if (threadIdx.x == 0) {
            hiz_quad_level6(J, tile, s_l5);
            if (J.mip_count > 7) {
                uint32_t old;
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(ticket) : "memory");
                const uint32_t last = (old + 1u == J.tiles_x * J.tiles_y) ? 1u : 0u;
                if (last) *ticket = 0u;  // every other tile of this job has taken its ticket
                s_last = last;
            }
        }
    }
    hiz_quad_copy0(J, X0, Y0, q, v);
    if (J.mip_count <= 7) return;
    __syncthreads();
    if (s_last) hiz_tail(J, (uint32_t)q, 4u);
}

}  // namespace helio
