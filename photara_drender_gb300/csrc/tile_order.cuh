// The order in which the 16 x 8 pixel tiles of many views are shaded, and their adjoints run, when the texture
// does not stay in L2: by the part of the texture a tile samples, over all views. In view order a view's samples
// sweep the whole texture (a view of 1024 x 1024 pixels touches 58 MB of a 4096 x 4096 atlas), so every view
// fetches its texels, and the gradient texels it adds into, from DRAM again; sorted, the views that see the same
// patch follow one another and each line is moved about once.
#pragma once

#include <cuda_runtime.h>

#include "pdr_common.cuh"
#include "pdr_internal.h"

namespace pdr {

constexpr uint32_t kOrderTileW = 16, kOrderTileH = 8;
constexpr uint32_t kOrderSide = 64;                          // texture blocks along u and v
constexpr uint32_t kOrderBins = kOrderSide * kOrderSide + 1;  // and one for tiles without a probed sample

constexpr uint64_t kOrderMinTextureBytes = 128u << 20;  // about L2

struct TileOrder {
    uint32_t* order;   // [views * tiles] view * tiles + tile, or nullptr (row-major view order)
    uint16_t* bins;    // [views * tiles]
    uint32_t* counts;  // [kOrderBins], then the bins' cursors
};

inline size_t tile_order_bytes(uint64_t tiles) {
    return align_up(tiles * sizeof(uint32_t)) + align_up(tiles * sizeof(uint16_t)) + align_up(kOrderBins * sizeof(uint32_t));
}

inline TileOrder tile_order_at(void* base, uint64_t tiles) {
    char* c = static_cast<char*>(base);
    TileOrder o;
    o.order = reinterpret_cast<uint32_t*>(c);
    c += align_up(tiles * sizeof(uint32_t));
    o.bins = reinterpret_cast<uint16_t*>(c);
    c += align_up(tiles * sizeof(uint16_t));
    o.counts = reinterpret_cast<uint32_t*>(c);
    return o;
}

// The bin of texture coordinate uv under an address mode.
__device__ __forceinline__ uint32_t order_bin(float2 uv, uint32_t mode) {
    auto block = [&](float x) -> uint32_t {
        float t = x;
        if (mode == 1) t = x - floorf(x);
        else if (mode == 2) t = fabsf(x - 2.0f * rintf(0.5f * x));
        return (uint32_t)fminf(fmaxf(t * (float)kOrderSide, 0.0f), (float)(kOrderSide - 1));  // NaN: block 0
    };
    return block(uv.y) * kOrderSide + block(uv.x);
}

// Bin, count and position of one tile, by a thread of a block of kOrderThreads: `covered(view, pixel)` gives a
// pixel's triangle + 1 or 0 (the tile's middle, else four pixels with their loads in flight together), `coordinate(view, pixel,
// covered)` its texture coordinate; the tile takes the first covered pixel's bin. Atomics on the counts: one per
// distinct bin of a warp, and one per block for the tiles without a sample, which share a bin.
constexpr int kOrderThreads = 256;

template <class Covered, class Coordinate>
__device__ __forceinline__ void order_tile(uint32_t entry, uint32_t total, FastDiv tiles, FastDiv tcx, uint32_t W,
                                           uint32_t H, uint32_t mode, const TileOrder& o, Covered&& covered,
                                           Coordinate&& coordinate) {
    constexpr int kProbes = 5;
    constexpr uint32_t at[kProbes] = {8u | 4u << 8, 3u | 1u << 8, 12u | 1u << 8, 3u | 6u << 8, 12u | 6u << 8};
    const bool live = entry < total;
    uint32_t bin = kOrderBins - 1u;
    if (live) {
        const uint32_t view = tiles.quotient(entry), tile = entry - view * tiles.divisor;
        const uint32_t ty = tcx.quotient(tile), tx = tile - ty * tcx.divisor;
        auto probe = [&](int k) {
            const uint32_t x = min(tx * kOrderTileW + (at[k] & 255u), W - 1u), y = min(ty * kOrderTileH + (at[k] >> 8), H - 1u);
            return (size_t)y * W + x;
        };
        size_t where = probe(0);
        uint32_t first = covered(view, where);
        if (!first) {
            size_t pix[kProbes];
            uint32_t hit[kProbes];
#pragma unroll
            for (int k = 1; k < kProbes; ++k) {
                pix[k] = probe(k);
                hit[k] = covered(view, pix[k]);
            }
#pragma unroll
            for (int k = kProbes - 1; k > 0; --k)
                if (hit[k]) {
                    first = hit[k];
                    where = pix[k];
                }
        }
        if (first) bin = order_bin(coordinate(view, where, first), mode);
        o.bins[entry] = (uint16_t)bin;
    }
    const uint32_t lane = threadIdx.x & 31u;
    const int empty = __syncthreads_count(live && bin == kOrderBins - 1u);
    if (threadIdx.x == 0 && empty) atomicAdd(o.counts + kOrderBins - 1u, (uint32_t)empty);
    const bool counts = live && bin != kOrderBins - 1u;
    const unsigned peers = __match_any_sync(0xffffffffu, counts ? bin : 0x10000u);
    if (counts && (peers & ((1u << lane) - 1u)) == 0u) atomicAdd(o.counts + bin, (uint32_t)__popc(peers));
}

// Scans the counts and scatters the tiles, after the caller's kernel over order_tile.
cudaError_t launch_order_tiles(const TileOrder& o, uint64_t tiles, cudaStream_t stream);

// Worth its launches (16 us for 8 views at 1024 x 1024, 60 for 64) when L2 cannot hold the texture and the views
// sample it densely enough to meet again: half a pixel per texel over all of them. Measured forward + adjoint with a
// 4096 x 4096 texture (268 MB) and views of 1024 x 1024, sorted against view order: 64 views 4.51 against 4.90 ms,
// 16 1.21 against 1.31, 8 0.675 against 0.707, 4 0.412 against 0.392; 16 views of a 2048 x 2048 one 1.143 against
// 1.130.
inline bool order_pays(uint64_t texture_texels, uint32_t views, uint64_t pixels_per_view) {
    return texture_texels * 16u >= kOrderMinTextureBytes && views > 1 && pixels_per_view * views * 2u >= texture_texels;
}

}  // namespace pdr
