// Forward rendering of many views through a visibility buffer: the outputs of binning + raster_forward_kernel
// (raster.cu) bit for bit, without tile lists.
//
// Three launches per group of views: the triangles (one per lane) into the group's keys, the few large
// triangles a CTA at a time, and one thread per pixel that recomputes the winner's outputs and shades it.
//
// Why: the tile path lists, stages and sets up a triangle once per 16 x 16 tile it touches (2.1 times on 200k
// triangles at 1024 x 1024) behind tile barriers, after five binning launches. Here a triangle is set up once and
// a covered pixel costs one 64-bit atomicMin without a return value. Measured, tile path -> this one, fused
// forward with 3 attributes and a texture: 64 views of 200k triangles at 1024 x 1024 4.02 -> 2.84 ms (triangles
// 1.09, shading 1.67, clearing the keys 0.08), 8 views of 500k at 2048 x 1536 1.51 -> 0.83, 8 of 5k at 512 x 512
// 0.131 -> 0.117, one of 1.2k at 256 x 256 43 -> 25 us; 12 triangles filling 1024 x 1024 0.61 -> 0.07 ms, and no
// scene measured slower, so the renders take this path at every size.
//
// What bounds it: the triangles instruction issue (83% of issue slots; about 90 warp instructions per triangle,
// each multiply and add separate for the reference's rounding), the shading DRAM (5.2 TB/s: 100 bytes written per
// covered pixel) and, behind it, its chain of gathers. Checking the key before the atomic costs more than the
// atomics it saves (1.09 -> 1.39 ms).
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/pdr_capi.h"
#include "pdr_common.cuh"
#include "pdr_internal.h"
#include "tile_order.cuh"
#include "visibility.cuh"

namespace pdr {
namespace {

constexpr uint32_t kVisWarps = 4;
constexpr size_t kKeyBytes = 512u << 20;
constexpr uint32_t kShadeW = kOrderTileW, kShadeH = kOrderTileH;

// warp_triangles triangles per warp: 32, or fewer where 32 would leave the chip idle.
__global__ void __launch_bounds__(32 * kVisWarps, 10)
visibility_kernel(const float4* __restrict__ clip_all, uint32_t V, const uint3* __restrict__ idx, uint32_t T, uint32_t W,
                  uint32_t H, const float4* __restrict__ viewports, uint32_t cull, uint32_t view0,
                  uint32_t warp_triangles, unsigned long long* __restrict__ keys, uint32_t* __restrict__ queue,
                  uint32_t* __restrict__ queue_count) {
    __shared__ VisWarp warps[kVisWarps];
    VisView v;
    v.clip = clip_all + (size_t)(view0 + blockIdx.y) * V;
    v.idx = idx;
    v.V = V;
    v.T = T;
    v.W = W;
    v.H = H;
    v.cull = cull;
    v.vp = viewports[view0 + blockIdx.y];
    v.keys = keys + (size_t)blockIdx.y * W * H;
    const NdcAxis ax(v.vp.x, v.vp.z), ay(v.vp.y, v.vp.w);
    const uint32_t warp = threadIdx.x >> 5;
    vis_warp(v, ax, ay, (blockIdx.x * kVisWarps + warp) * warp_triangles, warp_triangles, warps[warp], queue_count,
             [&](uint32_t slot, uint32_t t) { queue[slot] = blockIdx.y * T + t; });
}

// Triangles with large candidate rectangles: bands of rows, enough of them to occupy the grid.
__global__ void __launch_bounds__(256)
visibility_large_kernel(const float4* __restrict__ clip_all, uint32_t V, const uint3* __restrict__ idx, uint32_t T,
                        uint32_t W, uint32_t H, const float4* __restrict__ viewports, uint32_t cull, uint32_t view0,
                        unsigned long long* __restrict__ keys, const uint32_t* __restrict__ queue,
                        const uint32_t* __restrict__ queue_count) {
    const uint32_t n = *queue_count;
    if (n == 0) return;
    const uint32_t bands = vis_bands(n);
    const uint64_t items = (uint64_t)n * bands;
    for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t entry = queue[item / bands], band = (uint32_t)(item % bands);
        const uint32_t view = entry / T;
        VisView v;
        v.clip = clip_all + (size_t)(view0 + view) * V;
        v.idx = idx;
        v.V = V;
        v.T = T;
        v.W = W;
        v.H = H;
        v.cull = cull;
        v.vp = viewports[view0 + view];
        v.keys = keys + (size_t)view * W * H;
        vis_band(v, entry - view * T, band, bands);
    }
}

// The outputs of every pixel of a group of views from its key, a CTA per tile in `order` (tile_order.cuh) or view by
// view. Images are those of all views; a pixel's index counts from their first element. CTAs that stay resident
// and load the next tile's keys ahead, which the adjoint gains from, measured slower here (1.39 -> 1.50 ms): the
// stores bound this kernel.
template <bool kDeriv, bool kShade, int kA>
__global__ void __launch_bounds__(kShadeW * kShadeH, kShade ? 12 : 16)
shade_kernel(const float4* __restrict__ clip_all, uint32_t V, const uint3* __restrict__ idx, uint32_t T, uint32_t W,
             uint32_t H, const float4* __restrict__ viewports, uint32_t view0, FastDiv tcx,
             const unsigned long long* __restrict__ keys, float4* __restrict__ raster, float4* __restrict__ deriv,
             ShadeArgs shade, FastDiv tiles, const uint32_t* __restrict__ order) {
    const uint32_t entry = order ? __ldg(order + blockIdx.x) : blockIdx.x;
    const uint32_t group_view = tiles.quotient(entry), tile = entry - group_view * tiles.divisor;
    const uint32_t ty = tcx.quotient(tile), tx = tile - ty * tcx.divisor;
    const uint32_t px = tx * kShadeW + threadIdx.x % kShadeW, py = ty * kShadeH + threadIdx.x / kShadeW;
    if (px >= W || py >= H) return;
    const size_t P = (size_t)W * H, pix = (size_t)py * W + px;
    const uint32_t view = view0 + group_view;
    RasterView v;
    v.clip = clip_all + (size_t)view * V;
    v.idx = idx;
    v.V = V;
    v.T = T;
    v.W = W;
    v.H = H;
    v.cull = 0;
    v.vp = viewports[view];
    v.raster = raster;
    v.deriv = deriv;
    v.shade = shade;
    const unsigned long long key = __ldcs(keys + group_view * P + pix);
    shade_pixel<kDeriv, kShade, kA>(v, px, py, view * P + pix, key == ~0ull ? 0u : (uint32_t)key + 1u);
}

// The bin of every tile of a group of views: the uv of a vertex of the triangle seen at the probed pixels.
__global__ void __launch_bounds__(kOrderThreads)
order_bins_kernel(const uint3* __restrict__ idx, uint32_t W, uint32_t H, FastDiv tcx, FastDiv tiles, uint32_t total,
                  uint32_t mode, const float2* __restrict__ uv_attrs, const unsigned long long* __restrict__ keys,
                  TileOrder o) {
    const size_t P = (size_t)W * H;
    order_tile(
        blockIdx.x * kOrderThreads + threadIdx.x, total, tiles, tcx, W, H, mode, o,
        [&](uint32_t view, size_t pix) {
            const unsigned long long key = __ldg(keys + view * P + pix);
            return key == ~0ull ? 0u : (uint32_t)key + 1u;
        },
        [&](uint32_t, size_t, uint32_t winner) { return __ldg(uv_attrs + idx[winner - 1].x); });
}

uint32_t group_views(uint32_t views, uint32_t W, uint32_t H) {
    const size_t per_view = (size_t)W * H * sizeof(unsigned long long);
    return (uint32_t)std::min<size_t>(std::min(views, 65535u), std::max<size_t>(1, kKeyBytes / per_view));
}

}  // namespace

namespace {

struct DirectWorkspace {
    uint32_t *queue_count, *queue;
    unsigned long long* keys;
    void* order;
    size_t bytes;
};

DirectWorkspace direct_workspace(void* base, uint32_t group, uint32_t T, uint32_t W, uint32_t H) {
    char* c = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* r = c ? c + off : nullptr;
        off += align_up(bytes);
        return r;
    };
    DirectWorkspace w{};
    const uint64_t tiles = (uint64_t)((W + kShadeW - 1) / kShadeW) * ((H + kShadeH - 1) / kShadeH) * group;
    w.queue_count = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t)));
    w.queue = reinterpret_cast<uint32_t*>(take((size_t)group * T * sizeof(uint32_t)));
    w.keys = reinterpret_cast<unsigned long long*>(take((size_t)group * W * H * sizeof(unsigned long long)));
    w.order = take(tile_order_bytes(tiles));
    w.bytes = off;
    return w;
}

__global__ void __launch_bounds__(1024) order_scan_kernel(uint32_t* __restrict__ counts) {
    // exclusive prefix sum of the kOrderBins counts, in place
    __shared__ uint32_t warp_sums[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr uint32_t kPer = (kOrderBins + 1023u) / 1024u;
    uint32_t v[kPer], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
        const uint32_t i = threadIdx.x * kPer + k;
        v[k] = i < kOrderBins ? counts[i] : 0u;
        sum += v[k];
    }
    uint32_t incl = sum;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = warp_sums[lane];
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += y;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    uint32_t at = incl - sum + (warp ? warp_sums[warp - 1] : 0u);
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
        const uint32_t i = threadIdx.x * kPer + k;
        if (i < kOrderBins) counts[i] = at;
        at += v[k];
    }
}

__global__ void __launch_bounds__(kOrderThreads) order_scatter_kernel(TileOrder o, uint32_t total) {
    __shared__ uint32_t warp_empty[kOrderThreads / 32], block_at;
    const uint32_t entry = blockIdx.x * kOrderThreads + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const bool live = entry < total;
    const uint32_t bin = live ? o.bins[entry] : 0x10000u;
    // tiles without a sample: one atomic per block
    const bool empty = live && bin == kOrderBins - 1u;
    const unsigned empties = __ballot_sync(0xffffffffu, empty);
    if (lane == 0) warp_empty[warp] = __popc(empties);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t n = 0;
        for (int w = 0; w < kOrderThreads / 32; ++w) {
            const uint32_t c = warp_empty[w];
            warp_empty[w] = n;
            n += c;
        }
        block_at = n ? atomicAdd(o.counts + kOrderBins - 1u, n) : 0u;
    }
    __syncthreads();
    if (empty) o.order[block_at + warp_empty[warp] + __popc(empties & below)] = entry;
    const unsigned peers = __match_any_sync(0xffffffffu, empty ? 0x10000u : bin);
    const int leader = __ffs(peers) - 1;
    uint32_t at = 0;
    if (live && !empty && (int)lane == leader) at = atomicAdd(o.counts + bin, (uint32_t)__popc(peers));
    at = __shfl_sync(0xffffffffu, at, leader) + __popc(peers & below);
    if (live && !empty) o.order[at] = entry;
}

}  // namespace

cudaError_t launch_order_tiles(const TileOrder& o, uint64_t tiles, cudaStream_t stream) {
    order_scan_kernel<<<1, 1024, 0, stream>>>(o.counts);
    order_scatter_kernel<<<(unsigned)((tiles + kOrderThreads - 1) / kOrderThreads), kOrderThreads, 0, stream>>>(
        o, (uint32_t)tiles);
    return cudaGetLastError();
}

size_t direct_workspace_bytes(uint32_t views, uint32_t T, uint32_t W, uint32_t H) {
    return direct_workspace(nullptr, group_views(views, W, H), T, W, H).bytes;
}

cudaError_t launch_raster_direct(const float* clip, uint32_t views, uint32_t V, const uint32_t* idx, uint32_t T,
                                 uint32_t W, uint32_t H, const float* viewports, uint32_t cull, void* workspace,
                                 float* raster, float* deriv, const RasterShade* shade, cudaStream_t stream) {
    const uint32_t group = group_views(views, W, H);
    const DirectWorkspace ws = direct_workspace(workspace, group, T, W, H);
    uint32_t *queue_count = ws.queue_count, *queue = ws.queue;
    unsigned long long* keys = ws.keys;
    const float4* c4 = reinterpret_cast<const float4*>(clip);
    const uint3* i3 = reinterpret_cast<const uint3*>(idx);
    const float4* v4 = reinterpret_cast<const float4*>(viewports);
    float4* r4 = reinterpret_cast<float4*>(raster);
    float4* d4 = reinterpret_cast<float4*>(deriv);
    const ShadeArgs sa = shade ? shade_args(*shade) : ShadeArgs{};
    const uint32_t tcx = (W + kShadeW - 1) / kShadeW, tcy = (H + kShadeH - 1) / kShadeH;
    const size_t P = (size_t)W * H;
    for (uint32_t view0 = 0; view0 < views; view0 += group) {
        const uint32_t n = std::min(group, views - view0);
        cudaError_t e = cudaMemsetAsync(queue_count, 0, sizeof(uint32_t), stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(keys, 0xff, n * P * sizeof(unsigned long long), stream);
        if (e != cudaSuccess) return e;
        // fewer triangles per warp while that leaves less than 16 warps per SM
        uint32_t per_warp = 32;
        while (per_warp > 1 && (uint64_t)((T + per_warp - 1) / per_warp) * n < (uint64_t)num_sms() * 16u) per_warp /= 2;
        const uint32_t warps = (T + per_warp - 1) / per_warp;
        visibility_kernel<<<dim3((warps + kVisWarps - 1) / kVisWarps, n), 32 * kVisWarps, 0, stream>>>(
            c4, V, i3, T, W, H, v4, cull, view0, per_warp, keys, queue, queue_count);
        visibility_large_kernel<<<(unsigned)num_sms() * 4u, 256, 0, stream>>>(c4, V, i3, T, W, H, v4, cull, view0, keys,
                                                                             queue, queue_count);
        const uint32_t tiles = tcx * tcy, total = tiles * n;
        const uint32_t* order = nullptr;
        if (shade && sa.sampled && order_pays((uint64_t)sa.tw * sa.th, n, P)) {
            const TileOrder o = tile_order_at(ws.order, total);
            e = cudaMemsetAsync(o.counts, 0, kOrderBins * sizeof(uint32_t), stream);
            if (e != cudaSuccess) return e;
            order_bins_kernel<<<(total + kOrderThreads - 1) / kOrderThreads, kOrderThreads, 0, stream>>>(
                i3, W, H, fast_div(tcx), fast_div(tiles), total, sa.mode, sa.uv_attrs, keys, o);
            e = launch_order_tiles(o, total, stream);
            if (e != cudaSuccess) return e;
            order = o.order;
        }
#define PDR_SHADE(D, S, A) \
    shade_kernel<D, S, A><<<total, kShadeW * kShadeH, 0, stream>>>(c4, V, i3, T, W, H, v4, view0, fast_div(tcx), keys, \
                                                                   r4, d4, sa, fast_div(tiles), order)
#define PDR_SHADE_A(A)            \
    case A:                       \
        if (d4)                   \
            PDR_SHADE(true, true, A); \
        else                      \
            PDR_SHADE(false, true, A); \
        break
        if (!shade) {
            if (d4) PDR_SHADE(true, false, 0); else PDR_SHADE(false, false, 0);
        } else {
            switch (sa.attr_out ? sa.A : 0u) {
                PDR_SHADE_A(0);
                PDR_SHADE_A(1);
                PDR_SHADE_A(2);
                PDR_SHADE_A(3);
                PDR_SHADE_A(4);
                PDR_SHADE_A(5);
                PDR_SHADE_A(6);
                PDR_SHADE_A(7);
                PDR_SHADE_A(8);
            }
        }
#undef PDR_SHADE_A
#undef PDR_SHADE
    }
    return cudaGetLastError();
}

}  // namespace pdr
