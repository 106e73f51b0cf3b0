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
#include "visibility.cuh"

namespace pdr {
namespace {

constexpr uint32_t kVisWarps = 4;
constexpr size_t kKeyBytes = 512u << 20;
constexpr uint32_t kShadeW = 16, kShadeH = 8;

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
    vis_warp(v, ax, ay, (blockIdx.x * kVisWarps + warp) * warp_triangles, warp_triangles, warps[warp], queue, queue_count,
             blockIdx.y * T);
}

// Triangles with large candidate rectangles: bands of rows, enough of them to occupy the grid.
__global__ void __launch_bounds__(256)
visibility_large_kernel(const float4* __restrict__ clip_all, uint32_t V, const uint3* __restrict__ idx, uint32_t T,
                        uint32_t W, uint32_t H, const float4* __restrict__ viewports, uint32_t cull, uint32_t view0,
                        unsigned long long* __restrict__ keys, const uint32_t* __restrict__ queue,
                        const uint32_t* __restrict__ queue_count) {
    const uint32_t n = *queue_count;
    if (n == 0) return;
    const uint32_t bands = min(64u, max(1u, 4u * gridDim.x / n));
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
        const NdcAxis ax(v.vp.x, v.vp.z), ay(v.vp.y, v.vp.w);
        VisTriangle t;
        if (!vis_setup(v, ax, ay, entry - view * T, t)) continue;
        const uint64_t rows = t.y1 - t.y0 + 1u;
        vis_rows(v, ax, ay, t, (uint32_t)(rows * band / bands), (uint32_t)(rows * (band + 1u) / bands));
    }
}

// The outputs of every pixel of a group of views from its key.
template <bool kDeriv, bool kShade, int kA>
__global__ void __launch_bounds__(kShadeW * kShadeH, kShade ? 12 : 16)
shade_kernel(const float4* __restrict__ clip_all, uint32_t V, const uint3* __restrict__ idx, uint32_t T, uint32_t W,
             uint32_t H, const float4* __restrict__ viewports, uint32_t view0, uint32_t tcx,
             const unsigned long long* __restrict__ keys, float4* __restrict__ raster, float4* __restrict__ deriv,
             ShadeArgs shade) {
    const uint32_t view = view0 + blockIdx.y;
    const uint32_t ty = blockIdx.x / tcx, tx = blockIdx.x - ty * tcx;
    const uint32_t px = tx * kShadeW + threadIdx.x % kShadeW, py = ty * kShadeH + threadIdx.x / kShadeW;
    if (px >= W || py >= H) return;
    const size_t P = (size_t)W * H, pix = (size_t)py * W + px;
    RasterView v;
    v.clip = clip_all + (size_t)view * V;
    v.idx = idx;
    v.V = V;
    v.T = T;
    v.W = W;
    v.H = H;
    v.cull = 0;
    v.vp = viewports[view];
    v.raster = raster + view * P;
    v.deriv = kDeriv ? deriv + view * P : nullptr;
    v.shade = shade;
    if (kShade) {
        if (shade.attr_out) v.shade.attr_out = shade.attr_out + view * P * shade.A;
        if (shade.uv_out) v.shade.uv_out = shade.uv_out + view * P;
        if (shade.sampled) v.shade.sampled = shade.sampled + view * P;
        if (shade.sdiff) v.shade.sdiff = shade.sdiff + view * P * 2;
    }
    const unsigned long long key = __ldcs(keys + blockIdx.y * P + pix);
    shade_pixel<kDeriv, kShade, kA>(v, px, py, pix, key == ~0ull ? 0u : (uint32_t)key + 1u);
}

uint32_t group_views(uint32_t views, uint32_t W, uint32_t H) {
    const size_t per_view = (size_t)W * H * sizeof(unsigned long long);
    return (uint32_t)std::min<size_t>(std::min(views, 65535u), std::max<size_t>(1, kKeyBytes / per_view));
}

}  // namespace

size_t direct_workspace_bytes(uint32_t views, uint32_t T, uint32_t W, uint32_t H) {
    const size_t g = group_views(views, W, H);
    return align_up(sizeof(uint32_t)) + align_up(g * T * sizeof(uint32_t)) +
           align_up(g * W * H * sizeof(unsigned long long));
}

cudaError_t launch_raster_direct(const float* clip, uint32_t views, uint32_t V, const uint32_t* idx, uint32_t T,
                                 uint32_t W, uint32_t H, const float* viewports, uint32_t cull, void* workspace,
                                 float* raster, float* deriv, const RasterShade* shade, cudaStream_t stream) {
    const uint32_t group = group_views(views, W, H);
    char* ws = static_cast<char*>(workspace);
    uint32_t* queue_count = reinterpret_cast<uint32_t*>(ws);
    uint32_t* queue = reinterpret_cast<uint32_t*>(ws + align_up(sizeof(uint32_t)));
    unsigned long long* keys =
        reinterpret_cast<unsigned long long*>(ws + align_up(sizeof(uint32_t)) + align_up((size_t)group * T * sizeof(uint32_t)));
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
        const dim3 grid(tcx * tcy, n);
#define PDR_SHADE(D, S, A) \
    shade_kernel<D, S, A><<<grid, kShadeW * kShadeH, 0, stream>>>(c4, V, i3, T, W, H, v4, view0, tcx, keys, r4, d4, sa)
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
