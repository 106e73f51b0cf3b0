// Rasterization straight into a visibility buffer (shaders/rasterize_forward.hlsl:45-175 without tile lists);
// shared by the many-view launch (visibility.cu) and the uneven multi-mesh batch (batch.cu).
//
// A pixel's winner is the minimum of (ordered depth bits << 32 | triangle) over the triangles that pass its
// edge tests (depth_key), so triangles may arrive in any order: each (triangle, pixel) pair that passes is one
// 64-bit atomicMin on the pixel's key in L2. The pairs tested are the reference's: a triangle reaches the
// pixels of the 16 x 16 tiles the reference's binning lists it in, narrowed to the candidate rectangle and
// row spans that provably hold every passing sample (raster_tile.cuh).
#pragma once

#include <cuda_runtime.h>
#include <float.h>

#include "pdr_common.cuh"
#include "raster_tile.cuh"

namespace pdr {

// One triangle of one view, ready for its candidates.
struct VisTriangle {
    // screen positions s0x, s0y, s1x, s1y; s2x, s2y, 1, triangle index. Vertices 1 and 2 of a clockwise triangle
    // are swapped: that negates its three edge values exactly, which is what the orientation sign does.
    float4 edge_a, edge_b;
    float4 p0, p1, p2;
    uint32_t x0, x1, y0, y1; // candidate rectangle in image pixels
    float err;               // bound on the edge values' rounding (pixel_bounds)
};

struct VisView {
    const float4* clip;      // [V] clip positions of this view
    const uint3* idx;        // [T]
    uint32_t V, T, W, H, cull;
    float4 vp;
    unsigned long long* keys;  // [H][W]
};

// The candidate rectangle of triangle t; false when it covers nothing.
__device__ __forceinline__ bool vis_setup(const VisView& v, const NdcAxis& ax, const NdcAxis& ay, uint32_t t,
                                          VisTriangle& o) {
    const uint3 vi = v.idx[t];
    if (vi.x >= v.V || vi.y >= v.V || vi.z >= v.V) return false;
    const float4 p0 = v.clip[vi.x], p1 = v.clip[vi.y], p2 = v.clip[vi.z];
    // src/rasterizer.cpp:73-125: the 16 x 16 tiles that list the triangle
    if (!(p0.w > 1e-8f) || !isfinite(p0.w) || !(p1.w > 1e-8f) || !isfinite(p1.w) || !(p2.w > 1e-8f) || !isfinite(p2.w))
        return false;
    const float s0x = p0.x / p0.w, s0y = p0.y / p0.w;
    const float s1x = p1.x / p1.w, s1y = p1.y / p1.w;
    const float s2x = p2.x / p2.w, s2y = p2.y / p2.w;
    if (!isfinite(s0x) || !isfinite(s0y) || !isfinite(s1x) || !isfinite(s1y) || !isfinite(s2x) || !isfinite(s2y))
        return false;
    const float min_x = fminf(s0x, fminf(s1x, s2x)), max_x = fmaxf(s0x, fmaxf(s1x, s2x));
    const float min_y = fminf(s0y, fminf(s1y, s2y)), max_y = fmaxf(s0y, fmaxf(s1y, s2y));
    if (max_x < -1.0f || min_x > 1.0f || max_y < -1.0f || min_y > 1.0f) return false;
    const float area = cross2(s1x - s0x, s1y - s0y, s2x - s0x, s2y - s0y);
    if (fabsf(area) <= 1e-12f || (v.cull == 1 && area <= 0.0f) || (v.cull == 2 && area >= 0.0f)) return false;
    const float4 vp = v.vp;
    const int32_t wm = (int32_t)v.W - 1, hm = (int32_t)v.H - 1;
    // pixel box (last pixel = ceil - 1, from 0 up: a box before the image ends at 0 like one on its border)
    const uint32_t bx0 = (uint32_t)clampi(f2i_sat(floorf((min_x * 0.5f + 0.5f) * vp.z + vp.x)), 0, wm) / kTile;
    const uint32_t by0 = (uint32_t)clampi(f2i_sat(floorf((min_y * 0.5f + 0.5f) * vp.w + vp.y)), 0, hm) / kTile;
    const uint32_t bx1 =
        (uint32_t)clampi(max(f2i_sat(ceilf((max_x * 0.5f + 0.5f) * vp.z + vp.x)), INT32_MIN + 1) - 1, 0, wm) / kTile;
    const uint32_t by1 =
        (uint32_t)clampi(max(f2i_sat(ceilf((max_y * 0.5f + 0.5f) * vp.w + vp.y)), INT32_MIN + 1) - 1, 0, hm) / kTile;
    if (bx1 < bx0 || by1 < by0) return false;
    const uint32_t xa = bx0 * kTile, xb = min((bx1 + 1u) * kTile, v.W), ya = by0 * kTile, yb = min((by1 + 1u) * kTile, v.H);
    const Bounds b = pixel_bounds(s0x, s0y, s1x, s1y, s2x, s2y, area, vp, 2.0f * ax.rcp, 2.0f * ay.rcp, xa, ya, xb, yb,
                                  ax.at(xa), ax.at(xb - 1u), ay.at(ya), ay.at(yb - 1u), o.err, o.x0, o.x1, o.y0, o.y1);
    if (b == Bounds::kNone) return false;
    if (b == Bounds::kWhole) {
        o.x0 = xa;
        o.x1 = xb - 1u;
        o.y0 = ya;
        o.y1 = yb - 1u;
    }
    const bool ccw = area > 0.0f;
    o.edge_a = make_float4(s0x, s0y, ccw ? s1x : s2x, ccw ? s1y : s2y);
    o.edge_b = make_float4(ccw ? s2x : s1x, ccw ? s2y : s1y, 1.0f, __uint_as_float(t));
    o.p0 = p0;
    o.p1 = p1;
    o.p2 = p2;
    return true;
}

// rasterize_forward.hlsl's edge tests and depth at sample (psx, psy): the pixel's key, or ~0 when the triangle
// does not cover it.
__device__ __forceinline__ bool vis_covers(float4 ea, float4 eb, float psx, float psy) {
    const float s0x = ea.x, s0y = ea.y, s1x = ea.z, s1y = ea.w, s2x = eb.x, s2y = eb.y;
    const float e0 = cross2(s1x - psx, s1y - psy, s2x - psx, s2y - psy);
    const float e1 = cross2(s2x - psx, s2y - psy, s0x - psx, s0y - psy);
    const float e2 = cross2(s0x - psx, s0y - psy, s1x - psx, s1y - psy);
    return !(fminf(e0, fminf(e1, e2)) < -1e-7f);  // a NaN fails no test, as in the reference
}

__device__ __forceinline__ unsigned long long vis_key(float4 p0, float4 p1, float4 p2, float psx, float psy,
                                                      uint32_t t) {
    const float q0x = p0.x - psx * p0.w, q0y = p0.y - psy * p0.w;
    const float q1x = p1.x - psx * p1.w, q1y = p1.y - psy * p1.w;
    const float q2x = p2.x - psx * p2.w, q2y = p2.y - psy * p2.w;
    const float a0 = cross2(q1x, q1y, q2x, q2y);
    const float a1 = cross2(q2x, q2y, q0x, q0y);
    const float a2 = cross2(q0x, q0y, q1x, q1y);
    const float ha = a0 + a1 + a2;
    if (fabsf(ha) <= 1e-12f) return ~0ull;
    const float iz = p0.z * a0 + p1.z * a1 + p2.z * a2;
    const float iw = p0.w * a0 + p1.w * a1 + p2.w * a2;
    if (fabsf(iw) <= 1e-12f) return ~0ull;
    return depth_key(clamp_hlsl(iz / iw, -1.0f, 1.0f), t);
}

__device__ __forceinline__ void vis_write(unsigned long long* slot, unsigned long long key) {
    if (key != ~0ull) atomicMin(slot, key);
}

constexpr uint32_t kVisSpanMin = 8;      // rectangles of more pixels are cut to row spans
constexpr uint32_t kVisMaxSide = 64;     // larger rectangles go to the queue of large triangles
constexpr uint32_t kVisMaxPixels = 1024;

// What a warp keeps of its (up to 32) triangles.
struct VisWarp {
    float4 edge_a[32], edge_b[32], p0[32], p1[32], p2[32];
    float4 span_a[32], span_g[32], span_m[32];  // span coefficients; m: -1 / beta of edge 2, sya, inv_dy
    uint4 tri[32];   // triangles with rows, in order: first row, slot | whole << 8, x0 | nx << 20, y0
    uint4 row[32];   // rows with candidates, in order: first candidate, first column, y | slot << 24, sample y
};

// Triangles [first, first + count) of a view, count <= 32, one per lane. Their rows are numbered with a prefix
// sum and taken 32 at a time, one per lane (its span of candidate columns); the rows' candidates are numbered
// the same way and taken 32 at a time, one per lane. So lanes stay busy whatever the triangles' sizes. A lane
// finds the owner of its row or candidate from the mask of owners whose last one falls in the batch. Large
// triangles take a slot of the caller's queue instead: enqueue(slot, triangle).
template <class Enqueue>
__device__ __forceinline__ void vis_warp(const VisView& v, const NdcAxis& ax, const NdcAxis& ay, uint32_t first,
                                         uint32_t count, VisWarp& w, uint32_t* queue_count, Enqueue&& enqueue) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    uint32_t rows = 0;
    uint4 entry = make_uint4(0u, 0u, 0u, 0u);
    bool large = false;
    if (lane < count && first + lane < v.T) {
        VisTriangle t;
        if (vis_setup(v, ax, ay, first + lane, t)) {
            const uint32_t nx = t.x1 - t.x0, ny = t.y1 - t.y0;
            large = nx >= kVisMaxSide || ny >= kVisMaxSide || (nx + 1u) * (ny + 1u) > kVisMaxPixels;
            if (!large) {
                rows = ny + 1u;
                w.edge_a[lane] = t.edge_a;
                w.edge_b[lane] = t.edge_b;
                w.p0[lane] = t.p0;
                w.p1[lane] = t.p1;
                w.p2[lane] = t.p2;
                const bool whole = (nx + 1u) * (ny + 1u) <= kVisSpanMin;
                if (!whole) {
                    const float sya = ay.at(t.y0), syc = ay.at(t.y1);
                    float nb2;
                    span_coefficients(t.edge_a, t.edge_b, t.err, nx, ny, ax.at(t.x0), ax.at(t.x1), sya, syc,
                                      w.span_a[lane], w.span_g[lane], nb2);
                    w.span_m[lane] = make_float4(nb2, sya, ny ? 1.0f / (syc - sya) : 0.0f, 0.0f);
                }
                entry = make_uint4(0u, lane | (whole ? 256u : 0u) | (nx << 16), t.x0, t.y0);
            }
        }
    }
    const unsigned larges = __ballot_sync(0xffffffffu, large);
    if (larges) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(queue_count, (uint32_t)__popc(larges));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (large) enqueue(at + __popc(larges & below), first + lane);
    }
    uint32_t last_row = rows;  // inclusive prefix sum
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, last_row, d);
        if (lane >= d) last_row += y;
    }
    const uint32_t total_rows = __shfl_sync(0xffffffffu, last_row, 31);
    const unsigned with_rows = __ballot_sync(0xffffffffu, rows > 0);
    if (rows > 0) {
        entry.x = last_row - rows;
        w.tri[__popc(with_rows & below)] = entry;
    }
    --last_row;
    __syncwarp();
    const float slx = 0.05f + 1e-6f * (v.vp.z + fabsf(v.vp.x));
    uint32_t tris_ended = 0;
    for (uint32_t row_base = 0; row_base < total_rows; row_base += 32) {
        // this batch's rows
        const uint32_t ends = __reduce_or_sync(
            0xffffffffu, rows > 0 && last_row >= row_base && last_row - row_base < 32u ? 1u << (last_row - row_base) : 0u);
        const uint32_t rank = tris_ended + __popc(ends & below);
        tris_ended += __popc(ends);
        uint32_t width = 0;
        uint4 row = make_uint4(0u, 0u, 0u, 0u);
        if (row_base + lane < total_rows) {
            const uint4 tr = w.tri[rank];
            const uint32_t slot = tr.y & 31u, nx = tr.y >> 16, y = tr.w + (row_base + lane - tr.x);
            const float psy = ay.at(y);
            uint32_t x_first = 0;
            if (tr.y & 256u) {
                width = nx + 1u;
            } else {
                const float4 m = w.span_m[slot];
                width = row_span(w.span_a[slot], w.span_g[slot], m.x, nx, psy, m.y, m.z, slx, x_first);
            }
            row = make_uint4(0u, tr.z + x_first, y | (slot << 24), __float_as_uint(psy));
        }
        uint32_t last = width;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, last, d);
            if (lane >= d) last += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, last, 31);
        const unsigned with_px = __ballot_sync(0xffffffffu, width > 0);
        if (width > 0) {
            row.x = last - width;
            w.row[__popc(with_px & below)] = row;
        }
        --last;
        __syncwarp();
        uint32_t rows_ended = 0;
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t c = base + lane;
            const uint32_t done = __reduce_or_sync(0xffffffffu,
                                                   width > 0 && last >= base && last - base < 32u ? 1u << (last - base) : 0u);
            const uint32_t r = rows_ended + __popc(done & below);
            rows_ended += __popc(done);
            if (c >= total) continue;
            const uint4 ow = w.row[r];
            const uint32_t x = ow.y + (c - ow.x), y = ow.z & 0xFFFFFFu, k = ow.z >> 24;
            const float psx = ax.at(x), psy = __uint_as_float(ow.w);
            const float4 ea = w.edge_a[k], eb = w.edge_b[k];
            if (!vis_covers(ea, eb, psx, psy)) continue;
            vis_write(v.keys + (size_t)y * v.W + x,
                      vis_key(w.p0[k], w.p1[k], w.p2[k], psx, psy, __float_as_uint(eb.w)));
        }
        __syncwarp();  // the row table is rewritten by the next batch
    }
    __syncwarp();
}

// Rows [r0, r1) of a large triangle's candidate rectangle, over the warps of a CTA.
__device__ __forceinline__ void vis_rows(const VisView& v, const NdcAxis& ax, const NdcAxis& ay, const VisTriangle& t,
                                         uint32_t r0, uint32_t r1) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t nx = t.x1 - t.x0, ny = t.y1 - t.y0;
    const float sya = ay.at(t.y0), syc = ay.at(t.y1), inv_dy = ny ? 1.0f / (syc - sya) : 0.0f;
    const float slx = 0.05f + 1e-6f * (v.vp.z + fabsf(v.vp.x));
    float4 A, G;
    float nb2;
    span_coefficients(t.edge_a, t.edge_b, t.err, nx, ny, ax.at(t.x0), ax.at(t.x1), sya, syc, A, G, nb2);
    for (uint32_t r = r0 + warp; r < r1; r += warps) {
        const uint32_t y = t.y0 + r;
        const float psy = ay.at(y);
        uint32_t first;
        const uint32_t width = row_span(A, G, nb2, nx, psy, sya, inv_dy, slx, first);
        for (uint32_t c = lane; c < width; c += 32) {
            const uint32_t x = t.x0 + first + c;
            const float psx = ax.at(x);
            if (!vis_covers(t.edge_a, t.edge_b, psx, psy)) continue;
            vis_write(v.keys + (size_t)y * v.W + x,
                      vis_key(t.p0, t.p1, t.p2, psx, psy, __float_as_uint(t.edge_b.w)));
        }
    }
}

// Bands of rows per queued triangle: enough items to occupy the grid.
__device__ __forceinline__ uint32_t vis_bands(uint32_t queued) { return min(64u, max(1u, 4u * gridDim.x / queued)); }

__device__ __forceinline__ void vis_band(const VisView& v, uint32_t triangle, uint32_t band, uint32_t bands) {
    const NdcAxis ax(v.vp.x, v.vp.z), ay(v.vp.y, v.vp.w);
    VisTriangle t;
    if (!vis_setup(v, ax, ay, triangle, t)) return;
    const uint64_t rows = t.y1 - t.y0 + 1u;
    vis_rows(v, ax, ay, t, (uint32_t)(rows * band / bands), (uint32_t)(rows * (band + 1u) / bands));
}

}  // namespace pdr
