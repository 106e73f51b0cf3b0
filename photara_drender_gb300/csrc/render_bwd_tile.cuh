// The fused adjoint of rasterize -> interpolate(attributes), interpolate(uv) -> texture for the
// pixels of 16 x 8 tiles; shared by the per-mesh launch (fused.cu) and the uneven multi-mesh batch (batch.cu).
// Their kernels run 128 threads a tile, each warp on two tile rows.
//
// One thread per pixel runs, in the reference's order and arithmetic, texture_grad_texture
// (double-exact weights, vector atomics, warp-aggregated for magnified textures), texture_grad_uv,
// interpolate_grad_attributes / interpolate_grad_raster for both attribute sets, and
// rasterize_backward for the summed raster gradient, everything in registers. Each pixel's vertex gradients
// then go to shared memory, and the warp sums them over all its pixels on the same triangle (neighbours in both
// rows): one lane per (triangle, corner, four values) adds its triangle's pixels and issues one 16-byte
// reduction. Summing with shuffles along runs of pixels took 24 values x 3 steps per pixel and a second merge
// between the rows.
//
// What bounds it: the latency of a pixel's chain of loads (raster value, triangle, vertices) at 32 warps per SM;
// issue is at 53%. Measured on 64 views of 200k triangles at 1024 x 1024 with a 4096 x 4096 texture: 2.66 ms
// before; 2.20 with the sums in shared memory, the texel position in floats, bounds decided without divisions and
// every gather issued before the texture work (900 -> 650 instructions per 32 pixels); 2.08 without the 24 bytes of
// uncovered pixels; 1.71 with resident CTAs that load the next tile's raster value and triangle ahead and tiles
// sorted by what they sample (tile_order.cuh; 1.92 in view order). Dropping the 155 M texel reductions leaves 1.69
// of the 2.20: they cost about a quarter.
#pragma once

#include <cuda_runtime.h>

#include "ndc_axis.cuh"
#include "pdr_common.cuh"
#include "pdr_internal.h"

namespace pdr {

__device__ __forceinline__ void red_v4(float* addr, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// 32 bytes with one load (addr 32-byte aligned), streaming.
__device__ __forceinline__ void load_v8_cs(const float4* addr, float4& a, float4& b) {
    asm volatile("ld.global.cs.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(addr));
}

// rasterize_backward.hlsl:78-90: whether pixel (px, py) lies in the triangle's clamped pixel bounds,
// floor(lo) <= px < ceil(hi), which is lo < px + 1 and hi > px. The bounds are first formed with approximate
// quotients: with `m` pixels to spare, far more than their error (2 ulp of each quotient scaled to pixels, and a
// few roundings; divisors from 2^126 on give 0 and are left out), they decide; otherwise, next to the bounds, the
// reference's divisions do.
__device__ __forceinline__ bool visited(float4 p0, float4 p1, float4 p2, float4 vp, uint32_t px, uint32_t py, uint32_t W,
                                        uint32_t H) {
    {
        const float s0x = __fdividef(p0.x, p0.w), s0y = __fdividef(p0.y, p0.w);
        const float s1x = __fdividef(p1.x, p1.w), s1y = __fdividef(p1.y, p1.w);
        const float s2x = __fdividef(p2.x, p2.w), s2y = __fdividef(p2.y, p2.w);
        const float lx = fminf(s0x, fminf(s1x, s2x)), hx = fmaxf(s0x, fmaxf(s1x, s2x));
        const float ly = fminf(s0y, fminf(s1y, s2y)), hy = fmaxf(s0y, fmaxf(s1y, s2y));
        const float mx = 0.05f + 2e-6f * (vp.z * (1.0f + fmaxf(fabsf(lx), fabsf(hx))) + fabsf(vp.x));
        const float my = 0.05f + 2e-6f * (vp.w * (1.0f + fmaxf(fabsf(ly), fabsf(hy))) + fabsf(vp.y));
        const float x = (float)px, y = (float)py;
        if (fmaxf(p0.w, fmaxf(p1.w, p2.w)) < 8e37f &&
            (lx * 0.5f + 0.5f) * vp.z + vp.x < x + 1.0f - mx && (hx * 0.5f + 0.5f) * vp.z + vp.x > x + mx &&
            (ly * 0.5f + 0.5f) * vp.w + vp.y < y + 1.0f - my && (hy * 0.5f + 0.5f) * vp.w + vp.y > y + my)
            return true;
    }
    const float s0x = p0.x / p0.w, s0y = p0.y / p0.w;
    const float s1x = p1.x / p1.w, s1y = p1.y / p1.w;
    const float s2x = p2.x / p2.w, s2y = p2.y / p2.w;
    const float mnx = fminf(s0x, fminf(s1x, s2x)), mny = fminf(s0y, fminf(s1y, s2y));
    const float mxx = fmaxf(s0x, fmaxf(s1x, s2x)), mxy = fmaxf(s0y, fmaxf(s1y, s2y));
    const int32_t x0 = clampi(f2i_sat(floorf((mnx * 0.5f + 0.5f) * vp.z + vp.x)), 0, (int32_t)W);
    const int32_t x1 = clampi(f2i_sat(ceilf((mxx * 0.5f + 0.5f) * vp.z + vp.x)), 0, (int32_t)W);
    const int32_t y0 = clampi(f2i_sat(floorf((mny * 0.5f + 0.5f) * vp.w + vp.y)), 0, (int32_t)H);
    const int32_t y1 = clampi(f2i_sat(ceilf((mxy * 0.5f + 0.5f) * vp.w + vp.y)), 0, (int32_t)H);
    return (int32_t)px >= x0 && (int32_t)px < x1 && (int32_t)py >= y0 && (int32_t)py < y1;
}

// One view of one mesh as the adjoint sees it. Images and per-view vertex arrays may be those of all views:
// a pixel's index counts from their first element, and `first_vertex` is the view's first vertex (kernel
// arguments then stay as they are, in constant memory instead of in registers).
struct BackwardView {
    const float4* clip;           // clip positions
    size_t first_vertex;
    uint32_t V, T, W, H;
    float4 vp;
    const float* attrs;           // [V][A], or nullptr
    const float2* uv_attrs;       // [V][2], or nullptr
    const float4* tex;            // [th][tw][4], or nullptr
    uint32_t tw, th, mode;
    const float2* uv;             // per pixel, or nullptr
    const float* grad_attr_out;   // A per pixel
    const float4* grad_sampled;   // per pixel
    float* g_clip;                // 4 per vertex
    float* g_attr;                // [V][A]
    float* g_uv;                  // [V][2]
    float* g_tex;                 // [th][tw][4]
    const float4* sdiff;          // 2 per pixel: texel differences of the forward's sample, or nullptr
    bool sdiff32;                 // sdiff is set and 32-byte aligned
    uint32_t* status;
    // When set: vertex-gradient records, vertex_record_floats(kA) per vertex (uv, attributes, clip x/y/w, zero
    // padding), added with 16-byte reductions and summed over the views afterwards
    // (vertex_grad_finish_kernel); g_clip, g_attr and g_uv are then not touched here.
    float* g_vtx;
};

// Floats per vertex-gradient record: uv 2 + attributes kA + clip x/y/w 3, rounded up to 16 bytes.
__host__ __device__ constexpr uint32_t vertex_record_floats(int kA) { return (uint32_t)((5 + kA + 3) / 4 * 4); }

constexpr int kBwdTileH = 8;                   // tile of 16 x kBwdTileH pixels
constexpr int kBwdThreads = 16 * kBwdTileH;

// Quads (16 bytes) of vertex gradients per pixel, three records, and their pitch in shared memory (odd: the
// 16-byte stores of a quarter warp hit different banks).
__host__ __device__ constexpr int vertex_quads(int kA) { return 3 * (int)vertex_record_floats(kA) / 4; }
__host__ __device__ constexpr int vertex_quad_pitch(int kA) { return vertex_quads(kA) | 1; }

template <int kA>
struct BackwardShared {
    float4 quads[kBwdThreads][vertex_quad_pitch(kA)];
    uint4 triangles[kBwdThreads / 32][32];  // per warp: the vertices of a triangle and the lanes on it
};

// CTAs per SM: 64 registers keep the chain of gathers of a pixel in flight without spills (64 views with three
// attributes: 8 CTAs 1.71 ms, 7 1.79, 9 1.85); eight attributes' records leave shared memory for 7.
__host__ __device__ constexpr int backward_ctas(int kA) { return kA < 8 ? 8 : 7; }

// What decides the rest of a pixel's loads: its raster value and its triangle's vertices.
struct PixelHead {
    float4 r;
    uint3 vi;
};

__device__ __forceinline__ uint3 head_triangle(float4 r, const uint3* __restrict__ idx, uint32_t T) {
    const uint32_t id = raster_id(r.w);
    return id != 0 && id <= T ? idx[id - 1] : make_uint3(0u, 0u, 0u);
}

// The adjoint of pixel (px, py) with index `pix` in the images, called by whole warps; h.r is zero outside the
// image. `ahead` runs once the pixel's own loads are consumed and before its sums: a place to start loads whose
// addresses wait for earlier ones.
// kTexAgg: texture-gradient taps warp-aggregated (1), plain (0), or decided from the texture and image
// sizes (-1: aggregated when the texture has fewer texels than the view has pixels).
template <int kA, int kTexAgg = -1, class Ahead>
__device__ __forceinline__ void render_backward_pixel(const BackwardView& v, uint32_t px, uint32_t py, size_t pix,
                                                      const PixelHead& h, BackwardShared<kA>& sh, Ahead&& ahead) {
    const uint32_t V = v.V, T = v.T, W = v.W, H = v.H;
    const uint32_t tw = v.tw, th = v.th, mode = v.mode;
    constexpr int kNV = 2 + kA + 3;  // per vertex: uv attributes, attributes, clip x/y/w
    constexpr int kR = (int)vertex_record_floats(kA);
    constexpr int kQ = kR / 4;
    const bool magnified = kTexAgg >= 0 ? kTexAgg == 1 : (uint64_t)tw * th < (uint64_t)W * H;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const float4 r = h.r;
    const uint3 vi = h.vi;
    const uint32_t id = raster_id(r.w);
    const bool valid = id != 0 && id <= T;  // contributes vertex gradients

    if (r.w != 0.0f) {
        // per-pixel inputs are read exactly once: loaded with the streaming (evict-first) hint so that L2
        // keeps the texture and the gradient texels the scatter below adds into (-0.24 ms on 64 views)
        float2 u = make_float2(0.0f, 0.0f);
        float4 gs = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (v.tex) {  // of covered pixels alone: an uncovered one's 24 bytes stay in DRAM
            u = __ldcs(v.uv + pix);
            gs = __ldcs(v.grad_sampled + pix);
        }
        const bool inside = valid && vi.x < V && vi.y < V && vi.z < V;
        // the triangle's gathers, all issued before the texture work that hides them
        float4 p0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), p1 = p0, p2 = p0;
        float2 t0 = make_float2(0.0f, 0.0f), t1 = t0, t2 = t0;
        constexpr int kN = kA > 0 ? kA : 1;
        float ga[kN];
        if (inside) {
            const float4* clip = v.clip + v.first_vertex;
            p0 = clip[vi.x];
            p1 = clip[vi.y];
            p2 = clip[vi.z];
            if (v.uv_attrs) {
                t0 = __ldg(v.uv_attrs + vi.x);
                t1 = __ldg(v.uv_attrs + vi.y);
                t2 = __ldg(v.uv_attrs + vi.z);
            }
        }
        if (valid) {
#pragma unroll
            for (int a = 0; a < kA; ++a) ga[a] = __ldcs(v.grad_attr_out + pix * kA + a);
        }
        float gux = 0.0f, guy = 0.0f;
        if (v.tex) {
            // texture_grad_uv (fp32)
            if (id != 0) {
                float4 du, dv;
                if (v.sdiff32) {
                    load_v8_cs(v.sdiff + pix * 2, du, dv);
                } else if (v.sdiff) {
                    // the forward's texel differences: the same values the gathers below compute
                    du = __ldcs(v.sdiff + pix * 2);
                    dv = __ldcs(v.sdiff + pix * 2 + 1);
                } else {
                    const float tx = u.x * (float)tw - 0.5f, ty = u.y * (float)th - 0.5f;
                    const int32_t bx = f2i_sat(floorf(tx)), by = f2i_sat(floorf(ty));
                    const float fx = tx - floorf(tx), fy = ty - floorf(ty);
                    const int32_t x0 = address_coordinate(bx, tw, mode), x1 = address_coordinate(add1(bx), tw, mode);
                    const int32_t y0 = address_coordinate(by, th, mode), y1 = address_coordinate(add1(by), th, mode);
                    const float4 c00 = __ldg(v.tex + (size_t)(uint32_t)y0 * tw + (uint32_t)x0);
                    const float4 c10 = __ldg(v.tex + (size_t)(uint32_t)y0 * tw + (uint32_t)x1);
                    const float4 c01 = __ldg(v.tex + (size_t)(uint32_t)y1 * tw + (uint32_t)x0);
                    const float4 c11 = __ldg(v.tex + (size_t)(uint32_t)y1 * tw + (uint32_t)x1);
                    du.x = (1.0f - fy) * (c10.x - c00.x) + fy * (c11.x - c01.x);
                    du.y = (1.0f - fy) * (c10.y - c00.y) + fy * (c11.y - c01.y);
                    du.z = (1.0f - fy) * (c10.z - c00.z) + fy * (c11.z - c01.z);
                    du.w = (1.0f - fy) * (c10.w - c00.w) + fy * (c11.w - c01.w);
                    dv.x = (1.0f - fx) * (c01.x - c00.x) + fx * (c11.x - c10.x);
                    dv.y = (1.0f - fx) * (c01.y - c00.y) + fx * (c11.y - c10.y);
                    dv.z = (1.0f - fx) * (c01.z - c00.z) + fx * (c11.z - c10.z);
                    dv.w = (1.0f - fx) * (c01.w - c00.w) + fx * (c11.w - c10.w);
                }
                const float ftw = (float)tw, fth = (float)th;
                gux += gs.x * (du.x * ftw);
                guy += gs.x * (dv.x * fth);
                gux += gs.y * (du.y * ftw);
                guy += gs.y * (dv.y * fth);
                gux += gs.z * (du.z * ftw);
                guy += gs.z * (dv.z * fth);
                gux += gs.w * (du.w * ftw);
                guy += gs.w * (dv.w * fth);
            }
            // texture_grad_texture: pixels with raster.w != 0, double-exact weights (rasterizer.cpp:198-229)
            {
                int32_t bx, by;
                float fx, fy;
                const int ex = exact_texel_coordinate(u.x, tw, &bx, &fx);
                const int ey = exact_texel_coordinate(u.y, th, &by, &fy);
                if (ex | ey) {
                    atomicMax(v.status + kStatusTexelError, ((ex | ey) & kTexelNonFinite) ? (uint32_t)kTexelNonFinite
                                                                                          : (uint32_t)kTexelRange);
                } else {
                    const int32_t xs0 = address_coordinate(bx, tw, mode), xs1 = address_coordinate(bx + 1, tw, mode);
                    const int32_t ys0 = address_coordinate(by, th, mode), ys1 = address_coordinate(by + 1, th, mode);
                    const float w0 = (1.0f - fx) * (1.0f - fy), w1 = fx * (1.0f - fy), w2 = (1.0f - fx) * fy,
                                w3 = fx * fy;
                    float* row0 = v.g_tex + (size_t)(uint32_t)ys0 * tw * 4;
                    float* row1 = v.g_tex + (size_t)(uint32_t)ys1 * tw * 4;
                    const size_t o0 = (size_t)(uint32_t)xs0 * 4, o1 = (size_t)(uint32_t)xs1 * 4;
                    red_add_v4_texel(row0 + o0, make_float4(w0 * gs.x, w0 * gs.y, w0 * gs.z, w0 * gs.w), magnified);
                    red_add_v4_texel(row0 + o1, make_float4(w1 * gs.x, w1 * gs.y, w1 * gs.z, w1 * gs.w), magnified);
                    red_add_v4_texel(row1 + o0, make_float4(w2 * gs.x, w2 * gs.y, w2 * gs.z, w2 * gs.w), magnified);
                    red_add_v4_texel(row1 + o1, make_float4(w3 * gs.x, w3 * gs.y, w3 * gs.z, w3 * gs.w), magnified);
                }
            }
        }
        if (valid) {
            const float bu = r.x, bv = r.y;
            // interpolate_grad_raster: uv attributes first, attributes accumulated on top
            float grx = 0.0f, gry = 0.0f;
            if (inside) {
                if (v.uv_attrs) {
                    grx += gux * (t0.x - t2.x);
                    gry += gux * (t1.x - t2.x);
                    grx += guy * (t0.y - t2.y);
                    gry += guy * (t1.y - t2.y);
                }
                if (kA > 0) {
                    float ax = 0.0f, ay = 0.0f;
#pragma unroll
                    for (int a = 0; a < kA; ++a) {
                        const float a0 = __ldg(v.attrs + (size_t)vi.x * kA + a), a1 = __ldg(v.attrs + (size_t)vi.y * kA + a);
                        const float a2 = __ldg(v.attrs + (size_t)vi.z * kA + a);
                        ax += ga[a] * (a0 - a2);
                        ay += ga[a] * (a1 - a2);
                    }
                    grx = grx + ax;
                    gry = gry + ay;
                }
            }
            // rasterize_backward for this pixel (same visit rule as the per-triangle loop)
            float gc3[3][3] = {{0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}};
            if (inside && !(grx == 0.0f && gry == 0.0f) &&
                !(p0.w <= 1e-8f || p1.w <= 1e-8f || p2.w <= 1e-8f) && visited(p0, p1, p2, v.vp, px, py, W, H)) {
                const NdcAxis axis_x(v.vp.x, v.vp.z, __frcp_rn(v.vp.z)), axis_y(v.vp.y, v.vp.w, __frcp_rn(v.vp.w));
                const float sx = axis_x.at(px), sy = axis_y.at(py);
                const float q0x = p0.x - sx * p0.w, q0y = p0.y - sy * p0.w;
                const float q1x = p1.x - sx * p1.w, q1y = p1.y - sy * p1.w;
                const float q2x = p2.x - sx * p2.w, q2y = p2.y - sy * p2.w;
                const float a0 = cross2(q1x, q1y, q2x, q2y);
                const float a1 = cross2(q2x, q2y, q0x, q0y);
                const float area = a0 + a1 + cross2(q0x, q0y, q1x, q1y);
                if (!(fabsf(area) <= 1e-12f)) {
                    const float eps = area >= 0.0f ? 1e-6f : -1e-6f;
                    const float inv = 1.0f / (area + eps);
                    const float b0 = a0 * inv, b1 = a1 * inv;
                    const float gb0 = grx * inv, gb1 = gry * inv;
                    const float gc = gb0 * b0 + gb1 * b1;
                    const float g0x = gc * (q2y - q1y) - gb1 * q2y;
                    const float g1x = gc * (q0y - q2y) + gb0 * q2y;
                    const float g2x = gc * (q1y - q0y) - gb0 * q1y + gb1 * q0y;
                    const float g0y = gc * (q1x - q2x) + gb1 * q2x;
                    const float g1y = gc * (q2x - q0x) - gb0 * q2x;
                    const float g2y = gc * (q0x - q1x) + gb0 * q1x - gb1 * q0x;
                    gc3[0][0] = g0x; gc3[0][1] = g0y; gc3[0][2] = -sx * g0x - sy * g0y;
                    gc3[1][0] = g1x; gc3[1][1] = g1y; gc3[1][2] = -sx * g1x - sy * g1y;
                    gc3[2][0] = g2x; gc3[2][1] = g2y; gc3[2][2] = -sx * g2x - sy * g2y;
                }
            }
            // interpolate_grad_attributes for uv and attributes: each distinct vertex once, with the
            // weight accumulated as interpolate_grad_attributes.hlsl:42-54 does; the records go to shared memory
            const uint32_t vs[3] = {vi.x, vi.y, vi.z};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint32_t vx = vs[k];
                bool first = vx < V;
#pragma unroll
                for (int j = 0; j < k; ++j) first = first && vs[j] != vx;
                float wgt = 0.0f;
                if (vi.x == vx) wgt += bu;
                if (vi.y == vx) wgt += bv;
                if (vi.z == vx) wgt += 1.0f - bu - bv;
                float rec[kR];
                rec[0] = first && v.uv_attrs ? wgt * gux : 0.0f;
                rec[1] = first && v.uv_attrs ? wgt * guy : 0.0f;
#pragma unroll
                for (int a = 0; a < kA; ++a) rec[2 + a] = first ? wgt * ga[a] : 0.0f;
#pragma unroll
                for (int c = 0; c < 3; ++c) rec[2 + kA + c] = gc3[k][c];
#pragma unroll
                for (int c = kNV; c < kR; ++c) rec[c] = 0.0f;
#pragma unroll
                for (int q = 0; q < kQ; ++q)
                    sh.quads[threadIdx.x][k * kQ + q] = make_float4(rec[4 * q], rec[4 * q + 1], rec[4 * q + 2], rec[4 * q + 3]);
            }
        }
    }
    __syncwarp();
    ahead();
    if (!__any_sync(0xffffffffu, valid)) return;
    // The warp's triangles, in the order of their first lanes, with the lanes on each.
    const unsigned same = __match_any_sync(0xffffffffu, valid ? id : (0x80000000u | lane));
    const bool leader = valid && (same & ((1u << lane) - 1u)) == 0u;
    const unsigned leaders = __ballot_sync(0xffffffffu, leader);
    if (leader) sh.triangles[warp][__popc(leaders & ((1u << lane) - 1u))] = make_uint4(vi.x, vi.y, vi.z, same);
    __syncwarp();
    const uint32_t tasks = (uint32_t)__popc(leaders) * (3u * kQ);
    const float4(*mine)[vertex_quad_pitch(kA)] = &sh.quads[warp * 32u];
    for (uint32_t task = lane; task < tasks; task += 32) {
        const uint32_t g = task / (3u * kQ), c = task - g * (3u * kQ);  // triangle; corner * kQ + quad
        const uint4 tri = sh.triangles[warp][g];
        const uint32_t corner = c / (uint32_t)kQ, q = c - corner * (uint32_t)kQ;
        const uint32_t vertex = corner == 0 ? tri.x : (corner == 1 ? tri.y : tri.z);
        uint32_t lanes = tri.w;
        float4 s = mine[__ffs(lanes) - 1][c];
        for (lanes &= lanes - 1u; lanes; lanes &= lanes - 1u) {
            const float4 o = mine[__ffs(lanes) - 1][c];
            s.x += o.x;
            s.y += o.y;
            s.z += o.z;
            s.w += o.w;
        }
        if (vertex >= V) continue;
        if (v.g_vtx) {
            red_v4(v.g_vtx + (v.first_vertex + vertex) * kR + q * 4u, s);
        } else {
            const float x[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = (int)q * 4 + k;
                if (j < 2) {
                    if (v.g_uv) atomicAdd(v.g_uv + (size_t)vertex * 2 + j, x[k]);
                } else if (j < 2 + kA) {
                    atomicAdd(v.g_attr + (size_t)vertex * kA + (j - 2), x[k]);
                } else if (j < kNV) {  // z of the clip gradient stays 0 (rasterize_backward.hlsl writes none)
                    atomicAdd(v.g_clip + (v.first_vertex + vertex) * 4 + (j == kNV - 1 ? 3 : j - 2 - kA), x[k]);
                }
            }
        }
    }
    __syncwarp();  // the warp's shared memory is rewritten by its next tile
}

// The vertex-gradient records of one vertex in all views into the outputs: each view's clip gradient (x, y, 0, w),
// and the uv and attribute gradients summed over the views in view order. Every output element is written, so
// none needs clearing first; with `add` they are added to outputs that were cleared and that others add to.
template <int kA>
__device__ __forceinline__ void sum_vertex_records(const float* __restrict__ rec_all, uint32_t views, uint32_t V,
                                                   uint32_t vtx, float* __restrict__ g_clip_all,
                                                   float* __restrict__ g_attr, float* __restrict__ g_uv,
                                                   bool add = false) {
    constexpr uint32_t kR = vertex_record_floats(kA);
    constexpr uint32_t kNV = 2 + kA + 3;
    float acc[2 + kA];
#pragma unroll
    for (int j = 0; j < 2 + kA; ++j) acc[j] = 0.0f;
    for (uint32_t view = 0; view < views; ++view) {
        const float4* rec = reinterpret_cast<const float4*>(rec_all + ((size_t)view * V + vtx) * kR);
        float r[kR];
#pragma unroll
        for (uint32_t c = 0; c < kR / 4; ++c) {
            const float4 q = __ldcs(rec + c);
            r[4 * c] = q.x;
            r[4 * c + 1] = q.y;
            r[4 * c + 2] = q.z;
            r[4 * c + 3] = q.w;
        }
#pragma unroll
        for (int j = 0; j < 2 + kA; ++j) acc[j] += r[j];
        const float4 clip = make_float4(r[kNV - 3], r[kNV - 2], 0.0f, r[kNV - 1]);
        if (add)
            red_v4(g_clip_all + ((size_t)view * V + vtx) * 4, clip);
        else
            reinterpret_cast<float4*>(g_clip_all)[(size_t)view * V + vtx] = clip;
    }
    if (add) {
        if (g_uv) {
            atomicAdd(g_uv + (size_t)vtx * 2, acc[0]);
            atomicAdd(g_uv + (size_t)vtx * 2 + 1, acc[1]);
        }
        if (g_attr) {
#pragma unroll
            for (int a = 0; a < kA; ++a) atomicAdd(g_attr + (size_t)vtx * kA + a, acc[2 + a]);
        }
        return;
    }
    if (g_uv) {
        g_uv[(size_t)vtx * 2] = acc[0];
        g_uv[(size_t)vtx * 2 + 1] = acc[1];
    }
    if (g_attr) {
#pragma unroll
        for (int a = 0; a < kA; ++a) g_attr[(size_t)vtx * kA + a] = acc[2 + a];
    }
}

}  // namespace pdr
