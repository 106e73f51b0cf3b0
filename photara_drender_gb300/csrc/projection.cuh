// The tests shaders/project_texture.hlsl applies to a texel before it reads the view's visibility:
// in front of the camera, inside the clip volume, inside the viewport and facing the camera at
// least min_view_cosine. Shared by the projection kernel and the ray caster, which traces only the
// texel-views that pass, so both decide identically.
#pragma once

#include <cuda_runtime.h>

#include "../../include/pdr_capi.h"
#include "pdr_common.cuh"

namespace pdr {

struct ProjectedTexel {
    float ppx, ppy, ndz;  // pixel position and NDC depth
    float vl, cosv;       // distance to the camera and cosine of the view angle
};

// a / d, b / d and c / d with one division: quotients by a fixed divisor as in NdcAxis, under its conditions.
__device__ __forceinline__ void quotients(float a, float b, float c, float d, float& qa, float& qb, float& qc) {
    const float lo = fminf(fminf(fabsf(a), fabsf(b)), fabsf(c)), hi = fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c));
    if (lo >= 1e-25f && hi <= 1e25f && d >= 1e-6f && d <= 1e9f && (__float_as_uint(d) & 0x7fffffu) != 0x7fffffu) {
        const float r = 1.0f / d;
        const auto quotient = [&](float n) {
            const float q = n * r;
            return __fmaf_rn(__fmaf_rn(-q, d, n), r, q);
        };
        qa = quotient(a);
        qb = quotient(b);
        qc = quotient(c);
    } else {
        qa = a / d;
        qb = b / d;
        qc = c / d;
    }
}

__device__ __forceinline__ bool project_texel(const pdr_projection_view& v, float px, float py, float pz, float nx,
                                              float ny, float nz, ProjectedTexel& o) {
    const float* M = v.world_to_clip;
    const float cw = M[12] * px + M[13] * py + M[14] * pz + M[15] * 1.0f;
    if (cw <= 1e-8f) return false;
    const float cx = M[0] * px + M[1] * py + M[2] * pz + M[3] * 1.0f;
    const float cy = M[4] * px + M[5] * py + M[6] * pz + M[7] * 1.0f;
    const float cz = M[8] * px + M[9] * py + M[10] * pz + M[11] * 1.0f;
    float ndx, ndy, ndz;
    quotients(cx, cy, cz, cw, ndx, ndy, ndz);
    if (ndx < -1.0f || ndy < -1.0f || ndx > 1.0f || ndy > 1.0f || ndz < -1.0f || ndz > 1.0f) return false;
    const float ppx = v.viewport[0] + (ndx * 0.5f + 0.5f) * v.viewport[2];
    const float ppy = v.viewport[1] + (ndy * 0.5f + 0.5f) * v.viewport[3];
    if (ppx < v.viewport[0] || ppy < v.viewport[1] || ppx >= v.viewport[0] + v.viewport[2] ||
        ppy >= v.viewport[1] + v.viewport[3])
        return false;
    // view direction before visibility: the facing test rejects half of all texel-views before the
    // visibility work, with the same outcome as the reference's order
    const float vx0 = v.camera_position[0] - px, vy0 = v.camera_position[1] - py;
    const float vz0 = v.camera_position[2] - pz;
    const float vl = sqrtf(vx0 * vx0 + vy0 * vy0 + vz0 * vz0);
    float dx, dy, dz;
    quotients(vx0, vy0, vz0, vl, dx, dy, dz);
    const float cosv = nx * dx + ny * dy + nz * dz;
    if (cosv < v.min_view_cosine) return false;
    o.ppx = ppx;
    o.ppy = ppy;
    o.ndz = ndz;
    o.vl = vl;
    o.cosv = cosv;
    return true;
}

// A view as project_gate reads it, staged in shared memory.
struct GateView {
    float4 row_x, row_y, row_z, row_w;  // world_to_clip
    float4 camera;                      // xyz, min_view_cosine
    float matrix_max;                   // largest magnitude of world_to_clip
    float pad[3];
};

__device__ __forceinline__ void gate_view(const pdr_projection_view& v, GateView& g) {
    const float* M = v.world_to_clip;
    g.row_x = make_float4(M[0], M[1], M[2], M[3]);
    g.row_y = make_float4(M[4], M[5], M[6], M[7]);
    g.row_z = make_float4(M[8], M[9], M[10], M[11]);
    g.row_w = make_float4(M[12], M[13], M[14], M[15]);
    g.camera = make_float4(v.camera_position[0], v.camera_position[1], v.camera_position[2], v.min_view_cosine);
    float m = 0.0f;
    for (int k = 0; k < 16; ++k) m = fmaxf(m, fabsf(M[k]));
    // a viewport far from the origin for its size rounds more than the margin: nothing is sure there
    const float vw = v.viewport[2], vh = v.viewport[3];
    const bool near = fabsf(v.viewport[0]) <= 16.0f * vw && fabsf(v.viewport[1]) <= 16.0f * vh && fminf(vw, vh) > 1e-20f &&
                      fmaxf(vw, vh) < 1e20f;
    g.matrix_max = near ? m : INFINITY;
}

enum class Gate { kReject, kUnsure, kPass };

// project_texel's decision where it is not close: a third of its instructions, no division, half of the texel-views
// gone after the facing test. kUnsure within 1e-4 of the facing limit or about 1e-5 of the clip volume's sides,
// far more than the roundings of either form (the viewport test is the clip volume's once more up to rounding); a NaN is
// unsure as well.
__device__ __forceinline__ Gate project_gate(const GateView& v, float px, float py, float pz, float nx, float ny,
                                             float nz) {
    const float vx = v.camera.x - px, vy = v.camera.y - py, vz = v.camera.z - pz;
    const float v2 = __fmaf_rn(vx, vx, __fmaf_rn(vy, vy, vz * vz)), vl = v2 * rsqrtf(v2);
    if (v2 < 1e-30f) return Gate::kUnsure;
    const float facing = __fmaf_rn(nx, vx, __fmaf_rn(ny, vy, nz * vz));
    if (facing < (v.camera.w - 1e-4f) * vl) return Gate::kReject;
    const float cw = __fmaf_rn(v.row_w.x, px, __fmaf_rn(v.row_w.y, py, __fmaf_rn(v.row_w.z, pz, v.row_w.w)));
    const float cx = __fmaf_rn(v.row_x.x, px, __fmaf_rn(v.row_x.y, py, __fmaf_rn(v.row_x.z, pz, v.row_x.w)));
    const float cy = __fmaf_rn(v.row_y.x, px, __fmaf_rn(v.row_y.y, py, __fmaf_rn(v.row_y.z, pz, v.row_y.w)));
    const float cz = __fmaf_rn(v.row_z.x, px, __fmaf_rn(v.row_z.y, py, __fmaf_rn(v.row_z.z, pz, v.row_z.w)));
    const float out = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz)));
    const float margin = 1e-5f * __fmaf_rn(v.matrix_max, fabsf(px) + fabsf(py) + fabsf(pz) + 1.0f, fabsf(cw)) + 1e-7f;
    if (out - cw > margin) return Gate::kReject;
    return facing >= (v.camera.w + 1e-4f) * vl && cw - out > margin && cw > margin ? Gate::kPass : Gate::kUnsure;
}

// Which texel of the atlas a thread of a 128-thread CTA takes. width 0: blockIdx.x * 128 + threadIdx.x. Otherwise a CTA
// takes 16 x 8 texels and a warp 8 x 4: a warp's texels lie on a quarter of the surface's diameter that 32 in a row do,
// so its rays visit the same nodes, its taps the same lines, and its views pass or fail together. Ray casting of a
// 2000 x 1500 atlas from 16 views 3233 -> 2750 us. Narrow atlases stay linear (below 16 most of a CTA lies outside).
struct AtlasTiles {
    uint32_t width;
    FastDiv blocks_x;
    __device__ __forceinline__ uint32_t texel(uint32_t N) const {  // N: none
        if (!width) return blockIdx.x * 128u + threadIdx.x;
        const uint32_t by = blocks_x.quotient(blockIdx.x), bx = blockIdx.x - by * blocks_x.divisor;
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
        const uint32_t x = bx * 16u + (warp & 1u) * 8u + (lane & 7u), y = by * 8u + (warp >> 1) * 4u + (lane >> 3);
        const uint64_t i = (uint64_t)y * width + x;
        return x < width && i < N ? (uint32_t)i : N;
    }
};

inline AtlasTiles atlas_tiles(uint32_t width, uint32_t N, uint32_t& blocks) {
    if (width < 16 || N > 0x7fffffffu) {
        blocks = (uint32_t)(((uint64_t)N + 127) / 128);
        return {0, fast_div(1)};
    }
    const uint32_t bx = (width + 15) / 16;
    blocks = bx * ((N / width + 7) / 8);
    return {width, fast_div(bx)};
}

}  // namespace pdr
