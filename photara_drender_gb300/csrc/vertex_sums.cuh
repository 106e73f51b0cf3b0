// Per-pixel vertex gradients summed over a warp's pixels on the same triangle before they are added to memory.
//
// Each lane puts what its pixel adds to every corner into shared memory; then one lane per (triangle, corner,
// value) sums the triangle's pixels in lane order and issues one atomic. Lanes next to each other take the values
// of one vertex, so a warp's atomics of a row of the output leave as one request. Neighbouring pixels mostly share a
// triangle: of 200k triangles at 1024 x 1024 a warp of 32 pixels in a row sees 10 to 13.
#pragma once

#include <cuda_runtime.h>

#include "pdr_common.cuh"

namespace pdr {

template <int kVals>
struct VertexSums {
    static constexpr int kPitch = kVals | 1;  // odd: the lanes' values of one index lie in different banks
    float vals[32][kPitch];
    uint4 triangles[32];  // vertices, lanes
};

// Called by whole warps. A valid lane's vals are set; value(s, lane, corner, c) forms what pixel `lane` adds to value
// c of a corner (c < count), add(vertex, c, sum) adds it. id: the triangle, equal exactly for equal triangles.
template <int kVals, class Value, class Add>
__device__ __forceinline__ void add_vertex_sums(VertexSums<kVals>& s, bool valid, uint32_t id, uint3 vi, uint32_t count,
                                                Value&& value, Add&& add) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    const unsigned same = __match_any_sync(0xffffffffu, valid ? id : (0x80000000u | lane));
    const bool leader = valid && (same & below) == 0u;
    const unsigned leaders = __ballot_sync(0xffffffffu, leader);
    if (leaders == 0u) return;
    if (leader) s.triangles[__popc(leaders & below)] = make_uint4(vi.x, vi.y, vi.z, same);
    __syncwarp();
    const uint32_t per = 3u * count, tasks = (uint32_t)__popc(leaders) * per;
    for (uint32_t task = lane; task < tasks; task += 32) {
        const uint32_t g = task / per, k = task - g * per, corner = k / count, c = k - corner * count;
        const uint4 t = s.triangles[g];
        float sum = 0.0f;
        for (uint32_t lanes = t.w; lanes; lanes &= lanes - 1u) sum += value(s, (uint32_t)__ffs(lanes) - 1u, corner, c);
        add(corner == 0 ? t.x : (corner == 1 ? t.y : t.z), c, sum);
    }
    __syncwarp();
}

}  // namespace pdr
