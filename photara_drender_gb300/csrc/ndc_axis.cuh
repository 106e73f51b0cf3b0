// Sample positions and divisions along one axis of a viewport.
#pragma once

#include <cuda_runtime.h>

#include "pdr_common.cuh"

namespace pdr {

// One axis of a viewport with the reciprocal of its size, for divisions by that size without a division: the
// quotient a / b by a fixed divisor is q = RN(a y), r = RN(a - q b), RN(q + r y) with y = RN(1 / b), which is
// correctly rounded (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990, theorem 8.2) unless b's significand is all ones, and while nothing under- or overflows:
// `exact` and the bounds on a keep both away. Otherwise the division itself.
struct NdcAxis {
    float v0, size, rcp;
    bool exact;
    __device__ __forceinline__ NdcAxis(float origin, float extent) : NdcAxis(origin, extent, 1.0f / extent) {}
    __device__ __forceinline__ NdcAxis(float origin, float extent, float reciprocal)
        : v0(origin), size(extent), rcp(reciprocal) {
        exact = extent >= 1e-6f && extent <= 1e9f && fabsf(origin) <= 1e9f &&
                (__float_as_uint(extent) & 0x7fffffu) != 0x7fffffu;
    }
    __device__ __forceinline__ float quotient(float a) const {  // exact, and a zero or of moderate size
        const float q = a * rcp;
        return __fmaf_rn(__fmaf_rn(-q, size, a), rcp, q);
    }
    // sample_ndc
    __device__ __forceinline__ float at(uint32_t p) const {
        if (!exact) return sample_ndc(p, v0, size);
        return quotient(((float)p - v0 + 0.5f) * 2.0f) - 1.0f;
    }
    // a / size
    __device__ __forceinline__ float divide(float a) const {
        const float m = fabsf(a);
        return exact && m >= 1e-25f && m <= 1e25f ? quotient(a) : a / size;
    }
};

}  // namespace pdr
