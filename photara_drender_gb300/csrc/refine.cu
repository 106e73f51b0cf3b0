// Texture-atlas refinement: view preparation, masked Charbonnier photometric gradient, seam
// gradient, chart-aware total variation and the dense Adam update, plus the native driver that
// launches the whole optimisation or records it as one CUDA graph.
//
// Reference path: src/texture_refiner.cpp:174-454, shaders/atlas_photometric_gradient.hlsl,
// atlas_seam_gradient.hlsl, atlas_adam_update.hlsl; total variation from
// python/photara_drender/atlas.py:84-115 (the native reference refiner has none; weight 0 keeps
// the reference's objective).
//
// Atlas state in HBM: texture, gradient, first and second moments, each [H][W][3] fp32 (the
// reference's layout), 16-byte aligned so the dense Adam pass moves float4s.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/pdr_capi.h"
#include "pdr_common.cuh"
#include "pdr_internal.h"

namespace pdr {
namespace {

constexpr int kPhotoThreads = 256;

// The kernels of a refinement follow one another directly, most of them a few microseconds long. Within a run and outside
// of a capture each but the first is launched while its predecessor still runs (programmatic stream serialization: its CTAs
// take the places that come free) and waits here until the predecessor has completed and its writes are visible: 60 steps
// on a 512 x 512 atlas 1787 -> 1515 us, 1000 on 64 x 64 10.9 -> 6.3 ms. Recorded into a graph the same edges gained nothing
// (9.5 and 9.9 ms), so captures get ordinary launches.
// A kernel has begun before its predecessors' writes are final, so what a kernel of the run writes (texture, gradient,
// moments) is read by coherent_load alone, after the wait: no load of it by a non-coherent path, and none that the compiler
// may move ahead of the wait, as it may a plain load through a restrict pointer (volatile assembly keeps its order).
// Everything written depends on such a load. Plain loads through pointers that the wait hands on were slower by 1 to 2% on
// 60 steps of a 512 x 512 atlas (1549 us, so 1521, in turn).
// Views, masks, coordinates, targets, pairs and charts may be read any way: the run's first kernel is launched
// ordinarily, so they were complete before any kernel of the run began. A caller's single step (pdr_refine_photometric and
// the like) follows kernels that may have written them, and is launched ordinarily as well.
__device__ __forceinline__ void wait_predecessor() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ float coherent_load(const float* p) {
    float v;
    asm volatile("ld.global.ca.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ float4 coherent_load(const float4* p) {
    float4 v;
    asm volatile("ld.global.ca.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// overlap: the stream's last work is a kernel of this run.
template <class... Params, class... Args>
cudaError_t launch_step(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t stream, bool overlap, Args... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.stream = stream;
    config.attrs = &attribute;
    if (overlap) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        const bool known = cudaStreamIsCapturing(stream, &capture) == cudaSuccess;
        if (!known) cudaGetLastError();
        config.numAttrs = known && capture == cudaStreamCaptureStatusNone ? 1 : 0;
    }
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// What a view's coordinates and weight come from.
struct ViewUv {
    const float* attributes;  // [V][2], at any address
    const uint3* idx;
    uint32_t V, T;
    float2* uv;      // [P]
    double* weight;  // [PDR_REFINE_WEIGHT_PARTS]: their sum is the sum of the mask
};

// texture_refiner.cpp:228-242: target RGB, mask = clamp(external mask) on covered pixels; with kUv also the texture
// coordinates (interpolate_forward_kernel's arithmetic) and the mask's sum, for which the raster and the mask were read
// twice more: a view of 320 x 240 in one launch of 3 us instead of four of 33, most of it a reduction on one SM.
template <bool kUv>
__global__ void __launch_bounds__(256)
prepare_view_kernel(const float* __restrict__ image, uint32_t C, const float* __restrict__ ext_mask,
                    const float4* __restrict__ raster, size_t P, float* __restrict__ target, float* __restrict__ mask,
                    ViewUv u) {
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    float m = 0.0f;
    if (p < P) {
        const float4 r = raster[p];
        target[p * 3] = image[p * C];
        target[p * 3 + 1] = image[p * C + 1];
        target[p * 3 + 2] = image[p * C + 2];
        if (r.w != 0.0f) {
            m = 1.0f;
            if (ext_mask) {
                const float e = ext_mask[p];
                m = e < 0.0f ? 0.0f : (1.0f < e ? 1.0f : e);  // std::clamp
            }
        }
        mask[p] = m;
        if (kUv) {
            float2 o = make_float2(0.0f, 0.0f);
            const uint32_t id = raster_id(r.w);
            if (id != 0 && id <= u.T) {
                const uint3 v = u.idx[id - 1];
                if (v.x < u.V && v.y < u.V && v.z < u.V) {
                    const float* a = u.attributes + (size_t)v.x * 2;
                    const float* b = u.attributes + (size_t)v.y * 2;
                    const float* c = u.attributes + (size_t)v.z * 2;
                    const float w = 1.0f - r.x - r.y;
                    o.x = r.x * __ldg(a) + r.y * __ldg(b) + w * __ldg(c);
                    o.y = r.x * __ldg(a + 1) + r.y * __ldg(b + 1) + w * __ldg(c + 1);
                }
            }
            u.uv[p] = o;
        }
    }
    if (kUv) {
        __shared__ double sums[8];
        double s = m;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31u) == 0) sums[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < 8; ++k) s += sums[k];
            if (s != 0.0) atomicAdd(u.weight + blockIdx.x % PDR_REFINE_WEIGHT_PARTS, s);
        }
    }
}

struct ClampTaps {
    uint32_t o[4];
    float w[4];
};

// atlas_photometric_gradient.hlsl:56-74 / atlas_seam_gradient.hlsl:31-48 (__float2int_rz saturates and takes NaN to 0)
__device__ __forceinline__ ClampTaps clamp_taps(float u, float v, uint32_t tw, uint32_t th) {
    const float px = u * (float)tw - 0.5f, py = v * (float)th - 0.5f;
    const int32_t bx = __float2int_rz(floorf(px)), by = __float2int_rz(floorf(py));
    const float fx = px - floorf(px), fy = py - floorf(py);
    const uint32_t x0 = (uint32_t)clampi(bx, 0, (int32_t)tw - 1), x1 = (uint32_t)clampi(add1(bx), 0, (int32_t)tw - 1);
    const uint32_t y0 = (uint32_t)clampi(by, 0, (int32_t)th - 1), y1 = (uint32_t)clampi(add1(by), 0, (int32_t)th - 1);
    ClampTaps t;
    t.o[0] = y0 * tw + x0;
    t.o[1] = y0 * tw + x1;
    t.o[2] = y1 * tw + x0;
    t.o[3] = y1 * tw + x1;
    t.w[0] = (1.0f - fx) * (1.0f - fy);
    t.w[1] = fx * (1.0f - fy);
    t.w[2] = (1.0f - fx) * fy;
    t.w[3] = fx * fy;
    return t;
}

// The refiner's gradient is [texels][4] (RGB and one unused float), so a bilinear tap adds its three
// channel values with one 16-byte vector reduction instead of three scalar atomics.
__device__ __forceinline__ void red_rgb(float* grad, uint32_t texel, float r, float g, float b) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(grad + (size_t)texel * 4), "f"(r), "f"(g),
                 "f"(b), "f"(0.0f)
                 : "memory");
}

__device__ __forceinline__ float block_sum(float v) {
    __shared__ float warp_sums[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) warp_sums[warp] = v;
    __syncthreads();
    float s = 0.0f;
    if (warp == 0) {
        s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    }
    return s;
}

// One launch covers the batch views of one step (blockIdx.y = batch slot); view choice follows
// texture_refiner.cpp:318-340: view = (step * batch + slot) % view_count.
// Bound by the latency of mask, coordinate and taps, one after the other. A CTA takes `rounds` x 256 pixels, so that
// warps wait for one another once (a third of the time with one pixel a thread) and read ahead. 4 views of 2048 x 1536
// into 4096 x 4096 texels: 256 us with one pixel a thread in 32 registers; with eight 201, in 40 registers 175 (spilling
// fewer), reading ahead in 48 168 (4.2 TB/s of memory traffic, most of it the gradient's lines); sixteen 218, four 177.
__global__ void __launch_bounds__(kPhotoThreads, 5)
photometric_kernel(const float* __restrict__ tex, uint32_t tw, uint32_t th, const pdr_refine_view* __restrict__ views,
                   uint32_t nviews, uint32_t step, uint32_t batch, float eps, float norm, uint32_t rounds,
                   float* __restrict__ grad, float* __restrict__ loss) {
    wait_predecessor();
    const pdr_refine_view v = views[((size_t)step * batch + blockIdx.y) % nviews];
    const float2* const uvs = reinterpret_cast<const float2*>(v.uv);
    float local = 0.0f;
    size_t p = (size_t)blockIdx.x * rounds * kPhotoThreads + threadIdx.x;
    const size_t end = min((size_t)v.pixel_count, p + (size_t)rounds * kPhotoThreads);
    // the next pixel's coordinate and the mask after it are read while this pixel's taps are under way
    const auto mask_at = [&](size_t q) { return q < end ? __ldg(v.mask + q) : 0.0f; };
    const auto uv_at = [&](float m, size_t q) { return m > 0.0f ? __ldg(uvs + q) : make_float2(0.0f, 0.0f); };
    float m_next = mask_at(p), m_after = mask_at(p + kPhotoThreads);
    float2 uv_next = uv_at(m_next, p);
    for (; p < end; p += kPhotoThreads) {
        const float m = m_next;
        const float2 uv = uv_next;
        m_next = m_after;
        uv_next = uv_at(m_next, p + kPhotoThreads);
        m_after = mask_at(p + 2 * kPhotoThreads);
        if (m > 0.0f) {
            const ClampTaps t = clamp_taps(uv.x, uv.y, tw, th);
            float og[3];
#pragma unroll
            for (uint32_t c = 0; c < 3; ++c) {
                float rendered = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k) rendered += coherent_load(tex + (size_t)t.o[k] * 3 + c) * t.w[k];
                const float d = rendered - v.target[p * 3 + c];
                const float robust = sqrtf(d * d + eps * eps);
                og[c] = d / robust * m * norm;
                local += robust * m * norm;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) red_rgb(grad, t.o[k], og[0] * t.w[k], og[1] * t.w[k], og[2] * t.w[k]);
        }
    }
    const float s = block_sum(local);
    if (threadIdx.x == 0 && s != 0.0f) atomicAdd(loss + step, s);
}

// atlas_seam_gradient.hlsl:50-100
__global__ void seam_kernel(const float* __restrict__ tex, uint32_t tw, uint32_t th, const float4* __restrict__ pairs,
                            uint32_t npairs, float eps, float norm, float* __restrict__ grad, float* __restrict__ loss,
                            uint32_t loss_index) {
    wait_predecessor();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float local = 0.0f;
    if (i < npairs) {
        const float4 pr = pairs[i];
        const ClampTaps a = clamp_taps(pr.x, pr.y, tw, th);
        const ClampTaps b = clamp_taps(pr.z, pr.w, tw, th);
        float g[3];
#pragma unroll
        for (uint32_t c = 0; c < 3; ++c) {
            float c0 = 0.0f, c1 = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c0 += coherent_load(tex + (size_t)a.o[k] * 3 + c) * a.w[k];
                c1 += coherent_load(tex + (size_t)b.o[k] * 3 + c) * b.w[k];
            }
            const float d = c0 - c1;
            const float robust = sqrtf(d * d + eps * eps);
            g[c] = d / robust * norm;
            local += robust * norm;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            red_rgb(grad, a.o[k], g[0] * a.w[k], g[1] * a.w[k], g[2] * a.w[k]);
            red_rgb(grad, b.o[k], -g[0] * b.w[k], -g[1] * b.w[k], -g[2] * b.w[k]);
        }
    }
    const float s = block_sum(local);
    if (threadIdx.x == 0 && s != 0.0f) atomicAdd(loss + loss_index, s);
}

// One pair term of the chart-aware TV gradient, d / sqrt(d^2 + eps^2) * scale, with the reciprocal
// square root (about 2 ulp) in place of a square root and an IEEE division: the TV gradient is held to
// a tolerance (atlas.py's autograd, 1e-6 relative), and the exact form made the fused TV + Adam pass
// instruction-bound (12 square roots and divisions per texel).
__device__ __forceinline__ float tv_term(float d, float eps, float scale) { return d * rsqrtf(d * d + eps * eps) * scale; }

// Chart-aware robust total variation of atlas.py:84-115 added into the gradient: each valid
// same-chart neighbour pair (right and down) contributes d / sqrt(d^2 + eps^2) * scale.
__global__ void tv_kernel(const float* __restrict__ tex, uint32_t tw, uint32_t th, const uint8_t* __restrict__ valid,
                          const int32_t* __restrict__ chart, float eps, float scale, float* __restrict__ grad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tw * th) return;
    const uint32_t x = i % tw, y = i / tw;
    if (!valid[i]) return;
    float g[3] = {0.0f, 0.0f, 0.0f};
    const int32_t ci = chart ? chart[i] : 0;
    // pairs (i, right), (i, down) subtract; pairs (left, i), (up, i) add
    const int64_t nb[4] = {x + 1 < tw ? (int64_t)i + 1 : -1, y + 1 < th ? (int64_t)i + tw : -1,
                           x > 0 ? (int64_t)i - 1 : -1, y > 0 ? (int64_t)i - tw : -1};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (nb[k] < 0) continue;
        const size_t j = (size_t)nb[k];
        if (!valid[j] || (chart && chart[j] != ci)) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float d = k < 2 ? tex[j * 3 + c] - tex[(size_t)i * 3 + c] : tex[(size_t)i * 3 + c] - tex[j * 3 + c];
            const float gg = tv_term(d, eps, scale);
            g[c] += k < 2 ? -gg : gg;
        }
    }
    float4* gp = reinterpret_cast<float4*>(grad) + i;
    float4 cur = *gp;
    cur.x += g[0];
    cur.y += g[1];
    cur.z += g[2];
    *gp = cur;
}

// One step's Adam constants. Divisions by the bias corrections are NdcAxis' quotients by a fixed divisor where these are
// exact: six of the nine divisions of a texel, of which the passes over the atlas were as much bound as by its bytes.
struct AdamStep {
    float lr, b1, b2, eps, bc1, bc2, r1, r2, cmin, cmax;
    bool exact;  // quotients by bc1 and bc2
    bool still;  // a texel without gradient and moments keeps its value
};

inline AdamStep adam_step(float lr, float b1, float b2, float eps, float bc1, float bc2, float cmin, float cmax) {
    const auto usable = [](float b) {
        uint32_t bits;
        std::memcpy(&bits, &b, 4);
        return b >= 1e-6f && b <= 1e6f && (bits & 0x7fffffu) != 0x7fffffu;
    };
    const bool exact = usable(bc1) && usable(bc2);
    const bool still = exact && std::isfinite(lr) && eps > 0.0f && b1 >= 0.0f && b1 <= 1.0f && b2 >= 0.0f && b2 <= 1.0f;
    return {lr, b1, b2, eps, bc1, bc2, 1.0f / bc1, 1.0f / bc2, cmin, cmax, exact, still};
}

__device__ __forceinline__ float fixed_quotient(float a, float b, float r) {
    const float q = a * r;
    return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// atlas_adam_update.hlsl:20-43 for the three values of one texel.
__device__ __forceinline__ void adam_texel(float (&x)[3], const float (&g)[3], float (&m)[3], float (&v)[3],
                                           const AdamStep& s) {
    uint32_t any = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) any |= __float_as_uint(g[c]) | __float_as_uint(m[c]) | __float_as_uint(v[c]);
    if (!any && s.still) {  // zero moments stay zero and the step is zero
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = clamp_hlsl(x[c], s.cmin, s.cmax);
        return;
    }
    float lo = INFINITY, hi = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        m[c] = s.b1 * m[c] + (1.0f - s.b1) * g[c];
        v[c] = s.b2 * v[c] + (1.0f - s.b2) * g[c] * g[c];
        lo = fminf(lo, fminf(fabsf(m[c]), fabsf(v[c])));
        hi = fmaxf(hi, fmaxf(fabsf(m[c]), fabsf(v[c])));
    }
    float c1[3], c2[3];
    if (s.exact && lo >= 1e-30f && hi <= 1e25f) {  // no product or remainder underflows: 2^-46 of lo is still a float
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            c1[c] = fixed_quotient(m[c], s.bc1, s.r1);
            c2[c] = fixed_quotient(v[c], s.bc2, s.r2);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            c1[c] = m[c] / s.bc1;
            c2[c] = v[c] / s.bc2;
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) x[c] = clamp_hlsl(x[c] - s.lr * c1[c] / (sqrtf(c2[c]) + s.eps), s.cmin, s.cmax);
}

// The gradient of a texel no tap has touched since it was cleared is zero already: not written again.
__device__ __forceinline__ void clear_gradient(float4* g, const float4& was) {
    if (__float_as_uint(was.x) | __float_as_uint(was.y) | __float_as_uint(was.z) | __float_as_uint(was.w))
        *g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

__global__ void adam_kernel(float* __restrict__ tex, float* __restrict__ grad, float* __restrict__ m1,
                            float* __restrict__ m2, size_t texels, AdamStep s) {
    wait_predecessor();
    // one texel per thread: texture and moments [texels][3], gradient [texels][4] read and cleared as one
    // float4 (four texels per thread, or four values with the gradient gathered, were slower). 16.8 M texels of which
    // few have moments, a seam polish step: 330 us writing every value and dividing nine times; with the quotients and
    // without rewriting zero gradients 291, without rewriting unchanged texels 199, without their arithmetic 132.
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < texels; t += stride) {
        const float4 d = coherent_load(reinterpret_cast<const float4*>(grad) + t);
        const float g[3] = {d.x, d.y, d.z};
        float x[3], m[3], v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x[c] = coherent_load(tex + t * 3 + c);
            m[c] = coherent_load(m1 + t * 3 + c);
            v[c] = coherent_load(m2 + t * 3 + c);
        }
        const float was[9] = {x[0], x[1], x[2], m[0], m[1], m[2], v[0], v[1], v[2]};
        adam_texel(x, g, m, v, s);
        // a texel that no view has reached keeps its value and its zero moments: nothing to write
        uint32_t changed = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            changed |= (__float_as_uint(x[c]) ^ __float_as_uint(was[c])) |
                       (__float_as_uint(m[c]) ^ __float_as_uint(was[3 + c])) |
                       (__float_as_uint(v[c]) ^ __float_as_uint(was[6 + c]));
        if (changed) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                tex[t * 3 + c] = x[c];
                m1[t * 3 + c] = m[c];
                m2[t * 3 + c] = v[c];
            }
        }
        clear_gradient(reinterpret_cast<float4*>(grad) + t, d);
    }
}

struct TvTexel {
    float c[3];
    int32_t chart;
    bool valid;
};

__device__ __forceinline__ TvTexel load_tv(const float* __restrict__ tex, const uint8_t* __restrict__ valid,
                                           const int32_t* __restrict__ chart, size_t t, bool inside) {
    TvTexel o = {{0.0f, 0.0f, 0.0f}, 0, false};
    if (inside) {
#pragma unroll
        for (int c = 0; c < 3; ++c) o.c[c] = coherent_load(tex + t * 3 + c);
        o.valid = __ldg(valid + t) != 0;
        if (chart) o.chart = __ldg(chart + t);
    }
    return o;
}

// The terms of the pair (a, b), b to the right of or below a: subtracted from a's gradient, added to b's.
__device__ __forceinline__ void pair_terms(const TvTexel& a, const TvTexel& b, float eps, float scale, float (&o)[3]) {
    const bool pair = a.valid && b.valid && a.chart == b.chart;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float term = tv_term(b.c[c] - a.c[c], eps, scale);
        o[c] = pair ? term : 0.0f;
    }
}

// The TV gradient of tv_kernel added to the photometric gradient, then the Adam update of adam_kernel into tex_out: one
// pass over the atlas for a step with total variation. tex_in and tex_out are different buffers, so every texel reads
// its neighbours' values from before the step, as the separate TV pass does. Bit-identical to tv_kernel followed by
// adam_kernel (a term left out there is a zero added here, to a sum that is never -0).
// A warp walks down `rows` rows of 32 columns: each pair's terms are computed once, the right ones shuffled to the next
// lane and the lower ones kept for the next row, and a texel's own values are read once. Bound by memory traffic (93 to
// 109 bytes a texel, 5.3 TB/s) and nearly as much by issue. 16.8 M texels: one texel a thread with all four neighbours'
// terms 379 us, this 312; without any of the arithmetic 286. Rows fetched ahead into registers 343, by asynchronous copies
// into shared memory 324 to 350: neither pays for the warps it costs.
__global__ void __launch_bounds__(256)
adam_tv_kernel(const float* __restrict__ tex_in, float* __restrict__ tex_out, float* __restrict__ grad,
               float* __restrict__ m1, float* __restrict__ m2, uint32_t tw, uint32_t th,
               const uint8_t* __restrict__ valid, const int32_t* __restrict__ chart, float tv_eps, float tv_scale,
               uint32_t rows, AdamStep s) {
    wait_predecessor();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t x = blockIdx.x * 256u + threadIdx.x;
    const uint32_t y0 = blockIdx.y * rows, y1 = min(y0 + rows, th);
    if (x - lane >= tw) return;
    const bool in = x < tw;
    // lanes 0 and 31 also read their outer neighbour
    const uint32_t ex = lane == 0 ? x - 1 : x + 1;
    const bool edge = (lane == 0 || lane == 31) && ex < tw;  // x - 1 wraps at x = 0
    size_t t = (size_t)y0 * tw + x;
    TvTexel cur = load_tv(tex_in, valid, chart, t, in);
    float up[3] = {0.0f, 0.0f, 0.0f};
    if (y0) pair_terms(load_tv(tex_in, valid, chart, t - tw, in), cur, tv_eps, tv_scale, up);
    for (uint32_t y = y0; y < y1; ++y, t += tw) {
        const TvTexel below = load_tv(tex_in, valid, chart, t + tw, in && y + 1 < th);
        const TvTexel side = load_tv(tex_in, valid, chart, t - x + ex, edge);
        float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float m[3] = {0.0f, 0.0f, 0.0f}, v[3] = {0.0f, 0.0f, 0.0f};
        if (in) {
            d = coherent_load(reinterpret_cast<const float4*>(grad) + t);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                m[c] = coherent_load(m1 + t * 3 + c);
                v[c] = coherent_load(m2 + t * 3 + c);
            }
        }
        TvTexel next;
#pragma unroll
        for (int c = 0; c < 3; ++c) next.c[c] = __shfl_down_sync(0xffffffffu, cur.c[c], 1);
        next.chart = __shfl_down_sync(0xffffffffu, cur.chart, 1);
        next.valid = __shfl_down_sync(0xffffffffu, (int)cur.valid, 1);
        if (lane == 31) next = side;
        float right[3], left[3], down[3];
        pair_terms(cur, next, tv_eps, tv_scale, right);
#pragma unroll
        for (int c = 0; c < 3; ++c) left[c] = __shfl_up_sync(0xffffffffu, right[c], 1);
        if (lane == 0) pair_terms(side, cur, tv_eps, tv_scale, left);
        pair_terms(cur, below, tv_eps, tv_scale, down);
        float g[3] = {d.x, d.y, d.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float sum = ((0.0f - right[c]) - down[c]) + left[c] + up[c];
            if (cur.valid) g[c] += sum;
            up[c] = down[c];
        }
        if (in) {
            float xv[3] = {cur.c[0], cur.c[1], cur.c[2]};
            adam_texel(xv, g, m, v, s);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                tex_out[t * 3 + c] = xv[c];
                m1[t * 3 + c] = m[c];
                m2[t * 3 + c] = v[c];
            }
            clear_gradient(reinterpret_cast<float4*>(grad) + t, d);
        }
        cur = below;
    }
}

}  // namespace

cudaError_t launch_adam_tv(const float* tex_in, float* tex_out, float* grad, float* m, float* v, uint32_t tw,
                           uint32_t th, const uint8_t* valid, const int32_t* chart, float tv_eps, float tv_scale,
                           float lr, float b1, float b2, float eps, float bc1, float bc2, float cmin, float cmax,
                           cudaStream_t stream, bool overlap) {
    // rows per warp: eight where the atlas still fills the chip several times, fewer below
    uint32_t rows = 8;
    const uint64_t strips = (uint64_t)((tw + 255) / 256) * th;  // CTAs at one row each
    while (rows > 1 && strips / rows < (uint32_t)num_sms() * 16u) rows >>= 1;
    if ((th + rows - 1) / rows > 65535u) rows = (th + 65534u) / 65535u;
    const dim3 grid((tw + 255) / 256, (th + rows - 1) / rows);
    return launch_step(adam_tv_kernel, grid, 256, stream, overlap, tex_in, tex_out, grad, m, v, tw, th, valid, chart, tv_eps, tv_scale,
                       rows, adam_step(lr, b1, b2, eps, bc1, bc2, cmin, cmax));
}

cudaError_t launch_prepare_view(const float* image, uint32_t C, const float* ext_mask, const float* raster, size_t P,
                                float* target, float* mask, cudaStream_t stream, const float* uv_attributes, uint32_t V,
                                const uint32_t* idx, uint32_t T, float* uv, double* weight) {
    const ViewUv u{uv_attributes, reinterpret_cast<const uint3*>(idx), V, T,
                   reinterpret_cast<float2*>(uv), weight};
    const auto kernel = uv ? prepare_view_kernel<true> : prepare_view_kernel<false>;
    kernel<<<(unsigned)((P + 255) / 256), 256, 0, stream>>>(image, C, ext_mask, reinterpret_cast<const float4*>(raster), P,
                                                            target, mask, u);
    return cudaGetLastError();
}

cudaError_t launch_photometric(const float* tex, uint32_t tw, uint32_t th, const pdr_refine_view* views,
                               uint32_t nviews, uint64_t max_pixels, uint32_t step, uint32_t batch, float eps,
                               float norm, float* grad, float* loss, cudaStream_t stream, bool overlap) {
    // pixels per thread: eight where the step still fills the chip, fewer below (4 views of 320 x 240: two 6.2 us, one
    // 7.5, four 6.9)
    uint32_t rounds = 8;
    while (rounds > 1 && max_pixels * batch / (kPhotoThreads * rounds) < (uint32_t)num_sms() * 3u) rounds >>= 1;
    const uint64_t per = (uint64_t)kPhotoThreads * rounds;
    const dim3 grid((unsigned)((max_pixels + per - 1) / per), batch);
    return launch_step(photometric_kernel, grid, kPhotoThreads, stream, overlap, tex, tw, th, views, nviews, step, batch, eps, norm,
                       rounds, grad, loss);
}

cudaError_t launch_seam(const float* tex, uint32_t tw, uint32_t th, const float* pairs, uint32_t npairs, float eps,
                        float norm, float* grad, float* loss, uint32_t loss_index, cudaStream_t stream, bool overlap) {
    return launch_step(seam_kernel, (npairs + 255) / 256, 256, stream, overlap, tex, tw, th, reinterpret_cast<const float4*>(pairs),
                       npairs, eps, norm, grad, loss, loss_index);
}

cudaError_t launch_tv(const float* tex, uint32_t tw, uint32_t th, const uint8_t* valid, const int32_t* chart, float eps,
                      float scale, float* grad, cudaStream_t stream) {
    tv_kernel<<<(tw * th + 255) / 256, 256, 0, stream>>>(tex, tw, th, valid, chart, eps, scale, grad);
    return cudaGetLastError();
}

cudaError_t launch_adam(float* tex, float* grad, float* m, float* v, size_t n, float lr, float b1, float b2, float eps,
                        float bc1, float bc2, float cmin, float cmax, cudaStream_t stream, bool overlap) {
    // n = texels * 3 values. One texel per thread (the loop strides only past 2^31 blocks): a grid capped at
    // eight CTAs per SM that looped over the arrays kept fewer loads in flight
    const size_t texels = n / 3;
    size_t blocks = (texels + 255) / 256;
    if (blocks > 0x7FFFFFFFu) blocks = 0x7FFFFFFFu;
    if (blocks == 0) blocks = 1;
    return launch_step(adam_kernel, (unsigned)blocks, 256, stream, overlap, tex, grad, m, v, texels,
                       adam_step(lr, b1, b2, eps, bc1, bc2, cmin, cmax));
}

// texture_refiner.cpp:316-415: the per-step scalars in the reference's float arithmetic.
void refine_schedule(const pdr_refine_options* o, uint32_t step, float* lr, float* bc1, float* bc2) {
    const float pi = std::acos(-1.0F);
    const float phase = static_cast<float>(step) / static_cast<float>(o->steps);
    *lr = o->minimum_learning_rate +
          0.5F * (o->learning_rate - o->minimum_learning_rate) * (1.0F + std::cos(pi * phase));
    *bc1 = 1.0F - std::pow(o->adam_beta1, static_cast<float>(step + 1));
    *bc2 = 1.0F - std::pow(o->adam_beta2, static_cast<float>(step + 1));
}

}  // namespace pdr
