// The raster kernels' division by a viewport size (csrc/ndc_axis.cuh NdcAxis::quotient: a product with the
// rounded reciprocal and two fused steps) against the division, bit for bit: every pixel of every integer size up
// to 2100 and some larger ones, random sizes and origins, and random dividends of moderate size.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

static float quotient(float a, float size) {
    const float rcp = 1.0f / size;
    const float q = a * rcp;
    return std::fmaf(std::fmaf(-q, size, a), rcp, q);
}

static uint32_t bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}

static long bad = 0, total = 0;

static void check(float a, float size) {
    if ((bits(size) & 0x7fffffu) == 0x7fffffu) return;  // left to the division
    ++total;
    const volatile float want = a / size;
    const float w = want, got = quotient(a, size);
    if (bits(w) != bits(got) && bad++ < 10) std::printf("%a / %a: %a, not %a\n", a, size, got, w);
}

int main() {
    auto axis = [](float v0, float size, int n) {
        for (int p = 0; p < n; ++p) check(((float)p - v0 + 0.5f) * 2.0f, size);
    };
    for (int n = 1; n <= 2100; ++n) axis(0.0f, (float)n, n);
    for (int n : {2560, 3000, 3840, 4095, 4096, 7680, 8192, 12345, 16384, 65535}) axis(0.0f, (float)n, n);
    std::mt19937 rng(7);
    std::uniform_real_distribution<float> u(-1.0f, 1.0f);
    for (int k = 0; k < 2000; ++k) axis(u(rng) * 500.0f, std::exp2(u(rng) * 12.0f), 500);
    for (int k = 0; k < 4000000; ++k) check(u(rng) * std::exp2(u(rng) * 80.0f), std::exp2(u(rng) * 19.0f));
    std::printf("%ld quotients, %ld differ\n", total, bad);
    return bad != 0;
}
