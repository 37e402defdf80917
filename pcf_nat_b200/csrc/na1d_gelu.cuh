// The normal distribution function of GELU, x Phi(x), and its derivative, Phi(x) + x phi(x): one value at a time for the passes over memory,
// two at a time for the kernels that keep the hidden layer on chip. Both forms do the same arithmetic, so that a network gives the same
// values whichever of them its sizes take.
//
// Phi(-|x|) = t P(t) e^{-x^2/2} with t = 1 / (1 + 0.29980 |x|): the substitution of Abramowitz & Stegun 7.1.26, with a polynomial of
// degree 7 fitted to e^{z^2} erfc(z) (relative error 4e-8 for |x| < 5.6, rising to 1e-4 beyond 9). The negative tail is a product, not
// 1 - erf, so it keeps its relative accuracy (in fp32 8e-7 for |x| < 4, 8e-6 to 9, 2e-5 to 12), and e^{-x^2/2} is shared with
// the density in the derivative. Over all bf16 values 94 results round the wrong way, over all fp16 values 3, against 118 and 370 of
// the framework's 1 + erf form (and 161 and 254 with the five terms of 7.1.26). Two special-function operations and ~15 fp32
// operations a value instead of the library erff's ~25 with a branch (165 us for 153600 x 1024 values; 116 us here, 98 us of HBM time).
// Minus infinity gives NaN, as zero times it does in the framework.
#pragma once
#include "na1d_tc_common.cuh"

namespace na1d {
namespace {

constexpr float kPhiSlope = 0.2998046875f;
__device__ __forceinline__ constexpr float phi_coef(int n) {
    constexpr float c[8] = {0.1195935606956482f,   0.12026944756507874f, 0.1013689711689949f,   0.1259254813194275f,
                            -0.05189161375164986f, 0.20701442658901215f, -0.15834912657737732f, 0.0360688753426075f};
    return c[n];
}
constexpr float kDensity = 0.3989422804014327f;   // 1 / sqrt(2 pi)

// e: e^{-x^2/2}
__device__ __forceinline__ void phi(float x, float& cdf, float& e) {
    const float t = tc::fast_rcp(fmaf(kPhiSlope, fabsf(x), 1.f));
    e = tc::fast_exp2(x * x * (-0.5f * kLog2e));
    float p = phi_coef(7);
#pragma unroll
    for (int n = 6; n >= 0; --n) p = fmaf(t, p, phi_coef(n));
    const float tail = p * t * e;
    cdf = x >= 0.f ? 1.f - tail : tail;
}

// pairs of fp32 values in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t&>(d))
        : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)), "l"(reinterpret_cast<const uint64_t&>(c)));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
    return d;
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

__device__ __forceinline__ void phi2(const float2 x, float2& cdf, float2& e) {
    const float2 u = fma2(both(kPhiSlope), make_float2(fabsf(x.x), fabsf(x.y)), both(1.f));
    const float2 t = make_float2(tc::fast_rcp(u.x), tc::fast_rcp(u.y)), y = mul2(mul2(x, x), both(-0.5f * kLog2e));
    e = make_float2(tc::fast_exp2(y.x), tc::fast_exp2(y.y));
    float2 p = both(phi_coef(7));
#pragma unroll
    for (int n = 6; n >= 0; --n) p = fma2(t, p, both(phi_coef(n)));
    p = mul2(p, t);
    // 1 - tail or tail, as one multiplication and addition each
    cdf = fma2(make_float2(x.x >= 0.f ? -p.x : p.x, x.y >= 0.f ? -p.y : p.y), e, make_float2(x.x >= 0.f ? 1.f : 0.f, x.y >= 0.f ? 1.f : 0.f));
}
__device__ __forceinline__ float2 gelu2(const float2 x) {
    float2 cdf, e;
    phi2(x, cdf, e);
    return mul2(x, cdf);
}
__device__ __forceinline__ void gelu_and_slope(const float2 x, float2& value, float2& slope) {
    float2 cdf, e;
    phi2(x, cdf, e);
    value = mul2(x, cdf);
    slope = fma2(mul2(x, both(kDensity)), e, cdf);
}

}  // namespace
}  // namespace na1d
