// fjb_math.cuh -- FP32 elementary functions of the per-pixel chain on the argument ranges it
// has, each within one or two units in the last place (no further off than the library
// function it stands for), without the library's handling of the rest: callers send
// arguments outside the stated range to the library.
//
// Why: the print/scan chain is bound by instruction issue (2300 per pixel with the general
// functions, division with its range fix-up, log10f, cbrtf, atan2f, hypotf, fmodf and the
// lookups' searches making up more than half). Seeds come from the MUFU, accuracy from one
// Newton-Raphson step on the defining equation; the logarithm is a series, the arctangent a fit,
// both derived here. With the packed spectrum and the table-started lookups: 1720 per pixel,
// 3840x2160 print scan 743 -> 609 us.
// Largest and rms error in ulp against FP64, here and the library, over 6e7 arguments of the
// stated ranges: quotient and root 0.50 / 0.29, the same (correctly rounded); log10 1.39 / 0.38
// and 2.07 / 0.54; cube root 0.74 / 0.31 and 1.16 / 0.33; x^(5/12) 1.23 / 0.34 and, from 0.003
// to 2, where it is used, 1.20 / 0.34 and 1.56 / 0.50; angle 1.74 / 0.37 and 2.05 / 0.47.
#pragma once

#include <cuda_runtime.h>

namespace fjb {

__device__ __forceinline__ float mufu_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float mufu_lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 2^x on the MUFU (ex2.approx.ftz.f32: relative error about 2^-22, flushes subnormal
// results to zero).
__device__ __forceinline__ float mufu_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float mufu_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// a / b for 1e-30 <= |b| <= 1e30 and finite |a| <= 1e30 whose quotient is in range: the
// reciprocal's quotient and one correction by its remainder (Newton-Raphson).
__device__ __forceinline__ float quotient(float a, float b) {
    const float r = mufu_rcp(b);
    const float q = a * r;
    return fmaf(fmaf(-q, b, a), r, q);
}
__device__ __forceinline__ bool divides(float b) {
    const float m = fabsf(b);
    return m >= 1e-30f && m <= 1e30f;
}

// sqrt(x) for 1e-30 <= x <= 1e30 (Newton-Raphson on 1 / sqrt).
__device__ __forceinline__ float root(float x) {
    const float r = mufu_rsqrt(x);
    const float s = x * r;
    return fmaf(fmaf(-s, s, x), 0.5f * r, s);
}

// x = 2^e m with m in [sqrt(1/2), sqrt(2)), and z = (m - 1) / (m + 1), so that
// ln m = 2 artanh z = 2 z (1 + z^2/3 + z^4/5 + ...), |z| <= 0.1716: terms beyond z^8/9 are
// below 3e-9 of the sum. Returns z times the sum beyond its first term. Positive normal x.
__device__ __forceinline__ float log_parts(float x, float& e, float& z) {
    const int i = __float_as_int(x) - 0x3f3504f3; // bits of sqrt(1/2)
    const int n = i >> 23;
    const float m = __int_as_float(__float_as_int(x) - (n << 23));
    e = (float)n;
    const float a = m - 1.0f;          // exact
    const float b = 2.0f + a, c = a - (b - 2.0f); // b + c = m + 1 exactly
    const float r = mufu_rcp(b);
    z = a * r;
    z = fmaf(fmaf(-z, c, fmaf(-z, b, a)), r, z);
    const float s = z * z;
    return z * (s * fmaf(s, fmaf(s, fmaf(s, 1.0f / 9.0f, 1.0f / 7.0f), 1.0f / 5.0f), 1.0f / 3.0f));
}
// Logarithms of positive normal x. Factors in two parts, so that each product's rounding
// falls below the sum's.
__device__ __forceinline__ float log10_normal(float x) {
    float e, z;
    const float q = log_parts(x, e, z);
    constexpr double k = 0.86858896380650365530, l = 0.30102999566398119521; // 2 log10 e, log10 2
    constexpr float kh = (float)k, kl = (float)(k - (double)kh);
    constexpr float lh = 0.301025390625f, ll = (float)(l - (double)lh); // e * lh is exact
    const float low = fmaf(z, kl, fmaf(q, kh, e * ll));
    return fmaf(e, lh, fmaf(z, kh, low));
}
// log10 of any x (the library where x is not positive, not finite or subnormal).
__device__ __forceinline__ float log10_any(float x) {
    return x >= 1e-37f && x <= 3.0e38f ? log10_normal(x) : log10f(x);
}

// Cube root: Newton-Raphson on y^3 = x.
__device__ __forceinline__ float cube_root(float v) {
    const float x = fabsf(v);
    if (!divides(x)) return v < 0.0f ? -cbrtf(-v) : cbrtf(v);
    const float y = mufu_exp2(mufu_lg2(x) * (1.0f / 3.0f));
    const float y2 = y * y;
    return copysignf(fmaf(fmaf(-y2, y, x), mufu_rcp(3.0f * y2), y), v);
}

// x^(1/2.4) = x^(5/12) for 1e-6 <= x <= 1e6: Newton-Raphson on y^12 = x^5 (the products'
// rounding reaches the result divided by twelve).
__device__ __forceinline__ float pow_5_12(float x) {
    const float y = mufu_exp2(mufu_lg2(x) * (5.0f / 12.0f));
    const float y2 = y * y, y4 = y2 * y2, y8 = y4 * y4, y12 = y8 * y4;
    const float x2 = x * x, x4 = x2 * x2, x5 = x4 * x;
    return fmaf(y * (1.0f / 12.0f), (x5 - y12) * mufu_rcp(y12), y);
}

// Angle of (x, y), not both zero, larger magnitude in quotient's range: an odd fit of
// arctan(q) / q on [0, 1] in q^2 (relative error 2.3e-8), octants by symmetry.
__device__ __forceinline__ float angle(float y, float x) {
    const float a = fabsf(x), b = fabsf(y);
    const bool steep = b > a;
    const float q = quotient(steep ? a : b, steep ? b : a);
    const float s = q * q;
    float p = 0.002920683706179261f;
    p = fmaf(p, s, -0.016367897391319275f);
    p = fmaf(p, s, 0.043211814016103745f);
    p = fmaf(p, s, -0.07552210986614227f);
    p = fmaf(p, s, 0.10666003078222275f);
    p = fmaf(p, s, -0.14211055636405945f);
    p = fmaf(p, s, 0.19993773102760315f);
    p = fmaf(p, s, -0.33333152532577515f);
    p = fmaf(p * s, q, q);
    // pi in two parts
    p = steep ? 1.57079637050628662109f - (p + 4.37113900018624283e-8f) : p;
    p = x < 0.0f ? 3.14159274101257324219f - (p + 8.74227800037248566e-8f) : p;
    return copysignf(p, y);
}

} // namespace fjb
