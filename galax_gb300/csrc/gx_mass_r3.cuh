// gx_mass_r3.cuh -- m (r^2)^(-3/2) to the last bit of FP64 without FP64 arithmetic.
//
// GB300 issues two FP64 lanes per clock and SM against 64 integer and 128 FP32 ones
// (measured: DFMA 1.9, IMAD 62, LOP3 63, FFMA 92 lanes per clock and SM), so an
// interaction is bound by the number of its FP64 instructions.  With rsqrt() it had
// 18: two differences, three for r^2, six in rsqrt, three products, two sums and the
// selects.  The factor m r^-3 needs none of them: its mantissa is formed here in 64-bit
// integers from the FP32 reciprocal square root, in about 90 instructions that issue in
// the shadow of the FP64 pipe, and six FP64 instructions are left (dx, dy, two fused
// multiply-adds for r^2, two for the sums).
//
// With r^2 = 2^(2k) z, 1 <= z < 4, and y = rsqrt(z) to 24 bits (|e| < 2^-20,
// e = 1 - z y^2),  z^(-3/2) = y^3 (1 - e)^(-3/2) = y^3 (1 + 3/2 e + 15/8 e^2 + ...)
// (binomial series; the e^3 term is below 2^-58).  e comes from the high half of a
// 64 x 64-bit product, so it is good to 2^-62, and every later step keeps at least 2^-60
// relative: the one rounding that counts is the last, to 53 bits.  Over 2e7 random (r^2, m)
// the result is within 0.52 ulp (rms 0.29); rsqrt() and three products reached 6.3 (1.46).
//
// Measured: the FP64 P2P at Plummer 1M (2.02e9 interactions) 57.3 -> 21.7 ms alone, 93 G
// interactions/s against the pipe's 103 G at six instructions each; the sampled exact sum
// (1000 targets, 1M bodies) 43.7 -> 11.3 ms.
//
// The exponents are kept apart, so no intermediate over- or underflows; r^2 or a mass
// outside 2^-400 .. 2^400 (2^-300 .. 2^300), zero, infinite or NaN takes the plain FP64
// formula and gives what it always gave.
#pragma once
#include <stdint.h>

#include <cuda_runtime.h>

// A mass split for mass_r3: m = mant 2^(ex - 63), 2^63 <= mant < 2^64; span is the
// number of r^2 exponents that the integer path takes with it (0: the plain formula).
struct __align__(16) GxMass {
    uint64_t mant;
    int32_t ex;
    uint32_t span;
};

constexpr int GX_R3_EXP_LO = 1023 - 400;  // biased exponents of r^2: 2^-400 .. 2^400
constexpr uint32_t GX_R3_EXP_SPAN = 801;

__device__ __forceinline__ GxMass gx_mass_split(double m) {
    const uint32_t hi = (uint32_t)__double2hiint(m), lo = (uint32_t)__double2loint(m);
    GxMass g;
    g.mant = ((uint64_t)(0x80000000u | __funnelshift_l(lo, hi, 11)) << 32) | (lo << 11);
    g.ex = (int32_t)(hi >> 20) - 1023;  // a negative mass has a huge exponent here and fails the test
    g.span = (uint32_t)(g.ex + 300) <= 600u ? GX_R3_EXP_SPAN : 0u;
    return g;
}

// z = r^2 2^(-2k) in [1, 4) with y = rsqrt(z) to 24 bits and e = 1 - z y^2
struct GxRoot {
    uint32_t yi;      // y 2^32
    uint64_t y2, y3;  // y^2 2^64 (exact), y^3 2^63
    int64_t e;        // e 2^63
    int k;
};

// hi, lo: the words of r^2, a normal positive FP64 number
__device__ __forceinline__ GxRoot gx_root(uint32_t hi, uint32_t lo) {
    GxRoot r;
    const int ex = (int)(hi >> 20);
    const int odd = (ex & 1) ^ 1;  // the unbiased exponent is 2k + odd
    r.k = (ex - 1023 - odd) >> 1;
    const uint32_t zh = 0x80000000u | __funnelshift_l(lo, hi, 11);
    const uint64_t z63 = ((uint64_t)zh << 32) | (lo << 11);  // z 2^(63 - odd)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;"
        : "=f"(y)
        : "f"(__uint_as_float(((zh >> 8) & 0x7fffffu) | ((uint32_t)(127 + odd) << 23))));
    y = fminf(fmaxf(y, 0.5f), 0x1.fffffep-1f);  // [1/2, 1): one exponent, so the bits are the fraction
    const uint32_t yi = 0x80000000u | (__float_as_uint(y) << 8);  // y 2^32
    r.yi = yi;
    r.y2 = (uint64_t)yi * yi;
    // e 2^63 = 2^63 - z y^2 2^63 (modulo 2^64: the difference fits in 44 bits)
    r.e = (int64_t)(0x8000000000000000ull - (__umul64hi(z63, r.y2) << odd));
    r.y3 = ((uint64_t)(uint32_t)(r.y2 >> 32) * yi + __umulhi((uint32_t)r.y2, yi)) >> 1;
    return r;
}

// mant 2^(ex - 63) r^-N from y^N 2^63 (N = 1, 3 or 5)
template <int N>
__device__ __forceinline__ double gx_root_pow(const GxRoot &r, uint64_t yn, uint64_t mant, int ex) {
    const float ef = (float)(int32_t)(r.e >> 20);  // e 2^43
    const int32_t q = __float2int_rn(ef * ef * ((float)(N * (N + 2)) * 0.125f * 0x1p-23f));  // second order, 2^63
    const int64_t c = (N / 2) * r.e + (r.e >> 1) + q;
    const uint64_t w = yn + (uint64_t)(__mul64hi((int64_t)yn, c << 16) >> 15);  // z^(-N/2) 2^63, in (2^-N, 1]
    const uint64_t f = __umul64hi(w, mant);  // times the mass's fraction, 2^62
    const int s = __clz((int)(f >> 32));
    const uint64_t n = f << s;
    const uint64_t d = (n >> 11) + ((n >> 10) & 1u);  // 53 bits, rounded; a carry moves into the exponent
    const int field = 1023 + ex - N * r.k - s;        // the leading bit of d adds 1 to the field
    return __longlong_as_double((long long)(d + ((uint64_t)(uint32_t)field << 52)));
}

// m r2^(-3/2); m is the mass that g was split from
__device__ __forceinline__ double gx_mass_r3(double r2, const GxMass &g, double m) {
    const uint32_t hi = (uint32_t)__double2hiint(r2), lo = (uint32_t)__double2loint(r2);
    if ((hi >> 20) - (uint32_t)GX_R3_EXP_LO >= g.span) {
        const double ir = rsqrt(r2);
        return m * (ir * ir * ir);
    }
    const GxRoot r = gx_root(hi, lo);
    return gx_root_pow<3>(r, r.y3, g.mant, g.ex);
}

// r2^(-3/2) and 3 r2^(-5/2) (the Hessian's factors); 2^-160 <= r2 <= 2^160 on the integer path
__device__ __forceinline__ void gx_r3_3r5(double r2, double &ir3, double &ir5x3) {
    const uint32_t hi = (uint32_t)__double2hiint(r2), lo = (uint32_t)__double2loint(r2);
    if ((hi >> 20) - (uint32_t)(1023 - 160) > 320u) {
        const double ir = rsqrt(r2);
        ir3 = ir * ir * ir;
        ir5x3 = 3.0 * (ir3 * ir * ir);
        return;
    }
    const GxRoot r = gx_root(hi, lo);
    ir3 = gx_root_pow<3>(r, r.y3, 0x8000000000000000ull, 0);
    ir5x3 = gx_root_pow<5>(r, __umul64hi(r.y3, r.y2), 0xc000000000000000ull, 1);
}

// r2^(-1/2)
__device__ __forceinline__ double gx_rsqrt(double r2) {
    const uint32_t hi = (uint32_t)__double2hiint(r2), lo = (uint32_t)__double2loint(r2);
    if ((hi >> 20) - (uint32_t)GX_R3_EXP_LO >= GX_R3_EXP_SPAN) return rsqrt(r2);
    const GxRoot r = gx_root(hi, lo);
    return gx_root_pow<1>(r, (uint64_t)r.yi << 31, 0x8000000000000000ull, 0);
}
