// Exact emulation of two pieces of host arithmetic the reference Sampler relies on, in a form that
// can run in parallel:
//
//  1. glibc's single-precision expf as x86-64 machines with FMA run it (the result every
//     TemperatureLogitTransform element goes through, src/cpp/src/sampling/logit_transformers.hpp:327-356).
//     The published algorithm: k = round(x * 32 / ln 2), r = x * 32 / ln 2 - k taken with one fused
//     multiply-add, exp(x) = 2^(k / 32) * (1 + r * C2 + r^2 * (C1 + r * C0)) in double precision with a
//     32-entry table of 2^(i / 32), rounded once to float.  The restatement below returns the same
//     bits as that libm for every finite input in [-103.9, 88.7] (checked exhaustively on the host by
//     tests/cpp/fsum_exact_test.cpp over a stride of the range and by the GPU test on the device).
//
//  2. A running float sum `s += x[i]` over non-negative terms in a fixed order
//     (logit_transformers.hpp:343-359, 105-125; sampling/sampler.cpp:1036-1074).  While s stays inside
//     one binade its ulp u is constant and fl(s + x) = s + u * round_half_even(x / u) is an integer
//     addition on S = s / u whose amount depends on S only through its parity (a tie x / u = q + 1/2
//     rounds to the even neighbour).  A term therefore acts as a two-state function
//         S -> S + a   (S even),   S -> S + b   (S odd),
//     and such functions compose associatively, so a block scan reproduces the sequential sum bit
//     for bit.  For a term that is not a tie a == b: those are plain translations and commute, which
//     is what lets a segment of sorted probabilities be summed unsorted (segment_sum.cuh).  A step that
//     leaves the binade (S reaches 2^24) is redone with real float additions.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define FSX_HD __host__ __device__ __forceinline__
#else
#define FSX_HD inline
#include <cmath>
#endif

namespace fsx {

// ---- expf -------------------------------------------------------------------------------------
// 2^(i / 32), i = 0..31, correctly rounded to double, with i << 47 subtracted from the bit pattern so
// that adding k << 47 puts floor(k / 32) into the exponent field.
#define FSX_EXP2_TABLE                                                                                  \
    0x3ff0000000000000ull, 0x3fefd9b0d3158574ull, 0x3fefb5586cf9890full, 0x3fef9301d0125b51ull,         \
    0x3fef72b83c7d517bull, 0x3fef54873168b9aaull, 0x3fef387a6e756238ull, 0x3fef1e9df51fdee1ull,         \
    0x3fef06fe0a31b715ull, 0x3feef1a7373aa9cbull, 0x3feedea64c123422ull, 0x3feece086061892dull,         \
    0x3feebfdad5362a27ull, 0x3feeb42b569d4f82ull, 0x3feeab07dd485429ull, 0x3feea47eb03a5585ull,         \
    0x3feea09e667f3bcdull, 0x3fee9f75e8ec5f74ull, 0x3feea11473eb0187ull, 0x3feea589994cce13ull,         \
    0x3feeace5422aa0dbull, 0x3feeb737b0cdc5e5ull, 0x3feec49182a3f090ull, 0x3feed503b23e255dull,         \
    0x3feee89f995ad3adull, 0x3feeff76f2fb5e47ull, 0x3fef199bdd85529cull, 0x3fef3720dcef9069ull,         \
    0x3fef5818dcfba487ull, 0x3fef7c97337b9b5full, 0x3fefa4afa2a490daull, 0x3fefd0765b6e4540ull,
static const uint64_t kExp2TabHost[32] = {FSX_EXP2_TABLE};
#if defined(__CUDACC__)
// Device copy.  Lanes of a warp index it with different values, and a constant-bank read with divergent addresses is replayed once per
// address: kernels keep an entry in each lane's registers.
static __device__ const uint64_t kExp2TabDev[32] = {FSX_EXP2_TABLE};
#endif

FSX_HD double u64_as_double(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double d; memcpy(&d, &u, 8); return d;
#endif
}
FSX_HD uint64_t double_as_u64(double d) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t u; memcpy(&u, &d, 8); return u;
#endif
}
FSX_HD uint32_t float_bits(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u; memcpy(&u, &f, 4); return u;
#endif
}
FSX_HD float bits_float(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f; memcpy(&f, &u, 4); return f;
#endif
}
FSX_HD double fma_rn(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
FSX_HD double mul_rn(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    return a * b;   // build with -ffp-contract=off
#endif
}
FSX_HD double add_rn(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
FSX_HD float fadd_rn(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}

// The sum and the scaling that every form below shares, for an argument from -104.5 to 88.72; entry(ki) is 2^(k / 32) as a double, from
// the low bits of k + 1.5 * 2^52.
template <class Entry>
FSX_HD float expf_scaled(double xd, Entry entry) {
    const double kInvLn2N = 0x1.71547652b82fep+0 * 32.0;
    const double kShift = 0x1.8p+52;
    const double kC0 = 0x1.c6af84b912394p-5 / 32768.0, kC1 = 0x1.ebfce50fac4f3p-3 / 1024.0, kC2 = 0x1.62e42ff0c52d6p-1 / 32.0;
    double kd = fma_rn(kInvLn2N, xd, kShift);
    const uint64_t ki = double_as_u64(kd);
    kd = add_rn(kd, -kShift);
    const double r = fma_rn(kInvLn2N, xd, -kd);
    const double s = entry(ki);
    const double z = fma_rn(kC0, r, kC1);
    const double r2 = mul_rn(r, r);
    double y = fma_rn(kC2, r, 1.0);
    y = fma_rn(z, r2, y);
    return (float)mul_rn(y, s);
}

// expf(x) with the host libm's bits.  Inputs at or below -103.972 give 0, -inf gives 0, NaN stays NaN;
// arguments above 88.7 do not occur here (the callers pass x - max <= 0) and saturate to +inf.
FSX_HD float expf_libm(float x, const uint64_t* tab) {
    if (!(x >= -103.972076f)) return x != x ? x : 0.0f;       // underflow to zero (and NaN passthrough)
    if (x > 88.72283f) return bits_float(0x7f800000u);
    return expf_scaled((double)x, [tab](uint64_t ki) { return u64_as_double(tab[ki & 31] + (ki << 47)); });
}

// x from -inf to 0 as a double for expf_scaled, in integers: four instructions instead of one at a quarter of the double unit's rate, which
// is a sixteenth of a warp's lanes per cycle.  Below -104.5 the exponential is zero as it is there; zeros and denormals become
// another number that small.
FSX_HD double nonpositive_as_double(float x) {
    const uint32_t b = float_bits(fmaxf(x, -104.5f));
    return u64_as_double((uint64_t)(((b & 0x7fffffffu) >> 3) + 0xb8000000u) << 32 | (b << 29));
}

#if !defined(__CUDA_ARCH__)
inline float expf_libm(float x) { return expf_libm(x, kExp2TabHost); }
#endif

// a / b correctly rounded (what the host's `/=` gives, logit_transformers.hpp:357-359) for a whole row
// that shares the divisor: with y = RN(1 / b), q0 = RN(a y), the remainder a - b q0 is exact in one fused
// multiply-add and RN(q0 + rem y) is the rounded quotient.  Small numerators, whose remainder would
// be a denormal, take the plain division.
FSX_HD float div_shared(float a, float b, float y) {
    if (!(a >= 0x1p-90f)) {
#if defined(__CUDA_ARCH__)
        return __fdiv_rn(a, b);
#else
        return a / b;
#endif
    }
#if defined(__CUDA_ARCH__)
    const float q0 = __fmul_rn(a, y);
    const float rem = __fmaf_rn(-q0, b, a);
    return __fmaf_rn(rem, y, q0);
#else
    const float q0 = a * y;
    const float rem = std::fma(-q0, b, a);
    return std::fma(rem, y, q0);
#endif
}

// ---- running float sums -------------------------------------------------------------------------
constexpr uint32_t kOne24 = 1u << 24;
constexpr uint32_t kSat = 1u << 26;   // amounts saturate here: any state that meets one has left its binade

// A float s >= 0 as (E, S): s = S * 2^(E - 150) with E the biased exponent (1 for zero and denormals,
// where S < 2^23) and S the significand with its hidden bit.
FSX_HD uint32_t state_exp(float s) { const uint32_t e = float_bits(s) >> 23; return e ? e : 1u; }
FSX_HD uint32_t state_sig(float s) {
    const uint32_t b = float_bits(s);
    return (b >> 23) ? ((b & 0x7fffffu) | 0x800000u) : b;
}
FSX_HD float state_float(uint32_t E, uint32_t S) {   // S < 2^24; S < 2^23 only when E == 1
    return bits_float(S >= 0x800000u ? ((E << 23) | (S & 0x7fffffu)) : S);
}

struct Step {
    uint32_t a, b;   // amount added to an even / odd state
};
FSX_HD Step step_identity() { return Step{0u, 0u}; }
FSX_HD uint32_t sat_add(uint32_t x, uint32_t y) { const uint32_t z = x + y; return z > kSat ? kSat : z; }

// g after f
FSX_HD Step then(Step f, Step g) {
    return Step{sat_add(f.a, (f.a & 1u) ? g.b : g.a), sat_add(f.b, ((f.b + 1u) & 1u) ? g.b : g.a)};
}
FSX_HD uint32_t apply(Step f, uint32_t S) { return S + ((S & 1u) ? f.b : f.a); }

}  // namespace fsx
