// cumc_round.cuh — correctly rounded FP64 quotients and square roots without
// branches, for the Riemann solver.
//
// A face's HLL solve forms 21 quotients by only five divisors and eight
// square roots. Written with `/` and sqrt each of them carries its own range
// test and branch to a slow path, which cuts the solve into 29 short serial
// pieces that cannot overlap and repeats the divisor's reciprocal for every
// quotient. Here the reciprocal of a divisor is formed once and every quotient
// by it costs four multiply-adds; the caller checks the operand ranges once a
// face and takes the plain operators for a face outside them, so that the
// results are the IEEE ones, bit for bit, in every case.
//
// Method: Newton-Raphson from the hardware's approximate reciprocal (or
// reciprocal square root), then the remainder correction of P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990, which a fused multiply-add makes
// exact.
//
// Quotient a/b. Scale b to an integer in [2^52, 2^53). The corrected quotient
// q' = RN(q + r y), r = a - b q, differs from a/b before its rounding by
// |a/b - q| b |y - 1/b|. A quotient lies at least 2^-53/b (in units of a
// quotient in [1, 2)) from a rounding midpoint, and next to one |a/b - q| is
// half a unit in the last place, so q' is the rounded quotient when q is
// within one unit and |y - 1/b| < 1/b^2. y = RN(1/b) satisfies that. The last
// Newton step gives it unless 1/b lies above a midpoint by at most four units
// of 2^-106/b; y1 is rounded upwards so that the one divisor where the miss
// would count (all significand bits set) starts from the upper side and is
// rounded right. q takes the reciprocal's own remainder along (a y + a lo),
// which keeps it within one unit.
//
// Square root. With g within one unit of sqrt(a) and h within 2^-52 (relative)
// of 1/(2 sqrt(a)), g' = RN(g + h (a - g^2)) is the rounded root: on the scale
// where the neglected second-order term is 1, a root is N away from its
// nearest midpoint with N = 7 mod 8, so it keeps its side unless N = -1.
// Only two significands have N = -1 (all bits set, and one above a power of
// two); their result depends on the seed, and the hardware's gives the rounded
// root over both exponent parities (tests/test_round.py).
//
// Ranges: a quotient needs b in 2^+-500, a finite, and a/b, unless a is zero, a
// normal number with its remainder above the subnormal ones; roots need a in
// 2^+-900. quot_group tests b in [2^-200, 2^200) and |a| zero or in
// [2^-800, 2^800), so that a/b lies in 2^+-1000.
#pragma once
#include <cfenv>
#include <cmath>
#include <cstring>
#ifdef __CUDACC__
#define CUMC_HD __host__ __device__ __forceinline__
#else
#define CUMC_HD inline
#endif

namespace cumc {

struct Recip {
    double y, lo;  // y + lo = 1/b to about 2^-100
};

// a b + c rounded upwards
CUMC_HD double fma_up(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_ru(a, b, c);
#else
    std::fesetround(FE_UPWARD);
    volatile double x = a, y = b, z = c;
    volatile double r = std::fma(x, y, z);
    std::fesetround(FE_TONEAREST);
    return r;
#endif
}
// b's reciprocal to within a unit from an approximation y0 with a relative
// error of at most 2^-19
CUMC_HD double recip_near(double b, double y0) {
    const double e = std::fma(-b, y0, 1.0);
    return fma_up(y0, std::fma(e, e, e), y0);
}
CUMC_HD Recip recip_refine(double b, double y0) {
    const double y1 = recip_near(b, y0);
    Recip r;
    r.y = std::fma(std::fma(-b, y1, 1.0), y1, y1);
    r.lo = std::fma(-b, r.y, 1.0) * r.y;
    return r;
}
// a/b, rounded to nearest; a zero comes back with the sign of an unspecified
// zero (quot_signed keeps a's)
CUMC_HD double quot(double a, double b, const Recip& r) {
    const double q = std::fma(a, r.lo, a * r.y);
    return std::fma(std::fma(-b, q, a), r.y, q);
}
// sqrt(a) from an approximation y0 of 1/sqrt(a) with a relative error of at
// most 2^-19; a > 0
CUMC_HD double root_refine(double a, double y0) {
    const double g0 = a * y0, h0 = 0.5 * y0;
    const double r0 = std::fma(-g0, h0, 0.5);  // (1 - a y0^2)/2
    const double s = std::fma(1.5 * r0, r0, r0);
    const double g = std::fma(g0, s, g0), h = std::fma(h0, s, h0);
    return std::fma(std::fma(-g, g, a), h, g);
}

// the approximate reciprocal (on the host, where only the tests come, with a
// relative error of the same size)
CUMC_HD double recip_seed(double b) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
#else
    return 1.0 / b * (1.0 + 0x1p-20);
#endif
}
CUMC_HD Recip recip_of(double b) { return recip_refine(b, recip_seed(b)); }
// a/b with a zero's sign kept; b > 0
CUMC_HD double quot_signed(double a, double b, const Recip& r) { return std::copysign(quot(a, b, r), a); }

// Out-of-range tracking on the two words of a double, integer pipe only (one
// instruction each for the sums with a minimum or maximum)
CUMC_HD unsigned hi_word(double x) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x);
#else
    unsigned long long u;
    std::memcpy(&u, &x, sizeof u);
    return (unsigned)(u >> 32);
#endif
}
CUMC_HD unsigned lo_word(double x) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(x);
#else
    unsigned long long u;
    std::memcpy(&u, &x, sizeof u);
    return (unsigned)u;
#endif
}
CUMC_HD unsigned add_max(unsigned a, unsigned b, unsigned m) {
#ifdef __CUDA_ARCH__
    return __viaddmax_u32(a, b, m);
#else
    return a + b > m ? a + b : m;
#endif
}
CUMC_HD unsigned add_min(unsigned a, unsigned b, unsigned m) {
#ifdef __CUDA_ARCH__
    return __viaddmin_u32(a, b, m);
#else
    return a + b < m ? a + b : m;
#endif
}
// range_max accumulates max(hi - lo_word) so that one unsigned compare covers
// several positive operands. magnitude orders a double by its size (twice the
// high word, and one for low bits: 0 for a zero alone, an infinity or a NaN above
// every number); tiny_min accumulates the smallest nonzero one less one (a zero
// counts as the largest)
constexpr unsigned RANGE_LO = (1023u - 200u) << 20, RANGE_SPAN = 400u << 20;  // [2^-200, 2^200)
CUMC_HD unsigned range_max(double x, unsigned m) { return add_max(hi_word(x), 0u - RANGE_LO, m); }
constexpr unsigned TINY = ((1023u - 800u) << 21) - 1u;  // 2^-800's magnitude, less one
constexpr unsigned HUGE_MAG = (1023u + 800u) << 21;     // 2^800's
CUMC_HD unsigned magnitude(double x) {
    const unsigned hi = hi_word(x), lo = lo_word(x);
    return hi + hi + (lo < 1u ? lo : 1u);
}
CUMC_HD unsigned tiny_min(unsigned mag, unsigned m) { return add_min(mag, ~0u, m); }

// a/b out of line, for the rare groups below
#ifdef __CUDACC__
static __host__ __device__ __noinline__ double plain_quot(double a, double b) { return a / b; }
#else
inline double plain_quot(double a, double b) { return a / b; }
#endif

// q[n] = a[n]/b for N numerators, the shared reciprocal
// where b and the numerators are in range, else the plain operator
// (a front that fades into a zero field carries numerators down through the
// denormals, so the test stands here and not around a whole face or cell)
template <int N>
CUMC_HD void quot_group(const double (&a)[N], double b, double (&q)[N]) {
    unsigned tiny = ~0u, huge = 0u;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int n = 0; n < N; ++n) {
        const unsigned mag = magnitude(a[n]);
        tiny = tiny_min(mag, tiny);
        huge = mag > huge ? mag : huge;
    }
    if (range_max(b, 0u) < RANGE_SPAN && tiny >= TINY && huge < HUGE_MAG) {
        const Recip r = recip_of(b);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int n = 0; n < N; ++n) q[n] = quot_signed(a[n], b, r);
    } else {
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int n = 0; n < N; ++n) q[n] = plain_quot(a[n], b);
    }
}

#ifdef __CUDACC__
__device__ __forceinline__ double rsqrt_seed(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return y;
}
__device__ __forceinline__ double root_of(double a) { return root_refine(a, rsqrt_seed(a)); }
// sqrt(max(a, 0))
__device__ __forceinline__ double root_pos(double a) { return __double_as_longlong(a) > 0 ? root_of(a) : 0.0; }

// FP32 reciprocal and root, rounded to nearest (the results of 1.0f/x and
// sqrtf, checked over every significand by the tests): one Newton step from
// the hardware's approximation and the remainder correction. x in 2^+-100.
__device__ __forceinline__ float recip_f(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}
__device__ __forceinline__ float root_f(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float g = x * y;
    return __fmaf_rn(__fmaf_rn(-g, g, x), 0.5f * y, g);
}
// max(bits - bits of 2^LO), as range_max: below `span << 23` for x in [2^LO, 2^(LO + span))
template <int LO>
__device__ __forceinline__ unsigned range_max_f(float x, unsigned m) {
    return __viaddmax_u32(__float_as_uint(x), 0u - ((unsigned)(127 + LO) << 23), m);
}
#endif

}  // namespace cumc
