// wf_math.cuh -- FP64 elementary functions and Julia-Base semantics used by the kernels.
//
// The FP64 form must reproduce Wflow.jl's Float64 arithmetic. Julia's Base semantics that
// matter on the path:
//   * min/max propagate NaN and order -0.0 < +0.0;
//   * clamp(x, lo, hi) = x > hi ? hi : (x < lo ? lo : x);
//   * cld(x, y) for floats = round((x - mod(x, -y)) / y)   (Base.div(x, y, RoundUp));
//   * round(x; sigdigits = d) = round(x * 10^k) / 10^k with k = d - hidigit(x);
//   * Wflow's pow(x, y) = exp(y * log(x))  (Wflow/src/utils.jl:470).
// exp/log/cbrt are implemented here from published methods so that host and device give
// identical results for identical inputs and no vendor math routine is involved:
//   * exp: Cody & Waite (1980) reduction x = k*ln2 + r with ln2 split in two, Taylor series of
//     exp(r) to degree 13, scaling by 2^k through the exponent bits;
//   * log: x = 2^e m, m in [sqrt(2)/2, sqrt(2)), f = m - 1, s = f/(2+f),
//     log(1+f) = f - (f^2/2 - s (f^2/2 + R)), R = sum_{i=1..10} 2 s^(2i) / (2i+1);
//   * cbrt: split off the exponent in thirds, Newton iterations on y^3 = m.
// Polynomials use explicit fma(); the translation units that include this header for the
// FP64 form are compiled with --fmad=false so nothing else is contracted.
//
// Device paths. On a GB300 every FP64-pipe instruction of a warp (DADD, DMUL, DFMA, compares,
// rint, conversions) holds its scheduler for 64 cycles, whatever the number of active lanes and
// however independent the instructions are, while an integer instruction takes about 4 (measured
// with chains of one instruction kind: 63.6 cycles per DFMA with 1 or 32 lanes and 1 or 4
// independent chains; a division 563, a square root 597, rcp.approx.ftz.f64 19). So the device
// paths below take comparisons, classifications and scalings by powers of two to the integer
// pipe, fuse a multiply and an add where the product is exact, and divide in 6 FP64 instructions.
// The results are the host paths' bit for bit.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define WF_HD __host__ __device__ __forceinline__
#else
#define WF_HD inline
#endif

#include <cmath>
#include <cstring>

namespace wfm {

WF_HD double from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double d;
    std::memcpy(&d, &b, 8);
    return d;
#endif
}
WF_HD uint64_t to_bits(double d) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t b;
    std::memcpy(&b, &d, 8);
    return b;
#endif
}
// FP64 comparisons on the integer pipe. order_key maps the values to integers of the same order
// (-0.0 just below +0.0), for everything but NaN.
WF_HD long long order_key(double x) {
    const long long b = (long long)to_bits(x);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
#ifdef __CUDACC__
// exponent field all ones: infinity or NaN
__device__ __forceinline__ bool special_(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }
#endif
WF_HD bool isnan_(double x) {
#ifdef __CUDA_ARCH__
    return (to_bits(x) & 0x7fffffffffffffffULL) > 0x7ff0000000000000ULL;
#else
    return x != x;
#endif
}
#ifdef __CUDACC__
// x in FP32, rounded towards zero, on the integer pipe (the conversion instruction is an FP64 one):
// exponent rebias and the leading 24 bits. Below 2^-126 it gives 0, from 2^128 on infinity (NaN
// too): for estimates only.
__device__ __forceinline__ float f32_of(double x) {
    const uint64_t b = to_bits(x) & 0x7fffffffffffffffULL;
    const uint32_t s = (uint32_t)__double2hiint(x) & 0x80000000u;
    uint32_t f = (uint32_t)((b - 0x3800000000000000ULL) >> 29);
    if (b < 0x3810000000000000ULL) f = 0u;
    if (b >= 0x47f0000000000000ULL) f = 0x7f800000u;
    return __uint_as_float(f | s);
}
#endif
// x < y and x == 0 as IEEE comparisons
WF_HD bool lt_(double x, double y) {
#ifdef __CUDA_ARCH__
    if (special_(x) || special_(y)) return x < y;
    return order_key(x) < order_key(y) && ((to_bits(x) | to_bits(y)) << 1) != 0;
#else
    return x < y;
#endif
}
WF_HD bool gt_(double x, double y) { return lt_(y, x); }
WF_HD bool le_(double x, double y) {  // x <= y
#ifdef __CUDA_ARCH__
    if (special_(x) || special_(y)) return x <= y;
    return order_key(x) <= order_key(y) || ((to_bits(x) | to_bits(y)) << 1) == 0;
#else
    return x <= y;
#endif
}
WF_HD bool is_zero_(double x) {
#ifdef __CUDA_ARCH__
    return (to_bits(x) << 1) == 0;
#else
    return x == 0.0;
#endif
}
WF_HD bool gt0_(double x) {  // x > 0
#ifdef __CUDA_ARCH__
    return (long long)to_bits(x) > 0 && to_bits(x) <= 0x7ff0000000000000ULL;
#else
    return x > 0.0;
#endif
}
WF_HD bool le0_(double x) {  // x <= 0
#ifdef __CUDA_ARCH__
    return ((long long)to_bits(x) <= 0 && to_bits(x) <= 0xfff0000000000000ULL);
#else
    return x <= 0.0;
#endif
}
WF_HD bool signbit_(double x) { return (to_bits(x) >> 63) != 0; }
WF_HD double fabs_(double x) { return from_bits(to_bits(x) & 0x7fffffffffffffffULL); }
WF_HD double rint_(double x) {
#ifdef __CUDA_ARCH__
    return rint(x);
#else
    return std::nearbyint(x);
#endif
}
WF_HD double fma_(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
WF_HD double fmod_(double x, double y) {
#ifdef __CUDA_ARCH__
    return fmod(x, y);
#else
    return std::fmod(x, y);
#endif
}
WF_HD double trunc_(double x) {
#ifdef __CUDA_ARCH__
    return trunc(x);
#else
    return std::trunc(x);
#endif
}
WF_HD double ceil_(double x) {
#ifdef __CUDA_ARCH__
    return ceil(x);
#else
    return std::ceil(x);
#endif
}
WF_HD double sqrt_(double x) {
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(x);
#else
    return std::sqrt(x);
#endif
}
WF_HD double copysign_(double x, double s) {
    return from_bits((to_bits(x) & 0x7fffffffffffffffULL) | (to_bits(s) & 0x8000000000000000ULL));
}

// Julia Base.min / Base.max / clamp for Float64
WF_HD double jmin(double x, double y) {
#ifdef __CUDA_ARCH__
    if (!special_(x) && !special_(y)) return order_key(x) < order_key(y) ? x : y;
#endif
    if (isnan_(x) || isnan_(y)) return x + y;
    if (x < y) return x;
    if (y < x) return y;
    return signbit_(x) ? x : y;
}
WF_HD double jmax(double x, double y) {
#ifdef __CUDA_ARCH__
    if (!special_(x) && !special_(y)) return order_key(x) > order_key(y) ? x : y;
#endif
    if (isnan_(x) || isnan_(y)) return x + y;
    if (x > y) return x;
    if (y > x) return y;
    return signbit_(x) ? y : x;
}
WF_HD double jclamp(double x, double lo, double hi) { return gt_(x, hi) ? hi : (lt_(x, lo) ? lo : x); }

// ---- division
//
// A quotient q = a r from a reciprocal r of b, corrected once by its exact remainder, is the
// correctly rounded a / b (Markstein, IBM J. Res. Dev. 34 (1990); Cornea, Harrison & Tang,
// Scientific Computing on Itanium-based Systems (2002), ch. 8) as long as nothing over- or
// underflows on the way, which quot_in_range checks on the exponents (the other cases take the
// compiler's division), and r is close enough to 1 / b. How close: with m_b the mantissa of b, a / b
// is at least 2^-53 / m_b ulps away from the middle of two values. Near a middle q is half an ulp
// from a / b, and the corrected quotient is off by half the relative error of r. A correctly rounded
// r, off by at most 2^-54 m_b, therefore always will do. rcp_raw's error is larger by the cube of its
// seed's, which is below 2^-22: at most 2^-53 (m_b / 2 + 2^-13). With that the condition holds, and q is
// next to a / b, for m_b below 2 - 2^-12; divisors closer below a power of two (below_power) take the
// compiler's division. (A seed of 2^-20, as rcp.approx.ftz.f64 gives it, does not do: of the quotients
// 2^-53 ulps from a middle 1 in 48,000 came out wrong, with m_b above 1.99.)
// With the reciprocal of a divisor that is used several times (a step size, a cell length) at hand
// the quotient costs 3 FP64 instructions, else 6 (563 cycles -> 192 / 403).
#ifdef __CUDACC__
__device__ __forceinline__ bool quot_in_range(double a, double b) {
    const int ea = (__double2hiint(a) >> 20) & 0x7ff, eb = (__double2hiint(b) >> 20) & 0x7ff;
    return ((unsigned)(ea - 160) <= 1700u || to_bits(a) == 0) && (unsigned)(eb - 160) <= 1700u &&
           ((unsigned)(ea - eb + 800) <= 1600u || to_bits(a) == 0);
}
// 1 / b to within 2^-22, b in range: the FP32 reciprocal (2^-23) of the leading 24 bits of b's mantissa,
// its exponent set on the integer pipe
__device__ __forceinline__ double rcp_seed(double b) {
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    const float m = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(m));
    const unsigned rb = __float_as_uint(r);
    return __hiloint2double((int)((rb >> 3) + 0x77f00000u - (hi & 0xfff00000u)), (int)(rb << 29));
}
// 1 / b to within 0.501 ulps, b in range: the seed's relative error e is taken to e^3
__device__ __forceinline__ double rcp_raw(double b) {
    const double r = rcp_seed(b);
    const double e = __fma_rn(-b, r, 1.0);
    return __fma_rn(__fma_rn(e, e, e), r, r);
}
__device__ __forceinline__ double quot_raw(double a, double b, double rb) {
    const double q = a * rb;
    return __fma_rn(__fma_rn(-b, q, a), rb, q);
}
// mantissa at least 2 - 2^-11
__device__ __forceinline__ bool below_power(double b) { return (__double2hiint(b) & 0xfffff) >= 0xffe00; }
// The reciprocal of b to keep for div_by_, 0 where the quotient has to take the compiler's division
__device__ __forceinline__ double rcp_kept(double b) {
    return quot_in_range(1.0, b) && !below_power(b) ? rcp_raw(b) : 0.0;
}
#endif
// a / b, correctly rounded
WF_HD double div_(double a, double b) {
#ifdef __CUDA_ARCH__
    if (quot_in_range(a, b) && !below_power(b)) return quot_raw(a, b, rcp_raw(b));
#endif
    return a / b;
}
// a / b, correctly rounded, for operands that are known to be in range (or a is +0)
WF_HD double div_mid_(double a, double b) {
#ifdef __CUDA_ARCH__
    if (!below_power(b)) return quot_raw(a, b, rcp_raw(b));
#endif
    return a / b;
}
// a / b, correctly rounded, with rb = 1 / b (correctly rounded, or rcp_kept's unless that is 0)
WF_HD double div_by_(double a, double b, double rb) {
#ifdef __CUDA_ARCH__
    if (quot_in_range(a, b)) return quot_raw(a, b, rb);
#endif
    (void)rb;
    return a / b;
}

constexpr double LN2_HI = 0x1.62e42fee00000p-1;
constexpr double LN2_LO = 0x1.a39ef35793c76p-33;
constexpr double INV_LN2 = 0x1.71547652b82fep+0;

WF_HD double exp(double x) {
#ifdef __CUDA_ARCH__
    // |x| < 700: no special case, a normal result, the scaling by 2^k an exponent addition; k has 11
    // bits and LN2_HI 33, so their product is exact and the fused subtraction rounds like the
    // separate one. 19 FP64 instructions.
    const bool plain = (__double2hiint(x) & 0x7fffffff) < 0x4085e000;
    if (!plain) {
#endif
    if (isnan_(x)) return x;
    if (x > 709.782712893384) return from_bits(0x7ff0000000000000ULL);
    if (x < -745.1332191019412) return 0.0;
#ifdef __CUDA_ARCH__
    }
    const double k = rint(x * INV_LN2);
    const double r = __fma_rn(-k, LN2_HI, x) - k * LN2_LO;
#else
    const double k = rint_(x * INV_LN2);
    const double r = (x - k * LN2_HI) - k * LN2_LO;
#endif
    double p = 0x1.6124613a86d09p-33;            // 1/13!
    p = fma_(p, r, 0x1.1eed8eff8d898p-29);       // 1/12!
    p = fma_(p, r, 0x1.ae64567f544e4p-26);       // 1/11!
    p = fma_(p, r, 0x1.27e4fb7789f5cp-22);       // 1/10!
    p = fma_(p, r, 0x1.71de3a556c734p-19);       // 1/9!
    p = fma_(p, r, 0x1.a01a01a01a01ap-16);       // 1/8!
    p = fma_(p, r, 0x1.a01a01a01a01ap-13);       // 1/7!
    p = fma_(p, r, 0x1.6c16c16c16c17p-10);       // 1/6!
    p = fma_(p, r, 0x1.1111111111111p-7);        // 1/5!
    p = fma_(p, r, 0x1.5555555555555p-5);        // 1/4!
    p = fma_(p, r, 0x1.5555555555555p-3);        // 1/3!
    p = fma_(p, r, 0.5);
    p = fma_(p, r, 1.0);
    p = fma_(p, r, 1.0);
    const int ki = (int)k;
#ifdef __CUDA_ARCH__
    if (plain) return from_bits(to_bits(p) + ((uint64_t)(int64_t)ki << 52));
#endif
    if (ki > 1023) return p * 0x1p1023 * from_bits((uint64_t)ki << 52);
    if (ki < -1022) return (p * from_bits((uint64_t)(ki + 1022 + 1023) << 52)) * 0x1p-1022;
    return p * from_bits((uint64_t)(ki + 1023) << 52);
}

WF_HD double log(double x) {
#ifdef __CUDA_ARCH__
    // A positive normal x: classification, scaling by powers of two and the choice of m on the
    // integer pipe, s by the 6-instruction division (f = 0 for x a power of two: s = 0), the exact
    // product e LN2_HI fused into the last addition. 28 FP64 instructions.
    const unsigned hx = (unsigned)__double2hiint(x);
    if (hx - 0x00100000u < 0x7fe00000u) {
        const bool up = (to_bits(x) & 0x000fffffffffffffULL) > 0x6a09e667f3bcdULL;
        const int ex = (int)(hx >> 20) - 1023 + (up ? 1 : 0);
        const double mx = from_bits((to_bits(x) & 0x000fffffffffffffULL) | (up ? 0x3fe0000000000000ULL : 0x3ff0000000000000ULL));
        const double f = mx - 1.0;
        const double b = 2.0 + f;
        const double s = div_mid_(f, b);
        const double s2 = s * s;
        double R = 0x1.8618618618618p-4;
        R = __fma_rn(R, s2, 0x1.af286bca1af28p-4);
        R = __fma_rn(R, s2, 0x1.e1e1e1e1e1e1ep-4);
        R = __fma_rn(R, s2, 0x1.1111111111111p-3);
        R = __fma_rn(R, s2, 0x1.3b13b13b13b14p-3);
        R = __fma_rn(R, s2, 0x1.745d1745d1746p-3);
        R = __fma_rn(R, s2, 0x1.c71c71c71c71cp-3);
        R = __fma_rn(R, s2, 0x1.2492492492492p-2);
        R = __fma_rn(R, s2, 0x1.999999999999ap-2);
        R = __fma_rn(R, s2, 0x1.5555555555555p-1);
        R = R * s2;
        const uint64_t ff = to_bits(f * f);  // (f f) / 2 = (f / 2) f: |f| is 0 or at least 2^-53
        const double hfsq = from_bits(ff != 0 ? ff - 0x0010000000000000ULL : 0);
        const double lm = f - (hfsq - s * (hfsq + R));
        const double de = (double)ex;
        return __fma_rn(de, LN2_HI, lm + de * LN2_LO);
    }
#endif
    if (isnan_(x) || x < 0.0) return from_bits(0x7ff8000000000000ULL);
    if (x == 0.0) return -from_bits(0x7ff0000000000000ULL);
    if (x == from_bits(0x7ff0000000000000ULL)) return x;
    int e = 0;
    uint64_t b = to_bits(x);
    if ((b >> 52) == 0) {
        x *= 0x1p54;
        b = to_bits(x);
        e = -54;
    }
    e += (int)((b >> 52) & 0x7ff) - 1023;
    double m = from_bits((b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL);
    if (m > 0x1.6a09e667f3bcdp+0) {
        m *= 0.5;
        e += 1;
    }
    const double f = m - 1.0;
    const double s = f / (2.0 + f);
    const double s2 = s * s;
    double R = 0x1.8618618618618p-4;        // 2/21
    R = fma_(R, s2, 0x1.af286bca1af28p-4);  // 2/19
    R = fma_(R, s2, 0x1.e1e1e1e1e1e1ep-4);  // 2/17
    R = fma_(R, s2, 0x1.1111111111111p-3);  // 2/15
    R = fma_(R, s2, 0x1.3b13b13b13b14p-3);  // 2/13
    R = fma_(R, s2, 0x1.745d1745d1746p-3);  // 2/11
    R = fma_(R, s2, 0x1.c71c71c71c71cp-3);  // 2/9
    R = fma_(R, s2, 0x1.2492492492492p-2);  // 2/7
    R = fma_(R, s2, 0x1.999999999999ap-2);  // 2/5
    R = fma_(R, s2, 0x1.5555555555555p-1);  // 2/3
    R = R * s2;
    const double hfsq = 0.5 * f * f;
    const double lm = f - (hfsq - s * (hfsq + R));
    const double de = (double)e;
    return de * LN2_HI + (lm + de * LN2_LO);
}

WF_HD double cbrt(double x) {
    if (isnan_(x) || x == 0.0 || fabs_(x) == from_bits(0x7ff0000000000000ULL)) return x;
    double ax = fabs_(x);
    int e = 0;
    uint64_t b = to_bits(ax);
    if ((b >> 52) == 0) {
        ax *= 0x1p54;
        b = to_bits(ax);
        e = -54;
    }
    e += (int)((b >> 52) & 0x7ff) - 1023;
    double m = from_bits((b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL);
    const int r = ((e % 3) + 3) % 3;
    const int q = (e - r) / 3;
    if (r == 1) m *= 2.0;
    if (r == 2) m *= 4.0;
    double y = 0.6 + 0.2 * m;
    // m in [1, 8), y in (0.5, 3): the residual is +0 or at least 2^-54
    for (int i = 0; i < 6; ++i) y = y - div_mid_(y * y * y - m, 3.0 * y * y);
    y = y * from_bits((uint64_t)(q + 1023) << 52);
    return x < 0.0 ? -y : y;
}

// Wflow.pow (utils.jl:470)
WF_HD double pow(double x, double y) { return exp(y * log(x)); }

// Base.div(x, y, RoundUp) (cld) for y > 0
WF_HD double cld(double x, double y) {
#ifdef __CUDA_ARCH__
    // The smallest integer n with n y >= x: the rounded quotient's ceiling, moved by the sign of the
    // remainders, which a fused multiply-add gives exactly.
    if (gt0_(x) && quot_in_range(x, y)) {
        const double q = quot_raw(x, y, rcp_raw(y));
        if ((__double2hiint(q) & 0x7fffffff) < 0x41300000) {  // q < 2^20
            const double n = ::ceil(q);
            if (gt0_(__fma_rn(-n, y, x))) return n + 1.0;
            if (le0_(__fma_rn(-(n - 1.0), y, x))) return n - 1.0;
            return n;
        }
    }
#endif
    const double r = fmod_(x, -y);
    double m;
    if (r == 0.0) {
        m = copysign_(0.0, -y);
    } else if ((r > 0.0) != (-y > 0.0)) {
        m = r + (-y);
    } else {
        m = r;
    }
    return rint_((x - m) / y);
}

// round(x; sigdigits = d) for finite x >= 0 (the path only rounds |dz| / 0.1)
WF_HD double round_sigdigits(double x, int sigdigits) {
    if (x == 0.0 || isnan_(x) || fabs_(x) == from_bits(0x7ff0000000000000ULL)) return x;
    const double ax = fabs_(x);
    int k = 0;
    double p = 1.0;
    if (ax >= 1.0) {
        while (ax >= p * 10.0 && k < 308) {
            p *= 10.0;
            ++k;
        }
    } else {
        while (ax < p && k > -330) {
            p /= 10.0;
            --k;
        }
    }
    const int d = sigdigits - (1 + k);
    if (d >= 0) {
        double sc = 1.0;
        for (int i = 0; i < d; ++i) sc *= 10.0;
        const double y = rint_(x * sc) / sc;
        return (y - y == 0.0) ? y : x;
    }
    double isc = 1.0;
    for (int i = 0; i < -d; ++i) isc *= 10.0;
    return rint_(x / isc) * isc;
}

}  // namespace wfm
