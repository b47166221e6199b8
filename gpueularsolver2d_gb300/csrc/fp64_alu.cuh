// fp64_alu.cuh -- FP64 division, square root and ordering on the integer
// units, with the results of the IEEE operations bit for bit.
//
// GB300 issues one FP64 warp instruction per SM every 16 cycles, in which the
// four schedulers can issue 64 others; an FP64 division or square root is
// seven to nine dependent FP64 instructions, an FP64 comparison one.  Here a
// division is about 55 integer instructions and a square root about 65, so the
// FP64 pipe is left to the additions and multiplications of the scheme.
// On a 1.05M-cell mesh, with the FP64 operations left out that these and exact
// powers of two make unnecessary (spectral_radius, roe_scaled, faces_cell64),
// pass A went from 1163 to 457 us per launch, pass B from 990 to 615 us, the FP64
// pipe still 77-81 % busy.
//
// Division: the classical digit recurrence in a high radix with quotient
// digits selected by multiplication with a short reciprocal of the divisor
// (Ercegovac and Lang, "Digital Arithmetic", 2004, ch. 5; Wong and Flynn, IEEE
// Trans. Computers 41, 1992): digits of 30, 19 and 4 bits from a 20-bit
// underestimate of the reciprocal, each followed by the exact remainder in
// 64-bit integers.  Every digit is an underestimate, so remainders stay
// non-negative; the last one is corrected by one.  The quotient's 54 leading
// bits round to nearest by their last bit, since a quotient of two 53-bit
// numbers is never half way between two others.  The square root is the same
// recurrence (30, 18 and 5 bits) with an underestimate of 1 / (2 sqrt(x)).
//
// Operands or results outside the normal range (zeros apart) set a flag, and the
// caller does the operation, or a whole formula of them (FastOps, IeeeOps), again
// in hardware: one branch for a formula instead of one per operation, which
// kept their chains from interleaving (8k cells: an iteration 164 -> 141 us).
// What tests a value without its sign is written with shifts and exponents: a
// masked sign or a test of the other bits for zero is compiled into an FP64
// instruction, a slot each (1.05M cells: pass A 294 -> 256 us, pass C 53 -> 45,
// pass D 103 -> 70).  Compiles for the host too (the seed is then the host's FP32
// division), where tests hold it against the host's own IEEE operations.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define E2D_HD __host__ __device__ __forceinline__
#define E2D_HD_SLOW static __host__ __device__ __noinline__
#else
#define E2D_HD inline
#define E2D_HD_SLOW inline
#endif

namespace e2d {

E2D_HD uint64_t bits_of(double v) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    memcpy(&u, &v, 8);
    return u;
#endif
}

E2D_HD double double_of(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, 8);
    return v;
#endif
}

E2D_HD uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

#ifndef __CUDA_ARCH__
#ifndef E2D_SEED_ULPS
#define E2D_SEED_ULPS 0  // host tests: the seed moved by this many units in the last place
#endif
E2D_HD float moved_seed(float v) {
    uint32_t u;
    memcpy(&u, &v, 4);
    u += E2D_SEED_ULPS;
    memcpy(&v, &u, 4);
    return v;
}
#endif

// FP32 seeds, good to one unit in the last place (rcp) and 2^-22 (rsqrt)
E2D_HD float seed_rcp(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return moved_seed(1.0f / x);
#endif
}
E2D_HD float seed_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return moved_seed((float)(1.0 / sqrt((double)x)));
#endif
}
E2D_HD float float_of(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float v;
    memcpy(&v, &u, 4);
    return v;
#endif
}

E2D_HD_SLOW double div_ieee(double a, double b) { return a / b; }
E2D_HD_SLOW double sqrt_ieee(double a) { return sqrt(a); }

// A divisor prepared for div_by: several numerators share the work.
struct Divisor {
    double b;
    uint64_t m;  // significand, bit 52 set
    uint32_t y;  // 2^32 / (m / 2^52), an underestimate good to 2^-20
    int e;       // biased exponent; 0 or 2047 (zero, subnormal, infinity, NaN): not prepared
};

E2D_HD Divisor divisor(double b) {
    Divisor d;
    const uint64_t u = bits_of(b);
    d.b = b;
    d.e = (int)(u >> 52) & 0x7ff;
    d.m = (u & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL;
    // top 24 bits as a float f in [1, 2): f <= m < f + 2^-23.  The factor
    // 1 - 2^-21 covers the seed's unit and makes y an underestimate.
    const float f = float_of(0x3f800000u | ((uint32_t)(u >> 29) & 0x7fffffu));
    d.y = (uint32_t)(seed_rcp(f) * 4294965248.0f);
    return d;
}

// Whether a value with exponent bits 0 is not zero.  (A test of all bits but the
// sign for zero is compiled into an FP64 comparison.)
E2D_HD bool subnormal(uint64_t u) { return (u & 0xFFFFFFFFFFFFFULL) != 0; }

// a / d.b, rounded to nearest even; bad is set, and the result void, where an
// operand or the result is outside the range.  Without branches: chains of these
// interleave, and one test after many of them decides whether they stand.
E2D_HD double div_fast(double a, const Divisor &d, bool &bad) {
    const uint64_t ua = bits_of(a);
    const int ea = (int)(ua >> 52) & 0x7ff;
    int e = ea - d.e + 1023;
    const bool zero = ea == 0;
    bad |= (zero ? subnormal(ua) : ea == 2047 || (unsigned)(e - 2) >= 2043u) | ((unsigned)(d.e - 1) >= 2046u);
    uint64_t r = (ua & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL;
    const int low = r < d.m;  // quotient of the significands in [1, 2)
    r = low ? r << 1 : r;
    e -= low;
    const uint32_t q1 = mul_hi((uint32_t)(r >> 22), d.y);  // 30 bits of fraction
    r = (r << 30) - (uint64_t)q1 * d.m;                    // < 2^11 m
    const uint32_t q2 = mul_hi((uint32_t)(r >> 32), d.y) >> 1;  // the next 19
    r = (r << 19) - (uint64_t)q2 * d.m;                         // < 2^10 m
    uint32_t q3 = mul_hi((uint32_t)(r >> 32), d.y) >> 16;  // the last 4
    r = (r << 4) - (uint64_t)q3 * d.m;
    q3 += r >= d.m;
    const uint64_t q = ((uint64_t)q1 << 23) + ((uint64_t)q2 << 4) + q3;  // 54 bits
    const uint64_t sign = (ua ^ bits_of(d.b)) & 0x8000000000000000ULL;
    const uint64_t mag = ((uint64_t)(uint32_t)(e - 1) << 52) + ((q + 1) >> 1);
    return double_of(sign | (zero ? 0 : mag));
}

E2D_HD double div_by(double a, const Divisor &d) {
    bool bad = false;
    const double q = div_fast(a, d, bad);
    return bad ? div_ieee(a, d.b) : q;
}

E2D_HD double ddiv(double a, double b) { return div_by(a, divisor(b)); }

// sqrt(x), rounded to nearest even; bad as in div_fast.
E2D_HD double sqrt_fast(double x, bool &bad) {
    const uint64_t u = bits_of(x);
    bad |= (uint32_t)(u >> 32) - 0x00100000u >= 0x7ff00000u - 0x00100000u;
    const int ex = (int)(u >> 52) - 1023;
    const uint32_t odd = (uint32_t)ex & 1u;
    const uint64_t m = ((u & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL) << odd;  // in [1, 4) 2^52
    const float f = float_of((0x3f800000u | ((uint32_t)(u >> 29) & 0x7fffffu)) + (odd << 23));
    const float y = seed_rsqrt(f);
    const uint32_t z = (uint32_t)(y * 2147481600.0f);        // 2^32 / (2 s), underestimated by 2^-20
    const uint32_t s1 = (uint32_t)((f * y) * 1073740800.0f);  // s 2^30, underestimated by 2^-20
    uint64_t r = (m << 8) - (uint64_t)s1 * s1;                // < 2^44
    const uint32_t s2 = mul_hi((uint32_t)(r >> 12), z);       // the next 18 bits
    r = (r << 36) - (((uint64_t)s1 * s2) << 19) - (uint64_t)s2 * s2;  // < 2^62
    const uint64_t sa = ((uint64_t)s1 << 18) + s2;
    const uint32_t s3 = mul_hi((uint32_t)(r >> 32), z) >> 11;  // the last 5
    r = (r << 10) - (sa << 6) * s3 - (uint64_t)s3 * s3;
    uint64_t s = (sa << 5) + s3;
    s += r > 2 * s;
    return double_of(((uint64_t)(uint32_t)(((ex - (int)odd) >> 1) + 1022) << 52) + ((s + 1) >> 1));
}

E2D_HD double dsqrt(double x) {
    bool bad = false;
    const double s = sqrt_fast(x, bad);
    return bad ? sqrt_ieee(x) : s;
}

// a * b, rounded to nearest even: the 106-bit product of the significands in
// 32-bit pieces, about 40 integer instructions.  For kernels that have integer
// issue slots left beside a busy FP64 pipe.  bad as in div_fast.
E2D_HD double mul_fast(double a, double b, bool &bad) {
    const uint64_t ua = bits_of(a), ub = bits_of(b);
    const int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff;
    const int e = ea + eb - 1023;
    const bool za = ea == 0, zb = eb == 0, zero = za | zb;
    bad |= (za & subnormal(ua)) | (zb & subnormal(ub)) | (ea == 2047) | (eb == 2047) |
           (!zero & ((unsigned)(e - 2) >= 2043u));
    const uint64_t x = (ua << 11) | 0x8000000000000000ULL, y = (ub << 11) | 0x8000000000000000ULL;
#ifdef __CUDA_ARCH__
    uint64_t hi = __umul64hi(x, y), lo = x * y;
#else
    const unsigned __int128 xy = (unsigned __int128)x * y;
    uint64_t hi = (uint64_t)(xy >> 64), lo = (uint64_t)xy;
#endif
    const int up = (int)(hi >> 63);  // product of the significands in [2, 4)
    hi = up ? hi : (hi << 1) | (lo >> 63);
    lo = up ? lo : lo << 1;
    hi |= lo != 0;                                        // sticky
    uint64_t m = hi >> 11;                                // 53 bits
    m += ((uint32_t)hi & 0x7ffu) + ((uint32_t)m & 1u) > 0x400u;  // to 2^53 at most
    const uint64_t sign = (ua ^ ub) & 0x8000000000000000ULL;
    return double_of(sign | (zero ? 0 : ((uint64_t)(uint32_t)(e - 1 + up) << 52) + m));
}
// (A product by itself: the form that the host's test holds against its own.)
E2D_HD_SLOW double mul_ieee(double a, double b) { return a * b; }
E2D_HD double imul(double a, double b) {
    bool bad = false;
    const double p = mul_fast(a, b, bad);
    return bad ? mul_ieee(a, b) : p;
}

// The operations of a kernel's FP64 formulas: on the integer units (mul: where INT
// says so), to be done again with the IEEE operations when bad is set.
struct FastOps {
    bool bad = false;
    typedef Divisor Div;
    E2D_HD Div over(double b) { return divisor(b); }
    E2D_HD double by(double a, const Div &d) { return div_fast(a, d, bad); }
    E2D_HD double div(double a, double b) { return div_fast(a, divisor(b), bad); }
    E2D_HD double sqrt(double x) { return sqrt_fast(x, bad); }
    template <bool INT> E2D_HD double mul(double a, double b) { return INT ? mul_fast(a, b, bad) : a * b; }
    E2D_HD double half(double x) {  // exact: one less in the exponent
        const uint64_t u = bits_of(x);
        const uint32_t e = (uint32_t)(u >> 52) & 0x7ff;
        bad |= (e == 0 ? subnormal(u) : e == 1 || e == 2047);
        return double_of(u - (e ? 1ULL << 52 : 0));
    }
};
struct IeeeOps {
    bool bad = false;
    typedef double Div;
    E2D_HD Div over(double b) { return b; }
    E2D_HD double by(double a, const Div &d) { return a / d; }
    E2D_HD double div(double a, double b) { return a / b; }
    E2D_HD double sqrt(double x) { return ::sqrt(x); }
    template <bool INT> E2D_HD double mul(double a, double b) { return a * b; }
    E2D_HD double half(double x) { return 0.5 * x; }
};

// Monotonic integer key of a double: keys of numbers order like the numbers
// (-0 just below +0); the inverse is the same map.
E2D_HD int64_t order_key(double v) {
    const int64_t k = (int64_t)bits_of(v);
    return k ^ (int64_t)((uint64_t)(k >> 63) >> 1);
}
E2D_HD double key_value(int64_t k) { return double_of((uint64_t)(k ^ (int64_t)((uint64_t)(k >> 63) >> 1))); }

// |x| < |y| on the bit patterns (finite values order like their magnitudes'
// bits; a NaN compares above every finite value).  Shifted, not masked: a masked
// sign is compiled into an FP64 instruction.
E2D_HD bool abs_less(double x, double y) { return bits_of(x) << 1 < bits_of(y) << 1; }

}  // namespace e2d
