// div_by.cuh -- correctly rounded FP64 division by a divisor known in advance
// (a parameter, or one value that several quotients of a site share).
//
// GB300's FP64 pipe issues one warp instruction in 16 cycles, and a general
// IEEE division costs it about nine instructions; the plain form takes 45 to
// 60 per site. With zh = RN(1/y) and zl ~ 1/y - zh known, the quotient takes
// one to four, and the same bits:
//   DIV_ONE      y = 1: x.
//   DIV_EXACT    y = 2^k: x zh, one rounding of the exact quotient, as x / y.
//   DIV_SHORT    y = Y 2^k, Y odd below 2^20: q = RN(x zh + RN(x zl)). Before
//                its last rounding q is within 2^-51 ulp of x/y, and x/y is no
//                nearer than 1/(2Y) > 2^-21 ulp to a rounding boundary (the
//                numerator of the distance is a non-zero integer).
//   DIV_MARKSTEIN  q = RN(x zh), r = x - q y (exact), RN(q + r zh).
//   DIV_CORRECT    the same from q = RN(x zh + RN(x zl)).
// The last two are Markstein's theorem (IBM J. Res. Dev. 34, 1990; Brisebarre,
// Muller and Raina, IEEE Trans. Comput. 53, 2004): if zh is the correctly
// rounded reciprocal and q is within one ulp of x/y, then RN(q + r zh) is the
// correctly rounded quotient. q = RN(x zh) is within one ulp when x's
// significand is not below y's (for any y), and otherwise when
// |1 - y zh| <= 2^-54 (error x |1/y - zh| below half an ulp, and half an ulp of
// rounding); DIV_CORRECT's q always is. Divisors outside [2^-100, 2^100], and
// those whose significand is all ones, take DIV_GENERAL, the IEEE division; so
// does any x that is neither 0 nor in [2^-823, 2^777], where a product or a
// remainder could leave the normal range (and infinities and NaN).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define DL_HD __host__ __device__ __forceinline__
#else
#define DL_HD inline
#endif

namespace dl {

enum { DIV_GENERAL = 0, DIV_ONE, DIV_EXACT, DIV_SHORT, DIV_MARKSTEIN, DIV_CORRECT };

struct DivBy {
    double y, zh, zl;
    int how;
};

DL_HD double div_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#else
    return fma(a, b, c);
#endif
}

DL_HD uint64_t div_bits(double v) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t b;
    memcpy(&b, &v, 8);
    return b;
#endif
}

// the divisor may take DIV_CORRECT: positive, in [2^-100, 2^100], significand not all ones
DL_HD bool div_divisor_ok(double y) {
    const uint64_t b = div_bits(y);
    const unsigned e = (unsigned)(b >> 52);
    return e >= 1023u - 100u && e <= 1023u + 100u && (b << 12) != 0xFFFFFFFFFFFFF000ull;
}

// numerators the short ways hold for: 0, or |x| in [2^-823, 2^777)
DL_HD bool div_numerator_ok(double x) {
    const uint64_t b = div_bits(x) << 1;
    return b == 0 || ((unsigned)(b >> 53) - 200u) < 1600u;
}

// kept out of line: the general division's code would be repeated at every quotient
#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double div_general(double x, double y) { return x / y; }
#else
inline double div_general(double x, double y) { return x / y; }
#endif

// q with the sign of x, which every quotient by a positive divisor has: of x = -0 the
// additions make +0 (zl < 0, or a remainder of +0)
DL_HD double div_signed(double q, double x) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double(__double2hiint(q) | (__double2hiint(x) & (int)0x80000000u), __double2loint(q));
#else
    return copysign(q, x);
#endif
}

DL_HD double div_short(double x, double zh, double zl) { return div_signed(div_fma(x, zh, x * zl), x); }

DL_HD double div_correct(double x, double y, double zh, double zl) {
    const double q = div_fma(x, zh, x * zl);
    return div_signed(div_fma(div_fma(-q, y, x), zh, q), x);
}

DL_HD double div_markstein(double x, double y, double zh) {
    const double q = x * zh;
    return div_signed(div_fma(div_fma(-q, y, x), zh, q), x);
}

DL_HD double div_by(double x, const DivBy& d) {
    if (d.how == DIV_ONE) return x;
    if (d.how == DIV_GENERAL || !div_numerator_ok(x)) return div_general(x, d.y);
    if (d.how == DIV_CORRECT) return div_correct(x, d.y, d.zh, d.zl);
    if (d.how == DIV_SHORT) return div_short(x, d.zh, d.zl);
    if (d.how == DIV_EXACT) return x * d.zh;
    return div_markstein(x, d.y, d.zh);
}

// x / 3: DIV_SHORT with 1/3 and the rest of it, 1/3 - RN(1/3) = 2^-54 / 3
DL_HD double div3(double x) {
    if (!div_numerator_ok(x)) return div_general(x, 3.0);
    return div_short(x, 1.0 / 3.0, 0x1.5555555555555p-56);
}

// the way for divisor y (host)
inline DivBy make_div_by(double y) {
    DivBy d = {y, 0.0, 0.0, DIV_GENERAL};
    if (y == 1.0) {
        d.how = DIV_ONE;
        return d;
    }
    if (!div_divisor_ok(y)) return d;
    d.zh = 1.0 / y;
    const double e = fma(-y, d.zh, 1.0);  // exact
    d.zl = e / y;
    int k;
    const double m = frexp(y, &k);  // [1/2, 1)
    const double short_y = ldexp(m, 20);
    if (m == 0.5) d.how = DIV_EXACT;
    else if (short_y == floor(short_y)) d.how = DIV_SHORT;
    else d.how = fabs(e) <= 0x1p-54 ? DIV_MARKSTEIN : DIV_CORRECT;
    return d;
}

}  // namespace dl
