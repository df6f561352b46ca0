// Correctly rounded acos, cos, sin and pow for the FP64 collision path.
//
// The reference's CCD root finder (isCoplanar, dcollid3d.cpp:425-450) and
// its impact-zone rotation (dcollid3d.cpp:163-169) call acos, cos, pow and
// sin, and near double roots those roots are very sensitive: a one-ulp change
// in one of these results can move a step's output by 1e-8 relative. The
// reference's results come from glibc, which rounds these functions correctly
// in all but roughly 0.1% of arguments; CUDA's versions allow 2 ulp. These
// functions return the correctly rounded result (barring arguments within
// about 1e-30 relative of a rounding midpoint), so they agree with the
// reference wherever glibc is correctly rounded.
//
// Method, from the mathematics: double-double arithmetic built on the exact
// error of a sum (two_sum) and of a product (fma); sin / cos by reduction
// modulo pi/2 with a three-part pi/2 (Cody and Waite) and their Taylor series
// to x^29 on [-pi/4, pi/4]; acos and asin by one Newton step on cos / sin from
// a starting value within a few ulp, using the half-angle identity
// acos(x) = 2 asin(sqrt((1-x)/2)) away from 0; pow(a, y) by one correction
// step r = r0 (1 + y ln a - ln r0) with ln in double-double from the atanh
// series. Series coefficients are 1/n!, 1/(2k+1), pi and ln 2 to ~300 bits,
// rounded to double-double.
//
// An FP64 instruction takes a GB300 warp ~64 cycles and a double-double Horner
// step ~30 of them, so each function first tries fixed point: the same Taylor
// series in 64- and 128-bit integers (namespace fx), to ~2^-78 with a bound.
// Its result counts only where everything within the bound rounds to the same
// double, which is then the correctly rounded one; about one argument in 2^24
// goes on to the double-double form (24,400 cycles for the sine and cosine of
// a zone's rotation). A step of 257 x 257 points in contact: its sub-tests
// 2.46 -> 1.53 ms; 24 sheets in FP64: 1.95 -> 1.06 ms; 256 sheets: zone solves
// 12.2 -> 10.0 ms.
//
// Every routine is __host__ __device__ so the same code can be checked on the
// host; products use fma() explicitly and nothing relies on contraction.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define CR_HD __host__ __device__ __forceinline__
#else
#define CR_HD inline
#endif

namespace ccg {
namespace cr {

struct dd {
    double hi, lo;
};

CR_HD dd two_sum(double a, double b) {
    double s = a + b;
    double t = s - a;
    double e = (a - (s - t)) + (b - t);
    return dd{s, e};
}
CR_HD dd fast_two_sum(double a, double b) {
    double s = a + b;
    double e = b - (s - a);
    return dd{s, e};
}
CR_HD dd two_prod(double a, double b) {
    double p = a * b;
    double e = fma(a, b, -p);
    return dd{p, e};
}
CR_HD dd neg(dd x) { return dd{-x.hi, -x.lo}; }
CR_HD dd add(dd x, dd y) {
    dd s = two_sum(x.hi, y.hi);
    dd t = two_sum(x.lo, y.lo);
    s.lo += t.hi;
    s = fast_two_sum(s.hi, s.lo);
    s.lo += t.lo;
    return fast_two_sum(s.hi, s.lo);
}
CR_HD dd add_d(dd x, double y) {
    dd s = two_sum(x.hi, y);
    s.lo += x.lo;
    return fast_two_sum(s.hi, s.lo);
}
CR_HD dd mul(dd x, dd y) {
    dd p = two_prod(x.hi, y.hi);
    p.lo += x.hi * y.lo;
    p.lo += x.lo * y.hi;
    return fast_two_sum(p.hi, p.lo);
}
CR_HD dd mul_d(dd x, double y) {
    dd p = two_prod(x.hi, y);
    p.lo += x.lo * y;
    return fast_two_sum(p.hi, p.lo);
}
CR_HD dd div(dd x, dd y) {
    double q1 = x.hi / y.hi;
    dd r = add(x, neg(mul_d(y, q1)));
    double q2 = r.hi / y.hi;
    r = add(r, neg(mul_d(y, q2)));
    double q3 = r.hi / y.hi;
    return add_d(fast_two_sum(q1, q2), q3);
}

constexpr double kPiHi = 0x1.921fb54442d18p+1, kPiLo = 0x1.1a62633145c07p-53;

// ------------------------------------------------------------ fixed point
namespace fx {

typedef unsigned __int128 u128;
typedef __int128 i128;

CR_HD uint64_t mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((u128)a * b) >> 64);
#endif
}
CR_HD u128 make(uint64_t hi, uint64_t lo) { return ((u128)hi << 64) | lo; }
CR_HD int clz64(uint64_t v) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}
CR_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
CR_HD double of_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
// the upper half of a product of fractions (one unit below the exact floor at most)
CR_HD u128 mulhi128(u128 a, u128 b) {
    const uint64_t ah = (uint64_t)(a >> 64), al = (uint64_t)a, bh = (uint64_t)(b >> 64), bl = (uint64_t)b;
    const u128 m1 = (u128)ah * bl, m2 = (u128)al * bh;
    const u128 mid = (u128)(uint64_t)m1 + (uint64_t)m2 + mulhi64(al, bl);
    return (u128)ah * bh + (uint64_t)(m1 >> 64) + (uint64_t)(m2 >> 64) + (uint64_t)(mid >> 64);
}

// |x| - k pi/2 for 0 < |x| < 8 as (R / 2^128) 2^ex, R normalised, negative
// if neg; k mod 4 in q. False: outside the range, or too close to a multiple
// of pi/2 (or to 0) for the bound.
CR_HD bool reduce(double x, u128* R, int* ex, int* q, bool* neg) {
    const uint64_t b = bits_of(x);
    const int E = (int)((b >> 52) & 0x7ff);
    if (E < 1023 - 60 || E > 1023 + 2) return false;
    const uint64_t m = (b & (((uint64_t)1 << 52) - 1)) | ((uint64_t)1 << 52);
    *q = 0;
    *neg = false;
    const int k = (int)(fabsf((float)x) * 0.63661977f + 0.5f);  // 0 .. 5: |r| exceeds pi/4 by 1e-6 at most
    if (k == 0) {
        *R = (u128)m << 75;
        *ex = E - 1022;
        return true;
    }
    uint64_t kh, kl;  // k pi/2 in units of 2^-125
    switch (k) {
        case 1: kh = 0x3243f6a8885a308dull, kl = 0x313198a2e0370734ull; break;
        case 2: kh = 0x6487ed5110b4611aull, kl = 0x62633145c06e0e69ull; break;
        case 3: kh = 0x96cbe3f9990e91a7ull, kl = 0x9394c9e8a0a5159dull; break;
        case 4: kh = 0xc90fdaa22168c234ull, kl = 0xc4c6628b80dc1cd1ull; break;
        case 5: kh = 0xfb53d14aa9c2f2c1ull, kl = 0xf5f7fb2e61132405ull; break;
        default: return false;
    }
    const u128 X = (u128)m << (73 + E - 1023), K = make(kh, kl);
    *neg = X < K;
    u128 d = *neg ? K - X : X - K;
    d <<= 3;  // below 0.79 * 2^125 before
    if ((uint64_t)(d >> 64) < ((uint64_t)1 << 34)) return false;  // |r| < 2^-30
    const int lz = clz64((uint64_t)(d >> 64));
    *R = d << lz;
    *ex = -lz;
    *q = k & 3;
    return true;
}

// sin r or cos r of r = (R / 2^128) 2^ex, |r| < 0.786, as (M / 2^128) 2^*em,
// M >= 2^126, within 2^48 units of M (from the tail's 64 bits: 2^-62 times
// r^8 / 8! is 2^-80). The first terms are nested in 128 bits, the tail after
// them, 1 - w (1 - w' (1 - ...)) with w = r^2 / ((j-1) j), in 64.
CR_HD u128 sc(u128 R, int ex, bool cosine, int* em) {
#define FX_SEL(s, c) (cosine ? (c) : (s))
    u128 r2 = mulhi128(R, R);
    r2 = ex > -64 ? r2 >> (-2 * ex) : (u128)0;
    const uint64_t h = (uint64_t)(r2 >> 64);
    uint64_t g = ~mulhi64(h, FX_SEL(0x006d3a06d3a06d3aull, 0x0076b981dae6076cull));
    g = ~mulhi64(mulhi64(h, FX_SEL(0x0081848da8faf0d2ull, 0x008dda5202376948ull)), g);
    g = ~mulhi64(mulhi64(h, FX_SEL(0x009c09c09c09c09cull, 0x00ac7691840ac769ull)), g);
    g = ~mulhi64(mulhi64(h, FX_SEL(0x00bfa02fe80bfa03ull, 0x00d62b80d62b80d6ull)), g);
    g = ~mulhi64(mulhi64(h, FX_SEL(0x00f0f0f0f0f0f0f1ull, 0x0111111111111111ull)), g);
    g = ~mulhi64(mulhi64(h, FX_SEL(0x0138138138138138ull, 0x0168168168168168ull)), g);
    g = ~mulhi64(mulhi64(h, FX_SEL(0x01a41a41a41a41a4ull, 0x01f07c1f07c1f07cull)), g);
    g = ~mulhi64(mulhi64(h, FX_SEL(0x0253c8253c8253c8ull, 0x02d82d82d82d82d8ull)), g);
    u128 t = (u128)FX_SEL(0x00002e3bc74aad8eull, 0x0001a01a01a01a01ull) * g +
             mulhi64(FX_SEL(0x671f5583911ca003ull, 0xa01a01a01a01a01aull), g);
    t = FX_SEL(make(0x000d00d00d00d00dull, 0x00d00d00d00d00d0ull), make(0x005b05b05b05b05bull, 0x05b05b05b05b05b0ull)) -
        mulhi128(r2, t);
    t = FX_SEL(make(0x0222222222222222ull, 0x2222222222222222ull), make(0x0aaaaaaaaaaaaaaaull, 0xaaaaaaaaaaaaaaabull)) -
        mulhi128(r2, t);
    t = FX_SEL(make(0x2aaaaaaaaaaaaaaaull, 0xaaaaaaaaaaaaaaabull), make(0x8000000000000000ull, 0)) - mulhi128(r2, t);
    const u128 U = mulhi128(r2, t);
#undef FX_SEL
    *em = cosine ? 0 : ex;
    return cosine ? ~U : R - mulhi128(R, U);
}

constexpr uint64_t kErr = (uint64_t)1 << 50;  // units of M

// (v / 2^128) 2^em rounded to 53 bits, as the bits of a positive double.
CR_HD uint64_t round53(u128 v, int em) {
    const int lz = clz64((uint64_t)(v >> 64));
    const uint64_t top = (uint64_t)((v << lz) >> 64);
    const uint64_t mant = (top >> 11) + ((top >> 10) & 1);
    return ((uint64_t)(em - lz + 1022) << 52) + (mant - ((uint64_t)1 << 52));
}

// The double that M - kErr .. M + kErr round to; false if they do not agree.
CR_HD bool settle(u128 M, int em, double* out) {
    const u128 hi = M + kErr;
    if (hi < M) return false;
    const uint64_t b = round53(hi, em);
    *out = of_bits(b);
    return b == round53(M - kErr, em);
}

// cos x (want_cos) or sin x.
CR_HD bool sin_or_cos(double x, bool want_cos, double* out) {
    u128 R;
    int ex, q, em;
    bool neg;
    if (!reduce(x, &R, &ex, &q, &neg)) return false;
    const bool odd = (q & 1) != 0;
    const u128 M = sc(R, ex, odd != want_cos, &em);
    if (!settle(M, em, out)) return false;
    // signs: cos |x| is cos r, -sin r, -cos r, sin r; sin |x| is sin r, cos r, -sin r, -cos r
    bool minus = want_cos ? (q == 1 || q == 2) : q >= 2;
    if (neg && odd == want_cos) minus = !minus;      // r's sine
    if (!want_cos && (bits_of(x) >> 63)) minus = !minus;
    if (minus) *out = -*out;
    return true;
}

// acos x from y0, an estimate within a few ulp of acos x for |x| <= 1/2 and
// of acos |x| above: one Newton step, its residual exact in fixed point, its
// slope in FP32 (the step is 2^-50 of y0 or less). Up to 1/2 the residual is
// cos y0 - x; above, sin^2(y0 / 2) - (1 - |x|) / 2, whose relative precision
// does not fall as x nears 1. Near 0, where y0 is too close to pi / 2, the
// series pi / 2 - x - x^3 / 6 ends at 2^-130.
CR_HD bool acos_from(double x, double y0, double* out) {
    if (fabs(x) < 0x1p-26) {
        const dd t = two_sum(0.5 * kPiHi, -x);
        const double step = t.lo + (0.5 * kPiLo - x * x * x * (1.0 / 6.0));
        const double up = t.hi + (step + 0x1p-100);
        *out = up;
        return up == t.hi + (step - 0x1p-100);
    }
    const bool far = fabs(x) > 0.5;
    const double ax = fabs(x), other = far ? (1.0 - ax) * 0.5 : ax;  // exact: 1 - ax for ax in (0.5, 1]
    const uint64_t b = bits_of(other);
    const int E = (int)((b >> 52) & 0x7ff);
    if (E < 1023 - 60 || E >= 1023) return false;
    u128 R;
    int ex, q, em;
    bool neg;
    if (!reduce(far ? y0 * 0.5 : y0, &R, &ex, &q, &neg)) return false;
    const bool odd = (q & 1) != 0;
    u128 M = sc(R, ex, far ? odd : !odd, &em);
    u128 X = (u128)((b & (((uint64_t)1 << 52) - 1)) | ((uint64_t)1 << 52)) << 75;
    int eX = E - 1022;
    if (far) {  // (0, pi / 6]: q is 0
        if (q != 0 || neg) return false;
        M = mulhi128(M, M);
        em *= 2;
    }
    // both below one half at a common exponent, where 48 bits of them agree
    const int e = far ? (em > eX ? em : eX) + 1 : 1;
    if (e - em > 40 || e - eX > 64) return false;
    M >>= e - em;
    X >>= e - eX;
    bool minus = false;
    if (!far) {
        minus = q == 1 || q == 2;
        if (neg && odd) minus = !minus;
    }
    const i128 d = (minus ? -(i128)M : (i128)M) - (!far && (bits_of(x) >> 63) ? -(i128)X : (i128)X);
    const i128 top = d >> 16;
    if (top > ((i128)1 << 62) || top < -((i128)1 << 62)) return false;
    const double inv = (double)(1.0f / sqrtf((float)(1.0 - ax) * (float)(1.0 + ax)));
    double step = (double)(int64_t)top * of_bits((uint64_t)(e - 112 + 1023) << 52) * inv;
    double err = far ? y0 * 0x1p-74 : 0x1p-75;
    if (far) step *= -2.0;
    err += fabs(step) * 0x1p-20;
    double base = y0;
    if (far && x < 0.0) {  // pi - acos |x|
        const dd t = two_sum(kPiHi, -y0);
        base = t.hi;
        step = t.lo + (kPiLo - step);
        err += 0x1p-100;
    }
    const double up = base + (step + err);
    *out = up;
    return up == base + (step - err);
}

// a^y for y = 1.0 / 3.0 = 1/3 - 2^-54 / 3 from r0, an estimate of the cube
// root within a few ulp: a - r0^3 is exact in integers, and a^(y - 1/3) =
// exp(-ln a 2^-54 / 3) needs ln a to FP32.
CR_HD bool cube_root_from(double a, double r0, double* out) {
    const uint64_t ab = bits_of(a), rb = bits_of(r0);
    const int ea = (int)((ab >> 52) & 0x7ff) - 1075, er = (int)((rb >> 52) & 0x7ff) - 1075;
    const uint64_t one = (uint64_t)1 << 52;
    const uint64_t A = (ab & (one - 1)) | one, r = (rb & (one - 1)) | one;
    const int s = ea - 3 * er;
    if (ea <= -1075 || ea > 900 || er <= -1075 || s < 64 || s > 127) return false;
    // A 2^s - r^3, both below 2^160 and equal in their leading ~50 bits: their
    // difference modulo 2^128 is the difference
    const i128 d = (i128)(((u128)A << s) - (u128)r * r * r);
    const i128 top = d >> 50;
    if (top > ((i128)1 << 62) || top < -((i128)1 << 62)) return false;
    const double rd = (double)r;
    const double rel = (double)(int64_t)top * 0x1p50 / (3.0 * (rd * rd * rd));
    if (!(fabs(rel) < 0x1p-48)) return false;
    const double ln = 0.6931471805599453 * (ea + 52) + (double)logf((float)((double)A * 0x1p-52));
    const double step = r0 * (rel - ln * (0x1p-54 / 3.0));
    const double err = fabs(r0) * 0x1p-74;
    const double up = r0 + (step + err);
    *out = up;
    return up == r0 + (step - err);
}

}  // namespace fx

constexpr double kPio2_1 = 0x1.921fb54400000p+0, kPio2_2 = 0x1.0b4611a600000p-34, kPio2_3 = 0x1.3198a2e037073p-69;
constexpr double kTwoOverPi = 0x1.45f306dc9c883p-1;
constexpr double kLn2Hi = 0x1.62e42fefa39efp-1, kLn2Lo = 0x1.abc9e3b39803fp-56;

// sin(r)/r (cosine false) and cos(r) (cosine true) as polynomials in
// r2 = r*r (Taylor, to r^29 / r^28). Both have the same shape, so lanes of a
// warp that evaluate different ones run one instruction sequence.
CR_HD dd sc_poly(dd r2, bool cosine) {
#define CR_SEL(s, c) (cosine ? (c) : (s))
    double t = CR_SEL(0x1.259f98b4358adp-103, 0x1.0a18a2635085dp-98);
    t = t * r2.hi + CR_SEL(-0x1.d1ab1c2dccea3p-94, -0x1.88e85fc6a4e5ap-89);
    t = t * r2.hi + CR_SEL(0x1.3f3ccdd165fa9p-84, 0x1.f2cf01972f578p-80);
    t = t * r2.hi + CR_SEL(-0x1.761b41316381ap-75, -0x1.0ce396db7f853p-70);
    t = t * r2.hi + CR_SEL(0x1.71b8ef6dcf572p-66, 0x1.e542ba4020225p-62);
    t = t * r2.hi + CR_SEL(-0x1.2f49b46814157p-57, -0x1.6827863b97d97p-53);
    dd p = {t, 0.0};
    p = add(mul(p, r2), dd{CR_SEL(0x1.952c77030ad4ap-49, 0x1.ae7f3e733b81fp-45),
                           CR_SEL(0x1.ac981465ddc6cp-103, 0x1.1d8656b0ee8cbp-101)});
    p = add(mul(p, r2), dd{CR_SEL(-0x1.ae7f3e733b81fp-41, -0x1.93974a8c07c9dp-37),
                           CR_SEL(-0x1.1d8656b0ee8cbp-97, -0x1.05d6f8a2efd1fp-92)});
    p = add(mul(p, r2), dd{CR_SEL(0x1.6124613a86d09p-33, 0x1.1eed8eff8d898p-29),
                           CR_SEL(0x1.f28e0cc748ebep-87, -0x1.2aec959e14c06p-83)});
    p = add(mul(p, r2), dd{CR_SEL(-0x1.ae64567f544e4p-26, -0x1.27e4fb7789f5cp-22),
                           CR_SEL(0x1.c062e06d1f209p-80, -0x1.cbbc05b4fa99ap-76)});
    p = add(mul(p, r2), dd{CR_SEL(0x1.71de3a556c734p-19, 0x1.a01a01a01a01ap-16),
                           CR_SEL(-0x1.c154f8ddc6c00p-73, 0x1.a01a01a01a01ap-76)});
    p = add(mul(p, r2), dd{CR_SEL(-0x1.a01a01a01a01ap-13, -0x1.6c16c16c16c17p-10),
                           CR_SEL(-0x1.a01a01a01a01ap-73, 0x1.f49f49f49f49fp-65)});
    p = add(mul(p, r2), dd{CR_SEL(0x1.1111111111111p-7, 0x1.5555555555555p-5),
                           CR_SEL(0x1.1111111111111p-63, 0x1.5555555555555p-59)});
    p = add(mul(p, r2), dd{CR_SEL(-0x1.5555555555555p-3, -0x1.0000000000000p-1),
                           CR_SEL(-0x1.5555555555555p-57, 0x0.0p+0)});
    p = add(mul(p, r2), dd{0x1.0000000000000p+0, 0x0.0p+0});
#undef CR_SEL
    return p;
}

CR_HD dd sin_poly(dd r2) { return sc_poly(r2, false); }
CR_HD dd cos_poly(dd r2) { return sc_poly(r2, true); }

// atanh(u)/u as a polynomial in u2 = u*u (to u^46)
CR_HD dd atanh_poly(dd u2) {
    double t = 0x1.5c9882b931057p-6;
    t = t * u2.hi + 0x1.6c16c16c16c17p-6;
    t = t * u2.hi + 0x1.7d05f417d05f4p-6;
    t = t * u2.hi + 0x1.8f9c18f9c18fap-6;
    t = t * u2.hi + 0x1.a41a41a41a41ap-6;
    t = t * u2.hi + 0x1.bacf914c1bad0p-6;
    t = t * u2.hi + 0x1.d41d41d41d41dp-6;
    t = t * u2.hi + 0x1.f07c1f07c1f08p-6;
    t = t * u2.hi + 0x1.0842108421084p-5;
    t = t * u2.hi + 0x1.1a7b9611a7b96p-5;
    t = t * u2.hi + 0x1.2f684bda12f68p-5;
    t = t * u2.hi + 0x1.47ae147ae147bp-5;
    t = t * u2.hi + 0x1.642c8590b2164p-5;
    dd p = {t, 0.0};
    p = add(mul(p, u2), dd{0x1.8618618618618p-5, 0x1.8618618618618p-59});
    p = add(mul(p, u2), dd{0x1.af286bca1af28p-5, 0x1.af286bca1af28p-59});
    p = add(mul(p, u2), dd{0x1.e1e1e1e1e1e1ep-5, 0x1.e1e1e1e1e1e1ep-61});
    p = add(mul(p, u2), dd{0x1.1111111111111p-4, 0x1.1111111111111p-60});
    p = add(mul(p, u2), dd{0x1.3b13b13b13b14p-4, -0x1.3b13b13b13b14p-58});
    p = add(mul(p, u2), dd{0x1.745d1745d1746p-4, -0x1.745d1745d1746p-59});
    p = add(mul(p, u2), dd{0x1.c71c71c71c71cp-4, 0x1.c71c71c71c71cp-58});
    p = add(mul(p, u2), dd{0x1.2492492492492p-3, 0x1.2492492492492p-57});
    p = add(mul(p, u2), dd{0x1.999999999999ap-3, -0x1.999999999999ap-57});
    p = add(mul(p, u2), dd{0x1.5555555555555p-2, 0x1.5555555555555p-56});
    p = add(mul(p, u2), dd{0x1.0000000000000p+0, 0x0.0p+0});
    return p;
}

// x - k*pi/2 in double-double and the quadrant k mod 4 (|x| < 2^20).
CR_HD dd reduce_pio2(double x, int* quadrant) {
    double k = rint(x * kTwoOverPi);
    dd r = two_sum(x, -(k * kPio2_1));  // k*kPio2_1 is exact: 33-bit constant
    r = add(r, neg(two_prod(k, kPio2_2)));
    r = add(r, neg(two_prod(k, kPio2_3)));
    *quadrant = ((int)k) & 3;
    return r;
}

CR_HD void sincos_dd(double x, dd* s, dd* c) {
    int q;
    dd r = reduce_pio2(x, &q);
    dd r2 = mul(r, r);
    dd sr = mul(sin_poly(r2), r);
    dd cr_ = cos_poly(r2);
    switch (q) {
        case 0: *s = sr; *c = cr_; break;
        case 1: *s = cr_; *c = neg(sr); break;
        case 2: *s = neg(sr); *c = neg(cr_); break;
        default: *s = neg(cr_); *c = sr; break;
    }
}

// cos and sin each need one of the two polynomials (which one depends on
// the quadrant); the value is the one sincos_dd gives.
CR_HD double cos_slow(double x) {
    if (!(fabs(x) < 1048576.0)) return ::cos(x);  // outside the reduction range: not used here
    int q;
    const dd r = reduce_pio2(x, &q);
    const dd r2 = mul(r, r);
    switch (q) {
        case 0: return cos_poly(r2).hi;
        case 1: return neg(mul(sin_poly(r2), r)).hi;
        case 2: return neg(cos_poly(r2)).hi;
        default: return mul(sin_poly(r2), r).hi;
    }
}

CR_HD double sin_slow(double x) {
    if (x == 0.0) return x;
    if (!(fabs(x) < 1048576.0)) return ::sin(x);
    int q;
    const dd r = reduce_pio2(x, &q);
    const dd r2 = mul(r, r);
    switch (q) {
        case 0: return mul(sin_poly(r2), r).hi;
        case 1: return cos_poly(r2).hi;
        case 2: return neg(mul(sin_poly(r2), r)).hi;
        default: return neg(cos_poly(r2)).hi;
    }
}

CR_HD double cos(double x) {
    double r;
    return fx::sin_or_cos(x, true, &r) ? r : cos_slow(x);
}

CR_HD double sin(double x) {
    double r;
    return fx::sin_or_cos(x, false, &r) ? r : sin_slow(x);
}

// sin(x) and cos(x) of one argument: the same values as sin and cos.
CR_HD void sincos(double x, double* sn, double* cs) {
    if (fx::sin_or_cos(x, false, sn) && fx::sin_or_cos(x, true, cs)) return;
    if (!(fabs(x) < 1048576.0)) {
        *sn = x == 0.0 ? x : ::sin(x);
        *cs = ::cos(x);
        return;
    }
    if (x == 0.0) {
        *sn = x;
        *cs = cos_slow(x);
        return;
    }
    dd s, c;
    sincos_dd(x, &s, &c);
    *sn = s.hi;
    *cs = c.hi;
}

#ifdef __CUDACC__
// sincos(x) by a whole warp, every lane passing the same x: lane 1
// evaluates the cosine polynomial while the others evaluate the sine one
// (sc_poly, no divergence), which halves the serial chain of a one-lane
// sincos. Every lane gets the values sincos gives.
__device__ __forceinline__ void sincos_warp(double x, double* sn, double* cs) {
    {
        double v = 0.0;
        const bool ok = fx::sin_or_cos(x, (threadIdx.x & 31) == 1, &v);
        if (__all_sync(0xffffffffu, ok)) {
            *sn = __shfl_sync(0xffffffffu, v, 0);
            *cs = __shfl_sync(0xffffffffu, v, 1);
            return;
        }
    }
    if (!(fabs(x) < 1048576.0) || x == 0.0) {  // the same branch in every lane
        sincos(x, sn, cs);
        return;
    }
    int q;
    const dd r = reduce_pio2(x, &q);
    const dd r2 = mul(r, r);
    const bool cosine = (threadIdx.x & 31) == 1;
    const dd p = sc_poly(r2, cosine);
    const dd pr = mul(p, r);
    const dd v = cosine ? p : pr;
    const dd sr = {__shfl_sync(0xffffffffu, v.hi, 0), __shfl_sync(0xffffffffu, v.lo, 0)};
    const dd cr_ = {__shfl_sync(0xffffffffu, v.hi, 1), __shfl_sync(0xffffffffu, v.lo, 1)};
    switch (q) {
        case 0: *sn = sr.hi; *cs = cr_.hi; break;
        case 1: *sn = cr_.hi; *cs = neg(sr).hi; break;
        case 2: *sn = neg(sr).hi; *cs = neg(cr_).hi; break;
        default: *sn = neg(cr_).hi; *cs = sr.hi; break;
    }
}
#endif

// asin(t) for t in [0, 0.5] given as a double-double, as a double-double.
CR_HD dd asin_small_dd(dd t) {
    double z0 = ::asin(t.hi);
    dd s, c;
    sincos_dd(z0, &s, &c);
    dd num = add(t, neg(s));
    double corr = num.hi / c.hi;
    return two_sum(z0, corr);
}

// sqrt(u) of a double as a double-double.
CR_HD dd sqrt_dd(double u) {
    double t0 = ::sqrt(u);
    if (t0 == 0.0) return dd{0.0, 0.0};
    double res = fma(-t0, t0, u);
    return fast_two_sum(t0, res / (2.0 * t0));
}

CR_HD double acos_slow(double x) {
    if (fabs(x) <= 0.5) {
        double y0 = ::acos(x);
        dd s, c;
        sincos_dd(y0, &s, &c);
        dd num = add_d(c, -x);
        double corr = num.hi / s.hi;
        return y0 + corr;
    }
    if (x > 0.0) {
        double u = (1.0 - x) * 0.5;  // exact for x in (0.5, 1]
        if (u == 0.0) return 0.0;
        dd z = asin_small_dd(sqrt_dd(u));
        return 2.0 * (z.hi + z.lo);
    }
    double u = (1.0 + x) * 0.5;  // exact for x in [-1, -0.5)
    dd z = asin_small_dd(sqrt_dd(u));
    dd r = add(dd{kPiHi, kPiLo}, dd{-2.0 * z.hi, -2.0 * z.lo});
    return r.hi;
}

CR_HD double acos(double x) {
    const double y0 = ::acos(fabs(x) > 0.5 ? fabs(x) : x);
    if (!(fabs(x) < 1.0)) return x == 1.0 ? 0.0 : x == -1.0 ? kPiHi : y0;  // else NaN, as the library gives
    double r;
    return fx::acos_from(x, y0, &r) ? r : acos_slow(x);
}

// ln(x) for finite x > 0 as a double-double.
CR_HD dd log_dd(double x) {
    int k;
    double m = frexp(x, &k);  // x = m 2^k, m in [0.5, 1)
    if (m < 0.70710678118654752) {
        m *= 2.0;
        k -= 1;
    }
    dd num = dd{m - 1.0, 0.0};  // exact: m in [0.707, 1.414)
    dd den = two_sum(m, 1.0);
    dd u = div(num, den);
    dd u2 = mul(u, u);
    dd at = mul(atanh_poly(u2), u);
    dd lnm = dd{2.0 * at.hi, 2.0 * at.lo};
    dd kl = add(two_prod((double)k, kLn2Hi), two_prod((double)k, kLn2Lo));
    return add(lnm, kl);
}

// pow(a, y) for a and its result in 1e-300 .. 1e300
CR_HD double pow_slow(double a, double y) {
    double r0 = ::pow(a, y);
    if (!(r0 > 1.0e-300) || !(r0 < 1.0e300)) return r0;
    dd L = mul_d(log_dd(a), y);
    dd delta = add(L, neg(log_dd(r0)));
    return r0 + r0 * delta.hi;
}

// pow(a, y) for finite a > 0 (a = 0 gives 0 for y > 0).
CR_HD double pow(double a, double y) {
    if (!(a > 0.0) || !(a < 1.0e300) || a < 1.0e-300 || !(fabs(y) < 1.0e3)) return ::pow(a, y);
    if (a == 1.0) return 1.0;
    double r;
    if (y == 1.0 / 3.0 && fx::cube_root_from(a, ::cbrt(a), &r)) return r;
    return pow_slow(a, y);
}

}  // namespace cr
}  // namespace ccg
