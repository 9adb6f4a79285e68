// fpbits.cuh -- FP64 tests and compares taken from IEEE-754 bit patterns on
// the integer pipe, and the Irwin-Hall normal assembled from its bits.
//
// GB300 issues two FP64 lanes per clock per SM, so an FP64 compare holds the
// FP64 pipe as long as a multiply-add; the FP64 step kernel is bound by that
// pipe.  Each function here gives the FP64 compare's answer for every input
// (signed zeros, subnormals and infinities as the compare orders them, NaN
// false like the compare) in a few integer instructions.  A range test is one
// unsigned subtraction and compare: b in [lo, hi] <=> b - lo < hi - lo + 1.
// The header also compiles as plain C++ for the host, where the tests check
// every function against the compare it replaces.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define MPRW_FB __host__ __device__ __forceinline__
#else
#define MPRW_FB inline
#endif

namespace mprw {
namespace fb {

MPRW_FB unsigned long long bits(double v) {
#if defined(__CUDA_ARCH__)
  return (unsigned long long)__double_as_longlong(v);
#else
  unsigned long long b;
  std::memcpy(&b, &v, sizeof b);
  return b;
#endif
}

MPRW_FB double from_bits(unsigned long long b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double v;
  std::memcpy(&v, &b, sizeof v);
  return v;
#endif
}

// v > 1: bits in (bits(1), bits(+inf)]
MPRW_FB bool above1(double v) { return bits(v) - 0x3FF0000000000001ULL < 0x4000000000000000ULL; }
// v < 0: bits in (bits(-0), bits(-inf)]; -0 is not below 0
MPRW_FB bool below0(double v) { return bits(v) - 0x8000000000000001ULL < 0x7FF0000000000000ULL; }
// v > 0: bits in (bits(+0), bits(+inf)]
MPRW_FB bool above0(double v) { return bits(v) - 1ULL < 0x7FF0000000000000ULL; }
// v == 0: +0 or -0
MPRW_FB bool is0(double v) { return (bits(v) << 1) == 0ULL; }
// v == 1
MPRW_FB bool is1(double v) { return bits(v) == 0x3FF0000000000000ULL; }
// v >= 0: [+0, +inf] or -0
MPRW_FB bool nonneg(double v) {
  const unsigned long long b = bits(v);
  return (b <= 0x7FF0000000000000ULL) | (b == 0x8000000000000000ULL);
}
// |v| > 1/2: |v|'s bits in (bits(1/2), bits(+inf)]
MPRW_FB bool abs_above_half(double v) {
  return (bits(v) & 0x7FFFFFFFFFFFFFFFULL) - 0x3FE0000000000001ULL < 0x4010000000000000ULL;
}
// v > 1 or v < 0
MPRW_FB bool out01(double v) { return above1(v) | below0(v); }
// a < b for a, b > 0 (not NaN): the bit patterns of positive doubles are
// ordered as their values
MPRW_FB bool pos_lt(double a, double b) { return bits(a) < bits(b); }

// a < b and a == b for any two doubles.  Mapped to two's-complement keys
// (negative values: the magnitude bits flipped, so larger magnitudes are
// smaller keys; -0 first taken as +0) the keys are ordered as the values.
MPRW_FB bool isnan_bits(double v) { return (bits(v) & 0x7FFFFFFFFFFFFFFFULL) > 0x7FF0000000000000ULL; }
MPRW_FB long long order_key(double v) {
  long long b = (long long)bits(v);
  b = (b == (long long)0x8000000000000000ULL) ? 0LL : b;
  return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL);
}
MPRW_FB bool lt_any(double a, double b) {
  return !(isnan_bits(a) | isnan_bits(b)) & (order_key(a) < order_key(b));
}
MPRW_FB bool eq_any(double a, double b) {
  return !(isnan_bits(a) | isnan_bits(b)) & (order_key(a) == order_key(b));
}

// maxTime < t (the end of the tracking interval passed): for maxTime in
// [+0, +inf] exactly one unsigned range test on t's bits, t > maxTime <=>
// bits(t) in [bits(maxTime) + 1, bits(+inf)] (NaN and negative t fall
// outside); any other maxTime takes the FP64 compare.  In a kernel the branch
// is uniform (maxTime is the launch's).
MPRW_FB bool past_end(double maxTime, double t) {
  const unsigned long long km = bits(maxTime);
  if (km <= 0x7FF0000000000000ULL) return bits(t) - (km + 1ULL) < 0x7FF0000000000000ULL - km;
  return maxTime < t;
}

// |a b| > 1/2, the product rounded: from the exponents, and where those leave
// it open (significands whose product decides between 1/4 and 1) from the
// significands' leading 32 bits; the product itself only within 2^-29 of 1/2.
MPRW_FB unsigned mulhi_u(unsigned a, unsigned b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (unsigned)(((unsigned long long)a * b) >> 32);
#endif
}
MPRW_FB bool prod_above_half(double a, double b) {
  const unsigned long long ba = bits(a), bb = bits(b);
  const int ea = (int)((ba >> 52) & 0x7FF), eb = (int)((bb >> 52) & 0x7FF);
  const int e = ea + eb - 2046;  // |a b| in [2^e, 2^(e+2)) for normal a, b
  if ((unsigned)(ea - 1) < 2046u && (unsigned)(eb - 1) < 2046u) {
    if (e >= 0) return true;
    if (e <= -3) return false;
    const unsigned ha = 0x80000000u | (unsigned)((ba >> 21) & 0x7FFFFFFFu);
    const unsigned hb = 0x80000000u | (unsigned)((bb >> 21) & 0x7FFFFFFFu);
    const unsigned p = mulhi_u(ha, hb);  // significands' product in 2^-30, less than 3 units low
    const unsigned half = e == -1 ? 0x40000000u : 0x80000000u;
    if (p > half) return true;
    if (p < half - 3u) return false;
  } else if ((ba << 1) == 0ULL && eb < 2047) {
    return false;
  }
  return abs_above_half(a * b);
}

MPRW_FB int clz64(unsigned long long m) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)m);
#else
  return m ? __builtin_clzll(m) : 64;
#endif
}

// The Irwin-Hall(12) normal S*2^-32 - 6 of the 36-bit sum S of twelve 32-bit
// words, exact (|S - 6*2^32| < 2^36), assembled from its sign, exponent and
// mantissa: the same bits as (2^20 + S*2^-32) - (2^20 + 6) in FP64, +0 for
// S = 6*2^32.
MPRW_FB double ih12_normal(unsigned long long sum) {
  const long long k = (long long)sum - (6LL << 32);
  const unsigned long long m = (unsigned long long)(k < 0 ? -k : k);
  const int e = 63 - clz64(m);  // most significant bit, 0..35
  const unsigned long long b = ((unsigned long long)k & 0x8000000000000000ULL) |
                               ((unsigned long long)(e + 991) << 52) |  // 991 = 1023 - 32
                               ((m << (52 - e)) & 0x000FFFFFFFFFFFFFULL);
  return from_bits(m ? b : 0ULL);
}

// ---- division and square root on the integer pipe ---------------------------
// a / b and sqrt(x), correctly rounded to nearest, for FP64 operands: the same
// bits as the FP64 operators, which IEEE-754 rounds the same way.  An FP64
// division or square root is a chain of about nine dependent FP64 instructions,
// each holding GB300's FP64 pipe for 16 clocks per warp; here the FP64 pipe is
// not used at all.  The quotient (root) is built in three digits of a long
// division (digit-by-digit root): each digit is the running remainder's top 32
// bits times a 32-bit reciprocal (inverse root) taken from the FP32
// approximation, the remainder is carried exactly in 64-bit wrapping integers,
// and the last remainder decides the final unit.  With the reciprocal within
// 2^-20 relative (the FP32 approximations are within 2^-21.5, truncated
// operand included) the digits leave the 54-bit result at most one unit off
// before that last step; the host test runs both with the approximation
// perturbed either way.  A quotient of two 53-bit significands, and a root of
// one, never lies midway between two of them, so the extra (54th) bit alone
// rounds to nearest.
// Operands or quotients outside the plain normal range (zeros, subnormals,
// infinities, NaN, negative radicands, exponents at the ends) take the
// operator: div_plain / sqrt_plain tell.
#if !defined(__CUDA_ARCH__)
// the host stands in for the two FP32 approximations, off by this many ulps
inline int &host_approx_ulps() {
  static int k = 0;
  return k;
}
inline float host_approx(float r) {
  unsigned u;
  std::memcpy(&u, &r, 4);
  u += (unsigned)host_approx_ulps();
  std::memcpy(&r, &u, 4);
  return r;
}
#endif
// bits of the FP32 approximations 1/f and 1/sqrt(f), f given by its bits
MPRW_FB unsigned rcp_bits(unsigned f) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
#else
  float x, r;
  std::memcpy(&x, &f, 4);
  r = host_approx(1.0f / x);
  unsigned u;
  std::memcpy(&u, &r, 4);
  return u;
#endif
}
MPRW_FB unsigned rsqrt_bits(unsigned f) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
#else
  float x, r;
  std::memcpy(&x, &f, 4);
  r = host_approx((float)(1.0 / std::sqrt((double)x)));
  unsigned u;
  std::memcpy(&u, &r, 4);
  return u;
#endif
}
// an approximation in (1/2, 1), by its bits, as a 31-bit fraction (its rounding
// kept from reaching either end)
MPRW_FB int frac31(unsigned r) {
  r = r < 0x3F000000u ? 0x3F000000u : (r > 0x3F7FFFFFu ? 0x3F7FFFFFu : r);
  return (int)((r << 7) & 0x3FFFFF80u) | 0x40000000;
}
// (a * b) >> 32 of a signed and an unsigned 31-bit factor
MPRW_FB int mulhi_s(int a, int b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int)(((long long)a * (long long)b) >> 32);
#endif
}

// both operands normal, and the quotient and its half normal too
MPRW_FB bool div_plain(double a, double b) {
  const unsigned ea = ((unsigned)(bits(a) >> 52) & 0x7FFu) - 1u, eb = ((unsigned)(bits(b) >> 52) & 0x7FFu) - 1u;
  return (ea < 2046u) & (eb < 2046u) & (ea - eb + 1020u < 2042u);
}
// a / b * 2^-scale, scale 0 or 1, for div_plain operands
MPRW_FB double div_core(double a, double b, int scale) {
  const unsigned long long ba = bits(a), bb = bits(b);
  unsigned long long ma = (ba & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL;
  const unsigned long long mb = (bb & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL;
  int e = (int)((ba >> 52) & 0x7FF) - (int)((bb >> 52) & 0x7FF) + 1022 - scale;
  // quotient in [1, 2): shift a left when its significand is the smaller
  const bool less = ma < mb;
  ma <<= less ? 1 : 0;
  e -= less ? 1 : 0;
  // rho = 2^52 / mb in (1/2, 1): the divisor rounded up to 24 bits, so the
  // approximation stays below 1; q31 = rho 2^31
  const int q31 = frac31(rcp_bits(0x3F800001u + (unsigned)((bb >> 29) & 0x7FFFFFULL)));
  // ma / mb = ma * rho * 2^-52.  Digits: 2^-23, 2^-43, 2^-53
  const int q1 = (int)((unsigned)mulhi_s((int)(ma >> 23), q31) >> 5);          // ma (54 bits) -> 24 bits
  const long long r1 = (long long)((ma << 23) - (unsigned long long)(unsigned)q1 * mb);  // |r1| < 2^57
  const int q2 = mulhi_s((int)(r1 >> 26), q31) >> 5;
  const long long r2 = (long long)((unsigned long long)r1 << 20) - (long long)q2 * (long long)mb;  // |r2| < 2^57
  const int q3 = mulhi_s((int)(r2 >> 26), q31) >> 15;
  const long long r3 = (long long)((unsigned long long)r2 << 10) - (long long)q3 * (long long)mb;
  unsigned long long q = ((unsigned long long)(unsigned)q1 << 30) + (unsigned long long)((long long)q2 * 1024 + q3);
  q -= (r3 < 0) ? 1ULL : 0ULL;
  q += (r3 >= (long long)mb) ? 1ULL : 0ULL;
  // q = floor(a/b 2^53), 54 bits: round on its last bit; the carry of 1.11..1
  // moves into the exponent
  const unsigned long long m = (q + 1ULL) >> 1;
  return from_bits(((ba ^ bb) & 0x8000000000000000ULL) | (((unsigned long long)(unsigned)e << 52) + m));
}

// x normal and positive
MPRW_FB bool sqrt_plain(double x) { return bits(x) - 0x0010000000000000ULL < 0x7FE0000000000000ULL; }
// sqrt(x) for sqrt_plain x
MPRW_FB double sqrt_core(double x) {
  const unsigned long long b = bits(x);
  // x = m 4^k, m in [1, 4): M = m 2^52, 54 bits
  const unsigned odd = (unsigned)(b >> 52) & 1u;  // biased exponent odd: 1023 + even, m in [1, 2)
  const unsigned long long M = ((b & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL) << (odd ? 0 : 1);
  const unsigned e = ((unsigned)(b >> 52) + 1023u) >> 1;  // biased exponent of the root (even: m doubled)
  // rho = 1/sqrt(m) in (1/2, 1): m rounded up to its FP32 neighbour
  const int q31 = frac31(rsqrt_bits((odd ? 0x3F800001u : 0x40000001u) + (unsigned)((b >> 29) & 0x7FFFFFULL)));
  // root = s1 2^-23 + d2 2^-43 + d3 2^-53
  const unsigned s1 = (unsigned)mulhi_s((int)(M >> 23), q31) >> 5;              // m rho, 24 bits
  const long long r1 = (long long)(M - ((unsigned long long)s1 * s1 << 6));     // units 2^-52
  const int d2 = mulhi_s((int)(r1 >> 4), q31) >> 5;
  const long long t1 = (long long)((unsigned long long)s1 << 21);
  const long long r2 = (long long)((unsigned long long)r1 << 34) - (long long)d2 * (t1 + d2);  // units 2^-86
  const int d3 = mulhi_s((int)(r2 >> 18), q31) >> 15;
  const unsigned long long s2 = ((unsigned long long)s1 << 20) + (unsigned long long)(long long)d2;
  const long long r3 = (long long)((unsigned long long)r2 << 20) -
                       (long long)d3 * ((long long)(s2 << 11) + d3);            // units 2^-106
  unsigned long long q = (s2 << 10) + (unsigned long long)(long long)d3;
  const bool up = r3 > (long long)(2 * q);
  q -= (r3 < 0) ? 1ULL : 0ULL;
  q += up ? 1ULL : 0ULL;
  const unsigned long long m = (q + 1ULL) >> 1;
  return from_bits(((unsigned long long)(e - 1u) << 52) + m);
}

}  // namespace fb
}  // namespace mprw
