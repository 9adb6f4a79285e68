// Host check of fb::div_core and fb::sqrt_core (modpath-rw_gb300/csrc/fpbits.cuh)
// against the IEEE-754 operators, bit for bit, on operands the plain-range
// tests accept: random significands and exponents, significands at both ends
// of [1, 2), nearly equal operands, perfect squares and their neighbours, and
// exponents at the edges of the plain range -- with the FP32 approximations
// that start the digits perturbed by -4..4 units in the last place (the
// device's are within one or two of the correctly rounded ones used here).
// Prints "ok <n>" or the first mismatches; exit status 1 on a mismatch.
#include <cstdio>
#include <random>

#include "fpbits.cuh"

using namespace mprw::fb;

static long long g_checked = 0, g_bad = 0;

static void check_div(double a, double b) {
  if (!div_plain(a, b)) return;
  g_checked += 2;
  const double q = a / b, w = div_core(a, b, 0), h = div_core(a, b, 1);
  if ((bits(q) != bits(w) || bits(q * 0.5) != bits(h)) && g_bad++ < 20)
    std::printf("MISMATCH %a / %a = %a got %a, half %a\n", a, b, q, w, h);
}

static void check_sqrt(double x) {
  if (!sqrt_plain(x)) return;
  ++g_checked;
  const double r = std::sqrt(x), w = sqrt_core(x);
  if (bits(r) != bits(w) && g_bad++ < 20) std::printf("MISMATCH sqrt(%a) = %a got %a\n", x, r, w);
}

// |a b| > 1/2 against the rounded product's compare
static void check_prod(double a, double b) {
  ++g_checked;
  volatile double p = a * b;
  const bool want = std::fabs(p) > 0.5, got = prod_above_half(a, b);
  if (got != want && g_bad++ < 20) std::printf("MISMATCH |%a * %a| > 1/2: got %d want %d\n", a, b, got, want);
}

int main() {
  const unsigned long long sig = 0x000FFFFFFFFFFFFFULL;
  std::mt19937_64 rng(20240);
  for (int k = -4; k <= 4; ++k) {
    host_approx_ulps() = k;
    for (int i = 0; i < 500000; ++i) {
      unsigned long long ra = rng(), rb = rng();
      if (i % 7 == 0) ra |= 0x000FFFFFFFFF0000ULL;
      if (i % 11 == 0) rb |= 0x000FFFFFFF000000ULL;
      if (i % 13 == 0) rb &= ~0x000FFFFFFFFF0000ULL;
      if (i % 17 == 0) ra &= ~0x000000FFFFFFFF00ULL;
      if (i % 19 == 0) ra = (ra & ~sig) | ((rb + (unsigned)(i % 5) - 2) & sig);
      check_div(from_bits(ra), from_bits(rb));
      check_sqrt(from_bits(ra & 0x7FFFFFFFFFFFFFFFULL));
      if (i % 5 == 0) {
        const double y = from_bits(0x3000000000000000ULL | (rb & 0x0FFFFFFFF0000000ULL));
        check_sqrt(y * y);
        check_sqrt(std::nextafter(y * y, 1e308));
        check_sqrt(std::nextafter(y * y, 0.0));
      }
    }
    // the edges of the significand and exponent ranges against one another
    const unsigned long long m[] = {0, 1, 2, sig, sig - 1, sig >> 1, (sig >> 1) + 1, 0x0008000000000001ULL,
                                    0x000FFFFFE0000000ULL, 0x000FFFFFDFFFFFFFULL, 0x0000000020000000ULL};
    for (unsigned long long x : m)
      for (unsigned long long y : m)
        for (unsigned ea : {1u, 2u, 3u, 1022u, 1023u, 1024u, 2044u, 2045u, 2046u})
          for (unsigned eb : {1u, 2u, 3u, 1021u, 1022u, 1023u, 1024u, 1025u, 2045u, 2046u}) {
            const double a = from_bits(((unsigned long long)ea << 52) | x);
            const double b = from_bits(((unsigned long long)eb << 52) | y);
            check_div(a, b);
            check_div(-a, b);
            check_sqrt(a);
          }
  }
  // products around 1/2 (every exponent sum from 2^-4 to 2^1), at it exactly
  // and next to it, and with special values
  for (int i = 0; i < 3000000; ++i) {
    const unsigned long long ra = rng(), rb = rng();
    const int e = (int)(ra >> 60) - 8;
    double a = from_bits(((unsigned long long)(1023 + e) << 52) | (ra & sig));
    double b = from_bits(((unsigned long long)(1023 - e - 3 + (int)(rb >> 61) % 5) << 52) | (rb & sig));
    if (i % 3 == 0) b = 0.5 / a;
    if (i % 3 == 1 && i % 2) b = std::nextafter(0.5 / a, i % 4 == 1 ? 2.0 : 0.0);
    check_prod(i % 5 ? a : -a, b);
  }
  const double special[] = {0.0, -0.0, from_bits(1), 1e-310, 0.5, -0.5, 1.0, -1.0, std::nextafter(1.0, 2.0),
                            std::nextafter(0.5, 0.0), 2.0, 1e300, 1e-300, INFINITY, -INFINITY, (double)NAN};
  for (double a : special)
    for (double b : special) check_prod(a, b);
  // refused operands: zeros, subnormals, infinities, NaN, quotients (or their
  // halves) outside the normal range, negative radicands
  const double inf = INFINITY, tiny = from_bits(1), least = from_bits(0x0010000000000000ULL);
  for (double z : {0.0, -0.0, tiny, -tiny, inf, -inf, (double)NAN}) {
    g_checked += 3;
    if (div_plain(z, 1.0) || div_plain(1.0, z) || sqrt_plain(z)) {
      ++g_bad;
      std::printf("ACCEPTED %a\n", z);
    }
  }
  g_checked += 3;
  if (div_plain(least, 2.0) || div_plain(1e308, 1e-10) || sqrt_plain(-1.0)) {
    ++g_bad;
    std::printf("ACCEPTED an operand pair out of range\n");
  }
  if (g_bad) {
    std::printf("%lld mismatches of %lld\n", g_bad, g_checked);
    return 1;
  }
  std::printf("ok %lld\n", g_checked);
  return 0;
}
