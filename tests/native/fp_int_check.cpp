// Every function of csrc/fp_int.cuh against the host's FP64 arithmetic, and the
// canonical exp, log and cube root of csrc/canon_math.cuh against the oracle's:
// edge values, powers of two and their neighbours, and a seeded random sweep.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "canon_math.cuh"
#undef CM_LN2_HI
#undef CM_LN2_LO
#undef CM_INV_LN2
#undef CM_FN
namespace host {
#include "canon_math.h"   // the oracle's copy
}

using namespace gbrkc;

static int bad = 0;
static void fail(const char *what, double a, double b) {
  if (bad++ < 10) std::printf("%s differs at %a, %a\n", what, a, b);
}
static bool same(double a, double b) { return fpi_bits(a) == fpi_bits(b) || (a != a && b != b); }
static bool samef(float a, float b) { return fpi_fbits(a) == fpi_fbits(b) || (a != a && b != b); }

static void canon(double x) {
  if (!same(::cm_exp(x), host::cm_exp(x))) fail("cm_exp", x, 0);
  if (!same(::cm_log(x), host::cm_log(x))) fail("cm_log", x, 0);
  if (!same(::cm_cbrt(x), host::cm_cbrt(x))) fail("cm_cbrt", x, 0);
}

static void check(double a, double b) {
  if (!same(fpi_abs(a), std::fabs(a))) fail("fpi_abs", a, b);
  if (fpi_isnan(a) != (a != a)) fail("fpi_isnan", a, b);
  if (!samef(d2f(a), (float)a)) fail("d2f", a, b);
  const double p = std::fabs(a), q = std::fabs(b);
  if (nn_lt(p, q) != (p < q) || nn_le(p, q) != (p <= q)) fail("nn_lt / nn_le", p, q);
  if (fpi_is_zero(a) != (a == 0.0)) fail("fpi_is_zero", a, b);
  if (!same(mdiv(a, b), a / b)) fail("mdiv", a, b);
  if (p != p || q != q) return;
  if (!same(abs_max(a, b), p > q ? p : q)) fail("abs_max", a, b);
}

// quotients by the kinds of constant that the gating uses: a power of two, a
// short mantissa, a full one
static void constants(double a) {
#define GB_C(b) \
  if (!same(cdiv(a, b), a / (b))) fail("cdiv " #b, a, b);
  GB_C(8.0) GB_C(-16.0) GB_C(0.25) GB_C(3.0) GB_C(6.0) GB_C(7.0) GB_C(10.0) GB_C(-10.0) GB_C(12.5) GB_C(14.5) GB_C(20.0)
  GB_C(30.0) GB_C(17.0) GB_C(62.5) GB_C(83.0) GB_C(900.0) GB_C(-12.0) GB_C(14.9) GB_C(23.32708) GB_C(0.85) GB_C(0.099986667)
  GB_C(4.2) GB_C(-5.8) GB_C(1.9297e-1) GB_C(1048577.0) GB_C(2097151.0)
#undef GB_C
}

int main() {
  std::vector<double> v = {0.0, -0.0, 1.0, -1.0, 0.1, 1e-9, 65.0, -65.3, 1e300, -1e300, INFINITY, -INFINITY, NAN,
                           0x1p-1074, 0x1p-1022, 0x1p-149, 0x1p-150, 0x1.8p-150, 0x1p-126, 0x1.fffffffffffffp-127,
                           0x1.fffffep127, 0x1.ffffffp127, 0x1.fffffefffffffp127, 0x1p128, 0x1.000001p0,
                           0x1.0000010000001p0, 0x1.000003p0, 0x1.0000030000001p0, 0x1.fffffffp5};
  for (int e = -160; e <= 140; e++) {
    const double x = std::ldexp(1.0, e);
    for (double y : {x, std::nextafter(x, 0.0), std::nextafter(x, INFINITY), x * 1.5, -x}) v.push_back(y);
  }
  for (double x : {709.782712893384, 709.7827128933841, -745.1332191019412, -745.14, 704.0, -704.0, -744.0,
                   0x1.6a09e667f3bccp+0, 0x1.6a09e667f3bcdp+0, 0x1.6a09e667f3bcep+0}) v.push_back(x);
  for (double a : v) {
    canon(a);
    constants(a);
    for (double b : v) check(a, b);
  }
  std::mt19937_64 rng(7);
  for (int i = 0; i < 500000; i++) {
    uint64_t u = rng(), w = rng();
    canon(fpi_double(u));
    constants(fpi_double(u));
    constants(1.0 + (double)(u >> 12) * 0x1p-52);
    constants(-100.0 + (double)(w >> 11) * 0x1p-45);
    canon((double)(int64_t)w * 0x1p-63 * 800);
    canon(1.0 + (double)(int64_t)u * 0x1p-64);
    check(fpi_double(u), fpi_double(w));
    // magnitudes around 1, ties of the FP32 rounding among them
    const double x = fpi_double((u & 0x000fffffffffffffULL) | ((uint64_t)(1023 - 60 + (w % 120)) << 52));
    check(x, fpi_double(fpi_bits(x) ^ (w & 3)));
    check(fpi_double((fpi_bits(x) & ~0x1fffffffULL) | 0x10000000ULL | (w & 1)), x);
    // divisors and dividends with few set or few clear bits, and exact products
    const double m = fpi_double((fpi_bits(x) & 0xfff0000000000000ULL) | (0x000fffffffffffffULL - (w & 1023)));
    check(x, m);
    check(m, fpi_double(0x3ff0000000000000ULL + (w & 1023)));
    check(x * (double)(w & 0xffff), (double)(1 + (u & 0xffff)));
  }
  for (uint32_t u = 0; u < 0xffffff00u; u += 251) {
    const float f = fpi_float(u);
    if (!same(f2d(f), (double)f)) fail("f2d", f, 0);
  }
  for (float f : {0.0f, -0.0f, 0x1p-149f, 0x1p-126f, 0x1.fffffep127f, INFINITY, -INFINITY})
    if (!same(f2d(f), (double)f)) fail("f2d", f, 0);
  auto root = [](double x) {
    bool ok;
    const int s = int_sqrt(x, ok);
    const bool in = x >= 1.0 && x < 0x1p23;
    if (ok != in) fail("int_sqrt range", x, 0);
    if (ok && s != (int)std::sqrt(x)) fail("int_sqrt", x, s);
  };
  // every integer root's threshold, a few last places either side
  for (int s = 1; s <= 2900; s++) {
    double lo = (double)s * s, hi = lo;
    root(lo);
    for (int k = 0; k < 4; k++) {
      lo = std::nextafter(lo, 0.0);
      hi = std::nextafter(hi, INFINITY);
      root(lo);
      root(hi);
    }
  }
  for (int s = 1; s <= 4095; s++) {
    const double t = fpi_double(sqrt_reaches(s));
    if (!(std::sqrt(t) >= s) || std::sqrt(std::nextafter(t, 0.0)) >= s) fail("sqrt_reaches", s, t);
  }
  for (int i = 0; i < 3000000; i++) root(1.0 + std::ldexp((double)(rng() >> 11), -53) * std::ldexp(1.0, rng() % 23));
  for (double x : {0.0, 0.5, 0x1.fffffffffffffp-1, 0x1p23, 1e18, 1e300, (double)INFINITY, (double)NAN, -1.0}) root(x);
  std::printf(bad ? "%d differences\n" : "fp_int: all equal\n", bad);
  return bad != 0;
}
