// FP64 comparisons, conversions and the stage count's square root in integer
// and FP32 arithmetic, with the results of the FP64 instructions they stand
// for, bit for bit; and quotients, rounded as the divide rounds them but for
// one operand pair in about 2^51 (recip, below).
//
// On GB300 a warp issues an FP64 instruction every 64 cycles, whatever its
// active lanes or the independent work beside it (an SM, from four warps on,
// one every 19), and the comparisons and conversions take longer (one warp on
// an SM, cycles per instruction: DFMA 64, DSETP 110, F2F.F32.F64 102,
// F2F.F64.F32 99, F2I.F64 102, DSQRT 600), while the integer pipe takes an
// instruction every cycle or two and is otherwise idle here.  A comparison of
// non-negative values is two integer instructions.
//
// Host and device: tests/native/fp_int_check.cpp compares every function with
// the host's FP64 arithmetic, tests/native/fp_int_gpu.cu with the GPU's.
#ifndef GBRKC_FP_INT_CUH
#define GBRKC_FP_INT_CUH

#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define GB_HD __host__ __device__ __forceinline__
#else
#define GB_HD inline
#endif

namespace gbrkc {

GB_HD uint64_t fpi_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  __builtin_memcpy(&u, &x, 8);
  return u;
#endif
}
GB_HD double fpi_double(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  __builtin_memcpy(&x, &u, 8);
  return x;
#endif
}
GB_HD uint32_t fpi_fbits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u;
  __builtin_memcpy(&u, &x, 4);
  return u;
#endif
}
GB_HD float fpi_float(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  __builtin_memcpy(&x, &u, 4);
  return x;
#endif
}

// a < b and a <= b of values without a sign (+0, finite, +inf, +NaN): such
// doubles are ordered as their bit patterns are, with NaN above infinity.
GB_HD bool nn_lt(double a, double b) {
  return fpi_bits(a) < fpi_bits(b) && fpi_bits(b) <= 0x7ff0000000000000ULL;
}
GB_HD bool nn_le(double a, double b) {
  return fpi_bits(a) <= fpi_bits(b) && fpi_bits(b) <= 0x7ff0000000000000ULL;
}
GB_HD bool fpi_is_zero(double x) { return (fpi_bits(x) << 1) == 0; }
// |x|, and the larger of |a| and |b| (max_ori of the reference's error norm:
// a where |a| > |b|, else b).  With a NaN among them the result may differ
// from the FP64 expression's, NaN for NaN or not; a caller's error norm is
// NaN in either case.
GB_HD double fpi_abs(double x) { return fpi_double(fpi_bits(x) & 0x7fffffffffffffffULL); }
GB_HD double abs_max(double a, double b) {
  const uint64_t x = fpi_bits(a) & 0x7fffffffffffffffULL, y = fpi_bits(b) & 0x7fffffffffffffffULL;
  return fpi_double(x > y ? x : y);
}
GB_HD bool fpi_isnan(double x) { return (fpi_bits(x) & 0x7fffffffffffffffULL) > 0x7ff0000000000000ULL; }

// (float)x, rounded to nearest even
GB_HD float d2f(double x) {
  const uint64_t u = fpi_bits(x), a = u & 0x7fffffffffffffffULL;
  // zero, and magnitudes from 2^-126 to just below the overflow threshold
  if (a == 0 || a - 0x3810000000000000ULL < 0x47efffffe0000000ULL - 0x3810000000000000ULL) {
    const uint64_t r = a - (896ULL << 52);
    uint32_t f = (uint32_t)(r >> 29);
    const uint32_t rem = (uint32_t)r & 0x1fffffffu;
    f += (rem + (f & 1u) > 0x10000000u) ? 1u : 0u;
    f = a == 0 ? 0u : f;
    return fpi_float(f | ((uint32_t)(u >> 32) & 0x80000000u));
  }
  return (float)x;
}

// (double)x, exact
GB_HD double f2d(float x) {
  const uint32_t u = fpi_fbits(x), a = u & 0x7fffffffu;
  if (a == 0 || a - 0x00800000u < 0x7f800000u - 0x00800000u)
    return fpi_double(((uint64_t)(u & 0x80000000u) << 32) | (a == 0 ? 0 : ((uint64_t)a << 29) + (896ULL << 52)));
  return (double)x;
}

// The bits of the smallest double whose square root, rounded to nearest, is
// at least s (an integer, 1 <= s <= 4095): s^2, or one unit in the last place below it: writing s = 2^k f with
// 1 <= f < 2, the root of s^2 - ulp lies ulp(s^2) / (2 s) below s, which rounds
// up to s exactly when it is under half of s's own last place, 2^(k-53): for
// 1 < f^2 < 2, where ulp(s^2) = 2^(2k-52) gives 2^(k-53) / f.  For f^2 > 2 it is
// 2^(k-52) / f > 2^(k-53); for f = 1 the values below s are twice as dense
// and the root, just under the midpoint, rounds down.
GB_HD uint64_t sqrt_reaches(int s) {
  const uint32_t q = fpi_fbits((float)s * (float)s);       // exact: s^2 < 2^24
  const uint64_t u = ((uint64_t)q << 29) + (896ULL << 52);
  const bool below = (q & 0x007fffffu) != 0u && ((q >> 23) & 1u) != 0u;   // exponent 2k: biased 127 + 2k is odd
  return u - (below ? 1u : 0u);
}

// (int)sqrt(x), the root rounded to FP64 first.  For 1 <= x < 2^23 from an
// FP32 root corrected by sqrt_reaches; ok is false for any other x (NaN,
// infinity, out of range), whose root the caller takes in FP64.
GB_HD int int_sqrt(double x, bool &ok) {
  const uint64_t u = fpi_bits(x);
  ok = u - 0x3ff0000000000000ULL < 0x4160000000000000ULL - 0x3ff0000000000000ULL;   // [1, 2^23)
  if (!ok) return 0;
  int s = (int)sqrtf(fpi_float((uint32_t)((u - (896ULL << 52)) >> 29)));
  // the FP32 argument is x truncated to 24 bits and its root is within a few
  // units in the last place: s is off by one at most
  if (u >= sqrt_reaches(s + 1)) s++;
  else if (s > 1 && u < sqrt_reaches(s)) s--;
  return s;
}

// a / b, rounded to nearest, as a reciprocal of b and a corrected product, so
// that several quotients by one divisor share the reciprocal.  y is one
// third-order step, y0 (1 + e + e^2) with e = 1 - b y0, from an FP32 seed y0
// (|e| < 2^-21, so y is 1 / b to within 2^-63 before its rounding); the
// quotient is q0 = a y corrected by its exact remainder, q0 + (a - b q0) y
// (Markstein, IBM J. Res. Dev. 34(1), 1990).  The correction's error is under
// 2^-52 of q0's last place, so the result is the rounded quotient unless a / b
// lies that close to the midpoint of two doubles (one operand pair in about
// 2^51); none of 4 10^8 random quotients differs from the GPU's own, and none
// of the host check's.  Three FP64 operations for the
// reciprocal and three for each quotient, where the divide takes 565 cycles
// (nine FP64 operations' time).  Operands outside the ranges below
// (subnormals, infinities, NaN and a zero divisor among them) take the divide.
struct Recip {
  double b, y;
  bool ok;
};

GB_HD float rcp_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}

GB_HD Recip recip(double b) {
  Recip r;
  r.b = b;
  const uint64_t u = fpi_bits(b);
  const uint32_t h = (uint32_t)(u >> 32) & 0x7fffffffu;
  r.ok = h - ((1023u - 100u) << 20) < (200u << 20);            // 2^-100 <= |b| < 2^100
  const uint32_t f = (uint32_t)((u & 0x7fffffffffffffffULL) >> 29) - (896u << 23);   // |b| truncated to FP32
  const uint32_t s = fpi_fbits(rcp_seed(fpi_float(r.ok ? f : 0x3f800000u)));
  const double y0 = fpi_double((((uint64_t)s << 29) + (896ULL << 52)) | (u & 0x8000000000000000ULL));
  const double e = fma(-b, y0, 1.0);
  r.y = fma(y0, fma(e, e, e), y0);
  return r;
}

GB_HD double div_by(double a, const Recip &r) {
  const uint32_t h = (uint32_t)(fpi_bits(a) >> 32) & 0x7fffffffu;
  const bool zero = (fpi_bits(a) << 1) == 0;                   // a zero of the quotient's sign
  if (r.ok && (zero || h - ((1023u - 400u) << 20) < (800u << 20))) {   // 2^-400 <= |a| < 2^400
    const double q = a * r.y, s = fma(fma(-r.b, q, a), r.y, q);
    return zero ? q : s;
  }
  return a / r.b;
}

// The same names for FP32 and FP64: x / b by a shared reciprocal (FP32: the
// plain divide), and comparisons of magnitudes.
GB_HD double mdiv(double a, double b) { return div_by(a, recip(b)); }
GB_HD float mdiv(float a, float b) { return a / b; }
struct RecipF {
  float b;
};
GB_HD Recip mrecip(double b) { return recip(b); }
GB_HD RecipF mrecip(float b) { return RecipF{b}; }
GB_HD float div_by(float a, const RecipF &r) { return a / r.b; }
// Division by a constant b = B 2^e, B odd; everything but the operations on a
// folds at compile time.  B = 1: the exact product with 1 / b.  B < 2^21: the
// product with 1 / b in two parts, ch + cl, rounded once (Brisebarre & Muller,
// IEEE Trans. Comput. 57(2), 2008): it is within 2^-50 of a last place of
// a / b before its rounding, and a / b, a multiple of 2^j / B that is no
// midpoint of two doubles (A / B has no more bits than A), lies at least
// 1 / (2 B) of a last place from every midpoint.  Else the corrected product.
// The two-part product's range of a is div_by's.
GB_HD double cdiv(double a, double b) {
  const uint64_t m = fpi_bits(b) & 0x000fffffffffffffULL;
  const uint32_t h = (uint32_t)(fpi_bits(a) >> 32) & 0x7fffffffu;
  if (m == 0) return a * (1.0 / b);
  if ((m & 0xffffffffULL) == 0) {            // at most 20 bits behind the leading one: B < 2^21
    const double ch = 1.0 / b, cl = fma(-ch, b, 1.0) / b;
    const bool zero = (fpi_bits(a) << 1) == 0;
    if (zero || h - ((1023u - 400u) << 20) < (800u << 20)) {
      const double q = fma(a, ch, a * cl);
      return zero ? a * ch : q;
    }
    return a / b;
  }
  return div_by(a, Recip{b, 1.0 / b, true});
}
GB_HD float cdiv(float a, float b) { return a / b; }
// to<R>(x): an FP64 value in R; up(x): a value of R in FP64
template <typename R> GB_HD R to(double x);
template <> GB_HD double to<double>(double x) { return x; }
template <> GB_HD float to<float>(double x) { return d2f(x); }
GB_HD double up(double x) { return x; }
GB_HD double up(float x) { return f2d(x); }
GB_HD bool mag_gt(double a, double b) { return nn_lt(b, a); }
GB_HD bool mag_gt(float a, float b) { return a > b; }
GB_HD bool mag_lt(double a, double b) { return nn_lt(a, b); }
GB_HD bool mag_lt(float a, float b) { return a < b; }
GB_HD bool is_zero(double x) { return fpi_is_zero(x); }
GB_HD bool is_zero(float x) { return x == 0.0f; }

}  // namespace gbrkc
#endif
