// The integer and reciprocal forms of csrc/fp_int.cuh on the GPU against the
// GPU's own FP64 instructions: quotients (the reciprocal's seed is the
// device's there), quotients by the kinds of constant that the gating uses,
// conversions, comparisons and the stage count's root.  argv[1]: pairs, in
// millions.
#include <cstdio>
#include <cstdlib>

#include "fp_int.cuh"

using namespace gbrkc;

enum { QUOTIENT, CONSTANT, CONVERT, COMPARE, ROOT, KINDS };

__device__ uint64_t mix(uint64_t x) {
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}
__device__ bool same(double a, double b) { return fpi_bits(a) == fpi_bits(b) || (a != a && b != b); }
__device__ bool samef(float a, float b) { return fpi_fbits(a) == fpi_fbits(b) || (a != a && b != b); }

__global__ void check(unsigned long long pairs, unsigned long long *bad) {
  unsigned n[KINDS] = {};
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < pairs; i += step) {
    const uint64_t u = mix(2 * i), w = mix(2 * i + 1);
    // any bits; magnitudes within 2^60 of one; mantissas near one and two, and short ones
    double a = fpi_double(u), b = fpi_double(w);
    if ((i & 7) >= 2) {
      a = fpi_double((u & 0x800fffffffffffffULL) | ((963 + (u >> 52) % 120) << 52));
      b = fpi_double((w & 0x800fffffffffffffULL) | ((963 + (w >> 52) % 120) << 52));
    }
    if ((i & 7) == 6) b = fpi_double(fpi_bits(b) | 0x000ffffffffffc00ULL);
    if ((i & 7) == 7) b = fpi_double(fpi_bits(b) & 0xfff00000000003ffULL);
    const Recip r = recip(b);
    n[QUOTIENT] += !same(div_by(a, r), a / b) + !same(mdiv(b, a), b / a);
#define GB_C(c) n[CONSTANT] += !same(cdiv(a, c), a / (c));
    GB_C(3.0) GB_C(6.0) GB_C(10.0) GB_C(-12.0) GB_C(0.11) GB_C(0.85) GB_C(12.8433) GB_C(23.32708) GB_C(0.099986667) GB_C(4.0)
#undef GB_C
    const float f = fpi_float((uint32_t)u);
    n[CONVERT] += !samef(d2f(a), (float)a) + !same(f2d(f), (double)f);
    const double p = fabs(a), q = (w & 1) ? fabs(b) : fpi_double(fpi_bits(p) ^ (w & 6));
    n[COMPARE] += (nn_lt(p, q) != (p < q)) + (nn_le(p, q) != (p <= q));
    if (p == p && q == q) n[COMPARE] += !same(abs_max(a, q), p > q ? p : q);
    const double x = fpi_double((u & 0x000fffffffffffffULL) | ((1023 + (w >> 8) % 23) << 52));
    bool ok;
    const int s = int_sqrt(x, ok);
    n[ROOT] += !ok || s != (int)sqrt(x);
  }
  for (int k = 0; k < KINDS; k++)
    if (n[k]) atomicAdd(bad + k, (unsigned long long)n[k]);
}

int main(int argc, char **argv) {
  const unsigned long long pairs = 1000000ull * (argc > 1 ? strtoull(argv[1], nullptr, 10) : 1);
  unsigned long long *d = nullptr, bad[KINDS] = {};
  if (cudaMalloc(&d, sizeof bad) != cudaSuccess || cudaMemset(d, 0, sizeof bad) != cudaSuccess) return 2;
  check<<<1216, 128>>>(pairs, d);
  if (cudaMemcpy(bad, d, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  cudaFree(d);
  unsigned long long all = 0;
  for (int k = 0; k < KINDS; k++) all += bad[k];
  printf("%llu pairs: quotient %llu constant %llu convert %llu compare %llu root %llu\n%s\n", pairs, bad[QUOTIENT],
         bad[CONSTANT], bad[CONVERT], bad[COMPARE], bad[ROOT], all ? "differences" : "all equal");
  return all != 0;
}
