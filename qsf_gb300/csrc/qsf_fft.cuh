// qsf_fft.cuh -- FP64 complex helpers and the radix factorisation of a built length, as
// the plain row transforms take it and qsf_fft_plan_radices reports it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace qsf {

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
// ---------------------------------------------------------------------------
// Compile-time radix plans.  A line of N = 2^a 3^b 5^c points is transformed by
// floor(a/4) radix-16 passes, one radix 2/4/8 pass for the rest of 2^a, then the
// radix-3 and radix-5 passes.  The first pass needs no twiddles, so radix 16 goes
// first.
__host__ __device__ constexpr int count_factor(int n, int f) {
  int c = 0;
  while (n % f == 0) {
    n /= f;
    ++c;
  }
  return c;
}
__host__ __device__ constexpr bool is_smooth(int n) {
  int v = n;
  while (v % 2 == 0) v /= 2;
  while (v % 3 == 0) v /= 3;
  while (v % 5 == 0) v /= 5;
  return v == 1 && n > 1;
}
// log2 of the largest power-of-two radix of the plans (16)
#ifndef QSF_RADIX_LOG2
#define QSF_RADIX_LOG2 4
#endif
// Stage plan of an n-point transform: passes of radix 2^l2 (the main radix), one pass
// of the remaining power of two, then radix-3 and radix-5 passes.
__host__ __device__ constexpr int nstages(int n, int l2 = QSF_RADIX_LOG2) {
  const int a = count_factor(n, 2);
  return a / l2 + (a % l2 ? 1 : 0) + count_factor(n, 3) + count_factor(n, 5);
}
__host__ __device__ constexpr int radix_at(int n, int i, int l2 = QSF_RADIX_LOG2) {
  const int a = count_factor(n, 2);
  const int q = a / l2, r = a % l2;
  if (i < q) return 1 << l2;
  int k = i - q;
  if (r) {
    if (k == 0) return 1 << r;
    k -= 1;
  }
  return k < count_factor(n, 3) ? 3 : 5;
}
__host__ __device__ constexpr int ns_at(int n, int i, int l2 = QSF_RADIX_LOG2) {
  int p = 1;
  for (int j = 0; j < i; ++j) p *= radix_at(n, j, l2);
  return p;
}
}  // namespace qsf
