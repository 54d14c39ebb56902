// Exponentials in base 2 from a 64-entry table, for kernels whose time is their exponentials. Each
// translation unit that includes this has its own copy of the table in device memory, filled by
// exp2_tab_setup (outside any stream capture) and read into shared memory by exp2_tab_load.
#pragma once
#include <cmath>

#include "ocfd_device.cuh"

namespace ocfd {
constexpr int E2_N = 64;  // entries of the 2^(j / 64) table
static __device__ double g_exp2_tab[E2_N];

static inline cudaError_t exp2_tab_setup() {
  double tab[E2_N];
  for (int j = 0; j < E2_N; j++) tab[j] = (double)std::exp2((long double)j / E2_N);
  return cudaMemcpyToSymbol(g_exp2_tab, tab, sizeof(tab));
}
// the block's copy (at least E2_N threads, one-dimensional block); the caller synchronises
static __device__ __forceinline__ void exp2_tab_load(double* tab) {
  if (threadIdx.x < E2_N) tab[threadIdx.x] = g_exp2_tab[threadIdx.x];
}
// 2^y by table and polynomial (P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15, 1989): y = n / 64 + r, |r| <= 1 / 128,
// 2^y = 2^(n >> 6) tab[n & 63] 2^r with the Taylor polynomial of degree 5 (remainder 4e-17). Nine
// FP64 operations, 2.8e-16 for -1022 <= y <= 1022; the binary exponent is added as an integer and saturates
// there, so that a smaller result than 2^-1022 is about that and not 0 (|y| < 2^25: beyond it the low word
// wraps). NaN gives NaN, and so do infinities.
__device__ __forceinline__ double exp2_tab(double y, const double* tab) {
  constexpr double MAGIC = 6755399441055744.0;  // 1.5 2^52: the sum's low word is rint(64 y)
  const double t = fma(y, (double)E2_N, MAGIC);
  const double nf = t - MAGIC;
  const double r = fma(nf, -1.0 / E2_N, y);
  const int n = __double2loint(t);
  constexpr double L1 = 0.69314718055994530942;
  constexpr double c1 = L1, c2 = L1 * L1 / 2, c3 = L1 * L1 * L1 / 6, c4 = L1 * L1 * L1 * L1 / 24,
                   c5 = L1 * L1 * L1 * L1 * L1 / 120;
  const double q = fma(r, fma(r, fma(r, fma(r, c5, c4), c3), c2), c1) * r;
  const double tv = tab[n & (E2_N - 1)];
  const int ex = max(min(n >> 6, 1022), -1022);
  const double s = __hiloint2double(__double2hiint(tv) + (ex << 20), __double2loint(tv));
  return fma(s, q, s);
}
}  // namespace ocfd
