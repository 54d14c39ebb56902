// Fitted mixture transport (Wilke viscosity and conductivity, mixture-averaged diffusion) for
// N_SPEC > 1, in its own translation unit: comput_Amu_Amk_AMD with Flag_vis = Flag_cond = Flag_diff
// = 1 (Comput_flow_variables.f90:69-98; comput_vis_coeff, comput_thermal_conductivity,
// comput_diffusion_coeff of TRANSPORT_modules.f90:259-426). Other flag combinations keep
// k_transport (ocfd_flow.cuh).
#include <cmath>
#include <cstddef>
#include <stdexcept>

#include "ocfd_device.cuh"
#include "ocfd_exp2.cuh"
#include "ocfd_launch.h"

namespace ocfd {

// ---------------------------------------------------------------- constants of the fits
constexpr int TF_NS = 9, TF_NP = TF_NS * (TF_NS - 1) / 2;
struct TransFit {
  // base-2 exponents of sqrt(mu_k), kappa_k and 1 / D_ab as cubics in ln T (the unit factors of the
  // fits folded into the constant term); pairs (a, b), a < b, enumerated a-major
  double mu[TF_NS][4], kap[TF_NS][4], dif[TF_NP][4];
  // Wilke's sum over j as a quadratic in sqrt(mu_k): X_j phi_kj = X_j (1 + s_k c_kj / s_j)^2 / b_kj
  double wa[TF_NS][TF_NS], wb[TF_NS][TF_NS], wc[TF_NS][TF_NS];
  double rMi[TF_NS];
};
__constant__ TransFit cF;

// Fills the constants for the current set-up; called by ocfd_gpu_init, outside any capture.
cudaError_t transport_fit_setup(const DevConst& c, int ns) {
  if (ns < 2 || ns > TF_NS) return cudaSuccess;
  TransFit t{};
  const long double log2e = 1.0L / std::log(2.0L);
  int np = 0;
  for (int k = 0; k < ns; k++) {
    for (int m = 0; m < 4; m++) {
      t.mu[k][m] = (double)(0.5L * log2e * c.mu_an[k][m] + (m == 0 ? 0.5L * std::log2(0.1L) : 0.0L));
      t.kap[k][m] = (double)(log2e * c.k_an[k][m] + (m == 0 ? std::log2(1.0e-5L) : 0.0L));
    }
    for (int j = 0; j < ns; j++) {
      // phi_kj = (1 + s_k / s_j cc)^2 / b with cc = (M_j / M_k)^(1/4), b = sqrt(8 (1 + M_k / M_j))
      const long double cc = std::sqrt(std::sqrt((long double)c.Mi[j] / c.Mi[k]));
      const long double bi = 1.0L / std::sqrt(8.0L * (1.0L + (long double)c.Mi[k] / c.Mi[j]));
      t.wa[k][j] = (double)bi;
      t.wb[k][j] = (double)(2.0L * cc * bi);
      t.wc[k][j] = (double)(cc * cc * bi);
    }
    for (int b = k + 1; b < ns; b++, np++)
      for (int m = 0; m < 4; m++)
        t.dif[np][m] = (double)(-log2e * c.d_an[k][b][m] + (m == 0 ? std::log2(1.0e4L) : 0.0L));
    t.rMi[k] = 1.0 / c.Mi[k];
  }
  const cudaError_t e = cudaMemcpyToSymbol(cF, &t, sizeof(t));
  return e != cudaSuccess ? e : exp2_tab_setup();
}

// ocfd_gpu_chem_setup on an open flow solver replaces the masses of the mole fractions; the fits and the
// pair constants stay those of ocfd_gpu_init, as in k_transport.
cudaError_t transport_fit_masses(const DevConst& c, int ns) {
  if (ns < 2 || ns > TF_NS) return cudaSuccess;
  double r[TF_NS] = {};
  for (int k = 0; k < ns; k++) r[k] = 1.0 / c.Mi[k];
  return cudaMemcpyToSymbol(cF, r, sizeof(r), offsetof(TransFit, rMi));
}

// ---------------------------------------------------------------- arithmetic
__device__ __forceinline__ double cubic(const double* c, double L) {
  return fma(fma(fma(c[3], L, c[2]), L, c[1]), L, c[0]);
}

// One thread per cell: everything that depends on the cell alone (ln T, mole fractions, 1 / p) is
// formed once, every coefficient is an operand from constant memory, and the species' values stay in
// registers, so the kernel is bound by its FP64 operations (about 1300 per cell at 9 species: 54
// exponentials of 12, the Wilke quadratics 243). The form it replaces spread a cell over one thread
// per species with nine barriers' worth of shared-memory exchange: 9250 issued instructions per cell,
// 2400 of them FP64, at 27 % of the FP64 pipe. Measured on 384x256x32 cells, 9 species (contracted
// build): 1.540 -> 0.294 ms per launch, three quarters of the FP64 pipe; 97x61x43: 0.140 -> 0.033.
// 128 threads x 4 blocks leave 128 registers, which hold it without spills.
#ifndef OCFD_TFIT_THREADS
#define OCFD_TFIT_THREADS 128
#endif
#ifndef OCFD_TFIT_MINB
#define OCFD_TFIT_MINB 4
#endif
template <int NS>
__global__ void __launch_bounds__(OCFD_TFIT_THREADS, OCFD_TFIT_MINB)
    k_transport_fit(const double* __restrict__ T, const double* __restrict__ p, const double* __restrict__ di,
                    double* __restrict__ amu, double* __restrict__ amk, double* __restrict__ amd) {
  __shared__ double tab[E2_N];
  exp2_tab_load(tab);
  __syncthreads();
  const unsigned t = blockIdx.x * OCFD_TFIT_THREADS + threadIdx.x;
  if (t >= (unsigned)cC.N) return;
  const unsigned nx = (unsigned)cC.nx, ny = (unsigned)cC.ny;
  const unsigned jk = fast_div(t, nx, cC.mx, cC.sx), k0 = fast_div(jk, ny, cC.my, cC.sy);
  const int q = hidx((int)(t - jk * nx) + 1, (int)(jk - k0 * ny) + 1, (int)k0 + 1);
  const double Lt = log(T[q]);
  const double rp = rcp3(p[q]) * 1.013e5;
  double X[NS];
  double X0 = 0.0;
#pragma unroll
  for (int m = 0; m < NS; m++) {
    X[m] = __dmul_rn(di[(size_t)m * cC.H + q], cF.rMi[m]);
    X0 += X[m];
  }
  // Mole numbers take the mole fractions' place; their sum X0 enters where it does not cancel. Thereby
  // 1 - X_k is (X0 - X[k]) / X0, which is 0 where a species is alone, as with the reference's quotient; a
  // rounded product with 1 / X0 would leave one unit in the last place there, to be divided by 1e-20. (Of
  // rounded products, not contracted: X0 then equals X[k] beside traces below its last place as well.)
  // diffusion: ds_k = sum over j != k of X_j / D_kj, every pair's exponential once
  double ds[NS];
#pragma unroll
  for (int m = 0; m < NS; m++) ds[m] = 1.0e-20 * X0;
  {
    int np = 0;
#pragma unroll
    for (int a = 0; a < NS; a++)
#pragma unroll
      for (int b = a + 1; b < NS; b++, np++) {
        const double rD = exp2_tab(cubic(cF.dif[np], Lt), tab);
        ds[a] = fma(X[b], rD, ds[a]);
        ds[b] = fma(X[a], rD, ds[b]);
      }
  }
#pragma unroll
  for (int m = 0; m < NS; m++) amd[(size_t)m * cC.N + t] = (X0 - X[m]) * rp * rcp3(ds[m]);
  // conductivity: mean of the arithmetic and harmonic means
  {
    double a1 = 0.0, a2 = 0.0;
#pragma unroll
    for (int m = 0; m < NS; m++) {
      const double kk = exp2_tab(cubic(cF.kap[m], Lt), tab);
      a1 = fma(X[m], kk, a1);
      a2 = fma(X[m], rcp3(kk), a2);
    }
    amk[t] = 0.5 * fma(a1, rcp3(X0), X0 * rcp3(a2));
  }
  // viscosity: mu = sum_k X_k mu_k / sum_j X_j phi_kj
  double s[NS], Y[NS], Z[NS];  // sqrt(mu_k), X_k / s_k, X_k / mu_k
#pragma unroll
  for (int m = 0; m < NS; m++) {
    s[m] = exp2_tab(cubic(cF.mu[m], Lt), tab);
    const double r = rcp3(s[m]);
    Y[m] = X[m] * r;
    Z[m] = Y[m] * r;
  }
  double mu = 0.0;
#pragma unroll
  for (int k = 0; k < NS; k++) {
    double A = 0.0, B = 0.0, C = 0.0;
#pragma unroll
    for (int j = 0; j < NS; j++) {
      A = fma(cF.wa[k][j], X[j], A);
      B = fma(cF.wb[k][j], Y[j], B);
      C = fma(cF.wc[k][j], Z[j], C);
    }
    mu = fma(X[k] * (s[k] * s[k]), rcp3(fma(s[k], fma(s[k], C, B), A)), mu);
  }
  amu[t] = mu;
}

void launch_transport_fit(int ns, long long N, const double* T, const double* p, const double* di, double* amu,
                          double* amk, double* amd, cudaStream_t st) {
  const unsigned nb = (unsigned)((N + OCFD_TFIT_THREADS - 1) / OCFD_TFIT_THREADS);
#define TF(n) case n: k_transport_fit<n><<<nb, OCFD_TFIT_THREADS, 0, st>>>(T, p, di, amu, amk, amd); break;
  switch (ns) {
    TF(2) TF(3) TF(4) TF(5) TF(6) TF(7) TF(8) TF(9)
    default: throw std::runtime_error("N_SPEC must be 2..9");
  }
#undef TF
}
}  // namespace ocfd
