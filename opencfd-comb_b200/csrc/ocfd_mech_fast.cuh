// Linearised implicit Euler (CHEM_reactions.f90:473-567) of the compiled 9-species H2-air mechanism
// in the contracted build: the step of chem_step<9, ..., MECH_H2AIR9> with the matrix in registers.
// Differs from it by rounding only:
//  - T(E) starts its Newton iteration from the previous sub-step's temperature and evaluates the
//    range's summed polynomials by Horner's rule (the same convergence test, 1e-3 K, after which the
//    quadratic iteration is at rounding level);
//  - the reverse rates come from the equilibrium constants as products of 2^(F_i), F_i the Gibbs
//    potential of species i over T less that of its elements in H2 and O2 (which cancels in every
//    reaction), instead of one exponential and one division per reaction;
//  - the linear system is in moles (a diagonal similarity of the reference's mass form), the inert
//    N2 drops out, and the elimination is unpivoted in registers. A lane whose elimination met a
//    multiplier above MULT_MAX repeats it with partial pivoting (pivoted_step).
// Above the fits' last temperature the reference continues with a constant heat capacity; that is one
// more fit range here, so that hot reactors, and Newton's first guesses beyond it, take the same path.
// What is left, T below T_MIN or no T(E), takes the sub-step of chem_step<9, ..., MECH_H2AIR9>, its
// matrix in the block's shared memory.
// Bound by FP64 issue and its latency at eight warps per SM (254 registers with its callees, half of them the
// 8 x 8 matrix; the rates of progress wait in shared memory until it is assembled, so the two phases'
// values are not live together). About 1500 FP64 operations per sub-step against some 3500 with the
// matrix in shared memory, 42 equilibrium and rate exponentials of 20, and a division per pivot row.
// Measured against that form (k_chem_batch): 2^20 reactors with 22 sub-steps on average 20.9 -> 4.51 ms
// (0.88 -> 0.19 ns per sub-step), 60,001 at constant pressure 4.11 -> 0.90 ms, the cells of the
// 384x256x32 jet 3.19 -> 0.72 ms per step. 777 reactors on host arrays, up to a hundred sub-steps in a row
// on one thread each, whole call 3.8 -> 0.58 ms: the step's latency is below the cooperative kernel's, so
// batches of every size come here. 2^18 reactors, 20 sub-steps, at 300-400 K / 100-148 K / steam at
// 2500-4000 K / products at 5100-6500 K: 4.90 / 4.90 / 5.06 / 5.75 -> 1.24 / 1.25 / 1.30 / 1.37 ms. With steps
// so long that densities overshoot below zero (1e-7 s, a hundredth of radicals) 1.15 -> 0.57, with one
// reactor in sixty lost (1e-6 s) 2.28 -> 2.06. Below T_MIN the step is the same and slower than in its own
// kernel (85-99 K, one lane in three: 4.90 -> 7.9).
#pragma once
#include "ocfd_chem.cuh"
#include "ocfd_exp2.cuh"

#if OCFD_FMA_BUILD
#include <utility>

namespace ocfd {
namespace mech_fast {
using mech_h2air9::AF_TYPE;
using mech_h2air9::NR;
using mech_h2air9::NS;
using mech_h2air9::TR_REAC;
using mech_h2air9::VF;
using mech_h2air9::VR;
constexpr int NA = NS - 1;  // reacting species: all but the last (N2)
constexpr int NRG = OCFD_NTCT_MAX + 1;  // fit ranges, and the one above the last temperature
// Below T_MIN the partial products of 2^(F_i) and a rate may leave the exponent range: with the shipped
// tables they stay within 2^-888 and 2^456 at 90 K, which leaves 2^-134 to the concentrations.
constexpr double T_MIN = 90.0;
constexpr double MULT_MAX = 16.0;  // largest elimination multiplier taken without pivoting

constexpr bool inert_last() {
  for (int j = 0; j < NR; j++)
    if (VF[j][NS - 1] != 0 || VR[j][NS - 1] != 0) return false;
  return true;
}
static_assert(inert_last(), "the last species takes part in no reaction");
// O and H atoms of the species in the order that fast_step's potentials assume: O, O2, H2, H2O, OH, H, HO2, H2O2
constexpr int ATOMS[NA][2] = {{1, 0}, {2, 0}, {0, 2}, {1, 2}, {1, 1}, {0, 1}, {2, 1}, {2, 2}};
constexpr bool conserves_atoms() {
  for (int j = 0; j < NR; j++)
    for (int e = 0; e < 2; e++) {
      int t = 0;
      for (int i = 0; i < NA; i++) t += (VR[j][i] - VF[j][i]) * ATOMS[i][e];
      if (t != 0) return false;
    }
  return true;
}
static_assert(conserves_atoms(), "the elements' potentials cancel in every reaction");

struct Fast {
  // by fit range, so that the range in use is one stretch of the constant cache
  double e6[NRG][NS][6];  // internal energy of species k per density: R (c0-1), R c1/2, ..., R c4/5, R Ect
  double g2[NRG][NA][7];  // log2(e) times: c0, -c1/2, -c2/6, -c3/12, -c4/20, c5, -c6
  double bf2[NR][2], ef2[NR][2];  // log2(e) times the Arrhenius exponents
  double troe[NR][3];            // log10 Fc, ac, an
  double rM6[NS], M6[NS], RF[NS];  // 1e-6 / M, 1e6 M, R c5 (the formation term of update_Et)
  double rs;                     // R0 / p0 1e6 of the equilibrium constants
};
__constant__ Fast cM;

static inline cudaError_t setup(const DevConst& c) {
  Fast f{};
  const long double l2e = 1.0L / std::log(2.0L);
  for (int k = 0; k < NS; k++) {
    for (int j = 0; j < c.n_tct; j++) {
      const double* a = c.cf[k][j];
      f.e6[j][k][0] = (double)(((long double)a[0] - 1.0L) * c.Ri[k]);
      for (int m = 1; m < 5; m++) f.e6[j][k][m] = (double)((long double)a[m] * c.Ri[k] / (m + 1));
      f.e6[j][k][5] = (double)((long double)a[7] * c.Ri[k]);
      if (k < NA) {
        const long double w[7] = {1.0L, -1.0L / 2, -1.0L / 6, -1.0L / 12, -1.0L / 20, 1.0L, -1.0L};
        for (int m = 0; m < 7; m++) f.g2[j][k][m] = (double)(l2e * w[m] * a[m]);
      }
    }
    // e = e(tm) + cv(tm) (T - tm) and g = h(tm) + cp(tm) (T - tm) - T (s(tm) + cp(tm) ln(T / tm))
    // (dev_E, dev_gibbs) as a range with c0 alone
    const double* a = c.cf[k][c.n_tct - 1];
    const long double tm = c.tct_max, t2 = tm * tm, t3 = t2 * tm, t4 = t2 * t2, t5 = t4 * tm, l = std::log(tm);
    const long double cp = a[0] + a[1] * tm + a[2] * t2 + a[3] * t3 + a[4] * t4;
    const long double h = a[0] * tm + a[1] * t2 / 2 + a[2] * t3 / 3 + a[3] * t4 / 4 + a[4] * t5 / 5;
    const long double sm = a[0] * l + a[1] * tm + a[2] * t2 / 2 + a[3] * t3 / 3 + a[4] * t4 / 4 + a[6];
    f.e6[c.n_tct][k][0] = (double)((cp - 1.0L) * c.Ri[k]);
    f.e6[c.n_tct][k][5] = (double)((h - cp * tm + a[7]) * c.Ri[k]);
    if (c.realgas == 0)  // e = 5/2 R T at any temperature; the equilibrium constants keep the fits
      for (int j = 0; j < NRG; j++)
        for (int m = 0; m < 6; m++) f.e6[j][k][m] = m == 0 ? 2.5 * c.Ri[k] : 0.0;
    if (k < NA) {
      f.g2[c.n_tct][k][0] = (double)(l2e * cp);
      f.g2[c.n_tct][k][5] = (double)(l2e * (h + a[5] - cp * tm));
      f.g2[c.n_tct][k][6] = (double)(-l2e * (sm - cp * l));
    }
  }
  for (int j = 0; j < NR; j++) {
    for (int s = 0; s < 2; s++) {
      f.bf2[j][s] = (double)(l2e * c.bf[j][s]);
      f.ef2[j][s] = (double)(l2e * c.ef[j][s]);
    }
    if (AF_TYPE[j] == 1) {
      const double lfc = std::log10(c.fc_troe[j]);
      f.troe[j][0] = lfc;
      f.troe[j][1] = -0.4 - (double)0.67f * lfc;
      f.troe[j][2] = 0.75 - (double)1.27f * lfc;
    }
  }
  for (int k = 0; k < NS; k++) {
    f.rM6[k] = (double)(1.0e-6L / c.Mi[k]);
    f.M6[k] = c.Mi[k] * 1.0e6;
    f.RF[k] = c.Ri[k] * c.cf[k][0][5];
  }
  f.rs = 8.314 / 1.013e5 * 1.0e6;
  const cudaError_t e = cudaMemcpyToSymbol(cM, &f, sizeof(f));
  return e != cudaSuccess ? e : exp2_tab_setup();
}

// compile-time loops
template <int... I, class F>
__device__ __forceinline__ void sfor_(std::integer_sequence<int, I...>, F&& f) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void sfor(F&& f) {
  sfor_(std::make_integer_sequence<int, N>{}, f);
}

// fit range of T, the constant heat capacity above the last one included
__device__ __forceinline__ int range_of(double T) { return T > cC.tct_max ? cC.n_tct : trange(T); }
// energy polynomial of densities (or mass fractions) d in fit range j
struct EnergyPoly {
  double a[6];
  __device__ __forceinline__ EnergyPoly(const double* d, int j) {
#pragma unroll
    for (int m = 0; m < 6; m++) a[m] = 0.0;
#pragma unroll
    for (int k = 0; k < NS; k++)
#pragma unroll
      for (int m = 0; m < 6; m++) a[m] = fma(cM.e6[j][k][m], d[k], a[m]);
  }
  __device__ __forceinline__ double e(double T) const {
    return fma(T, fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]), a[5]);
  }
  __device__ __forceinline__ double cv(double T) const {
    return fma(T, fma(T, fma(T, fma(T, 5.0 * a[4], 4.0 * a[3]), 3.0 * a[2]), 2.0 * a[1]), a[0]);
  }
};
// a density (or mass fraction) below zero by more than a millionth of the whole: e(T) may then have several
// roots, and which one is found depends on the first guess
__device__ __forceinline__ bool negative(const double* d) {
  int sign = 0;
#pragma unroll
  for (int k = 0; k < NS; k++) sign |= __double2hiint(d[k]);
  if (sign >= 0) return false;
  double rho = 0.0, lo = 0.0;
#pragma unroll
  for (int k = 0; k < NS; k++) {
    rho += d[k];
    lo = fmin(lo, d[k]);
  }
  return !(lo >= -1.0e-6 * rho);
}
// T(E) from the starting value T, or from the reference's first guess when that is not positive or
// densities are negative; false when the iteration left the positive temperatures or did not converge
__device__ __forceinline__ bool newton_T(const double* d, double E, double& T) {
  if (negative(d)) T = 0.0;
  int jc = range_of(T);
  EnergyPoly P(d, jc);
  if (!(T > 0.0)) T = E / P.a[0];  // jc = 0
  bool ok = false;
  for (int it = 0; it <= 30 && T > 0.0; it++) {
    const int j = range_of(T);
    if (j != jc) { jc = j; P = EnergyPoly(d, j); }
    const double dT = (P.e(T) - E) * rcp3(P.cv(T));
    T = T - dT;
    if (fabs(dT) < 1.0e-3) {
      ok = T > 0.0;
      break;
    }
  }
  return ok;
}

// the pivoted step of one lane (rare), its matrix in the lane's column of shared memory: returns its
// zero-pivot flag
template <int TPB>
__device__ __noinline__ bool general_step(double* di, double& E, double dt, int* nfail, double* sp) {
  double d[NS], e = E;
#pragma unroll
  for (int i = 0; i < NS; i++) d[i] = di[i];
  const bool z = chem_step<NS, TPB, MECH_H2AIR9>(d, e, dt, nfail, Slab<TPB>{sp});
#pragma unroll
  for (int i = 0; i < NS; i++) di[i] = d[i];
  E = e;
  return z;
}

// I - dt J in moles and the right-hand side dt r from the rates of progress in sp
template <int TPB>
__device__ __forceinline__ void assemble(const double* c, double dt, const double* sp, double (&A)[NA][NA],
                                         double* b) {
  double rc[NA];
#pragma unroll
  for (int i = 0; i < NA; i++) {
    b[i] = 0.0;
    rc[i] = rcp3(c[i] + 1.0e-20) * dt;
#pragma unroll
    for (int j = 0; j < NA; j++) A[i][j] = i == j ? 1.0 : 0.0;
  }
  sfor<NR>([&](auto K) {
    constexpr int k = decltype(K)::value;
    const double fw = sp[(2 * k) * TPB], bw = sp[(2 * k + 1) * TPB];
    const double net = fw - bw;
    sfor<NA>([&](auto J) {
      constexpr int j = decltype(J)::value, a = VF[k][j], bb = VR[k][j], s = bb - a;
      if constexpr (s != 0) b[j] = fma((double)s, net, b[j]);
      if constexpr (a != 0 || bb != 0) {
        double dA;
        if constexpr (bb == 0) dA = (double)a * fw * rc[j];
        else if constexpr (a == 0) dA = -(double)bb * bw * rc[j];
        else dA = ((double)a * fw - (double)bb * bw) * rc[j];
        sfor<NA>([&](auto I) {
          constexpr int i = decltype(I)::value, si = VR[k][i] - VF[k][i];
          if constexpr (si != 0) A[i][j] = fma(-(double)si, dA, A[i][j]);
        });
      }
    });
  });
#pragma unroll
  for (int i = 0; i < NA; i++) b[i] *= dt;
}
// the solution from the eliminated system, the reciprocals of the pivots on the diagonal
__device__ __forceinline__ void back_substitute(const double (&A)[NA][NA], double* b) {
#pragma unroll
  for (int i = NA - 1; i >= 0; i--) {
    double s = b[i];
#pragma unroll
    for (int j = i + 1; j < NA; j++) s = fma(-A[i][j], b[j], s);
    b[i] = s * A[i][i];
  }
}
__device__ __forceinline__ void update(double* di, double& E, const double* b) {
#pragma unroll
  for (int i = 0; i < NA; i++) {
    const double dd = cM.M6[i] * b[i];
    di[i] = di[i] + dd;
    E = fma(-dd, cM.RF[i], E);
  }
}
// a and b change places where on is set (of their words, so that the rows stay registers)
__device__ __forceinline__ void exchange(bool on, double& a, double& b) {
  const int ah = __double2hiint(a), al = __double2loint(a), bh = __double2hiint(b), bl = __double2loint(b);
  a = __hiloint2double(on ? bh : ah, on ? bl : al);
  b = __hiloint2double(on ? ah : bh, on ? al : bl);
}
// the step of a lane whose elimination needs pivots, from the rates that fast_step left in sp: partial
// pivoting with the rows in registers, swapped by selects. Returns the zero-pivot flag.
template <int TPB>
__device__ __noinline__ bool pivoted_step(double* di, double& E, double dt, const double* sp) {
  double d[NS], c[NA], A[NA][NA], b[NA], e = E;
#pragma unroll
  for (int i = 0; i < NA; i++) {
    d[i] = di[i];
    c[i] = d[i] * cM.rM6[i];
  }
  assemble<TPB>(c, dt, sp, A, b);
  bool zero = false;
  sfor<NA>([&](auto K) {
    constexpr int k = decltype(K)::value;
    double most = fabs(A[k][k]);
    int kk = k;
    sfor<NA - 1 - k>([&](auto I) {
      constexpr int i = k + 1 + decltype(I)::value;
      const double v = fabs(A[i][k]);
      kk = v > most ? i : kk;
      most = v > most ? v : most;
    });
    zero = zero || most == 0.0;
    sfor<NA - 1 - k>([&](auto I) {
      constexpr int i = k + 1 + decltype(I)::value;
      sfor<NA - k>([&](auto J) {
        constexpr int j = k + decltype(J)::value;
        exchange(kk == i, A[k][j], A[i][j]);
      });
      exchange(kk == i, b[k], b[i]);
    });
    const double rp = rcp3(A[k][k]);
    sfor<NA - 1 - k>([&](auto I) {
      constexpr int i = k + 1 + decltype(I)::value;
      const double f = A[i][k] * rp;
      sfor<NA - 1 - k>([&](auto J) {
        constexpr int j = k + 1 + decltype(J)::value;
        A[i][j] = fma(-f, A[k][j], A[i][j]);
      });
      b[i] = fma(-f, b[k], b[i]);
    });
    A[k][k] = rp;
  });
  back_substitute(A, b);
  update(d, e, b);
#pragma unroll
  for (int i = 0; i < NA; i++) di[i] = d[i];
  E = e;
  return zero;
}

// The linearised step at temperature T in moles; false, with di and E as they were, when the elimination
// needs pivots. sp, tab: as in step.
template <int TPB>
__device__ __forceinline__ bool fast_step(double* di, double& E, double dt, double T, double* sp, const double* tab) {
  double c[NS];
#pragma unroll
  for (int i = 0; i < NS; i++) c[i] = di[i] * cM.rM6[i];
  {
    const double lt = log(T), rT = rcp3(T);
    // 2^(F_i) of O, H2O, OH, H, HO2, H2O2 (species 0, 3, 4, 5, 6, 7; O2 is 1, H2 is 2)
    double G[NA], e[NA], r[NA];
    {
      const int jc = range_of(T);
      const double l1 = 1.0 - lt;
#pragma unroll
      for (int i = 0; i < NA; i++) {
        const double* g = cM.g2[jc][i];
        G[i] = fma(T, fma(T, fma(T, fma(T, g[4], g[3]), g[2]), g[1]), fma(g[0], l1, fma(g[5], rT, g[6])));
      }
    }
    const double gO = 0.5 * G[1], gH = 0.5 * G[2];
    e[1] = e[2] = r[1] = r[2] = 1.0;
    e[0] = exp2_tab(G[0] - gO, tab);
    e[3] = exp2_tab(G[3] - gO - G[2], tab);
    e[4] = exp2_tab(G[4] - gO - gH, tab);
    e[5] = exp2_tab(G[5] - gH, tab);
    e[6] = exp2_tab(G[6] - G[1] - gH, tab);
    e[7] = exp2_tab(G[7] - G[1] - G[2], tab);
    r[0] = rcp3(e[0]); r[3] = rcp3(e[3]); r[4] = rcp3(e[4]); r[5] = rcp3(e[5]); r[6] = rcp3(e[6]); r[7] = rcp3(e[7]);
    const double rsT = cM.rs * T, rrsT = rcp3(rsT);
    sfor<NR>([&](auto K) {
      constexpr int k = decltype(K)::value;
      double M = 0.0;
      if constexpr (TR_REAC[k] == 1) {
#pragma unroll
        for (int i = 0; i < NS; i++) M = fma(c[i], cC.treff[k][i], M);
      }
      double w = cC.af[k][0] * exp2_tab(fma(cM.bf2[k][0], lt, -cM.ef2[k][0] * rT), tab);
      if constexpr (AF_TYPE[k] != 0) {
        const double w2 = cC.af[k][1] * exp2_tab(fma(cM.bf2[k][1], lt, -cM.ef2[k][1] * rT), tab);
        if constexpr (AF_TYPE[k] == 2) {
          w = w + w2;
        } else {  // Troe fall-off
          const double Prs = w / w2 * M;
          const double lp = log10(Prs) + cM.troe[k][1];
          const double q = lp / fma(-0.14, lp, cM.troe[k][2]);
          w = w2 * Prs / (1.0 + Prs) * exp2_tab(3.3219280948873623479 * cM.troe[k][0] / fma(q, q, 1.0), tab);
        }
      }
      if constexpr (TR_REAC[k] == 1 && AF_TYPE[k] != 1) w *= M;
      double fw = w, bw = w;
      sfor<NA>([&](auto I) {
        constexpr int i = decltype(I)::value, a = VF[k][i], b = VR[k][i], s = b - a;
        if constexpr (a >= 1) fw *= c[i];
        if constexpr (a >= 2) fw *= c[i];
        if constexpr (b >= 1) bw *= c[i];
        if constexpr (b >= 2) bw *= c[i];
        static_assert(a <= 2 && b <= 2, "stoichiometric coefficients up to 2");
        if constexpr (i != 1 && i != 2) {
          if constexpr (s >= 1) bw *= e[i];
          if constexpr (s >= 2) bw *= e[i];
          if constexpr (s <= -1) bw *= r[i];
          if constexpr (s <= -2) bw *= r[i];
        }
      });
      constexpr int sg = [] {
        int t = 0;
        for (int i = 0; i < NS; i++) t += VR[k][i] - VF[k][i];
        return t;
      }();
      static_assert(sg >= -1 && sg <= 1, "change of moles");
      if constexpr (sg == 1) bw *= rsT;
      if constexpr (sg == -1) bw *= rrsT;
      sp[(2 * k) * TPB] = fw;
      sp[(2 * k + 1) * TPB] = bw;
    });
  }
  double A[NA][NA], b[NA];
  assemble<TPB>(c, dt, sp, A, b);
  // elimination; the multipliers' magnitudes are compared by their high words
  unsigned mx = 0;
#pragma unroll
  for (int k = 0; k < NA - 1; k++) {
    const double rp = rcp3(A[k][k]);
#pragma unroll
    for (int i = k + 1; i < NA; i++) {
      const double f = A[i][k] * rp;
      mx = max(mx, (unsigned)__double2hiint(f) & 0x7fffffffu);
#pragma unroll
      for (int j = k + 1; j < NA; j++) A[i][j] = fma(-f, A[k][j], A[i][j]);
      b[i] = fma(-f, b[k], b[i]);
    }
    A[k][k] = rp;
  }
  A[NA - 1][NA - 1] = rcp3(A[NA - 1][NA - 1]);
  back_substitute(A, b);
  // NaN and infinity have the largest high words: they take the general step as well
  mx = max(mx, (unsigned)__double2hiint(A[NA - 1][NA - 1]) & 0x7fffffffu);
  if (mx > (unsigned)__double2hiint(MULT_MAX)) return false;
  update(di, E, b);
  return true;
}

// One sub-step. T: starting value in, temperature of the old state out. sp: the thread's column of
// SP_WORDS in shared memory (stride TPB), 2 NR rates of progress or the general step's matrix; tab: the
// exponential table; lanes: the mask of the lanes that take it.
constexpr int SP_WORDS = 2 * NR > NS * NS ? 2 * NR : NS * NS;
template <int TPB>
__device__ __forceinline__ bool step(unsigned lanes, double* di, double& E, double dt, double& T, int* nfail,
                                     double* sp, const double* tab) {
  // the lanes that take the step run its parts together: without the two barriers those of a rare path
  // and the others went on to their next sub-steps apart
  bool general = !newton_T(di, E, T), pivots = false, zero = false;
  if (general) T = 0.0;  // the next sub-step starts afresh
  general = general || T < T_MIN;
  __syncwarp(lanes);
  if (!general) pivots = !fast_step<TPB>(di, E, dt, T, sp, tab);
  __syncwarp(lanes);
  if (general || pivots) {  // by way of copies: di stays in registers
    double d1[NS], e1 = E;
#pragma unroll
    for (int i = 0; i < NS; i++) d1[i] = di[i];
    if (general) zero = general_step<TPB>(d1, e1, dt, nfail, sp);
    else zero = pivoted_step<TPB>(d1, e1, dt, sp);
#pragma unroll
    for (int i = 0; i < NS; i++) di[i] = d1[i];
    E = e1;
  }
  return zero;
}
// cp_restore from the sub-step's temperature
__device__ __forceinline__ void restore_p(double* di, double& E, double h0, double p0, double& T, int* nfail) {
  double rho = 0.0, Y[NS], R1 = 0.0, cf = 0.0, t = T;
#pragma unroll
  for (int k = 0; k < NS; k++) rho += di[k];
  const double rr = rcp3(rho);
#pragma unroll
  for (int k = 0; k < NS; k++) {
    Y[k] = di[k] * rr;
    R1 = fma(cC.Ri[k], Y[k], R1);
    cf = fma(cM.RF[k], Y[k], cf);
  }
  // the root in T is one for E > 0 and densities that are not negative; else the reference's way to it
  bool ok = E > 0.0;
  if (negative(Y)) t = 0.0;
  if (ok && !(t > 0.0)) ok = newton_T(di, E, t);
  if (ok) {
    int jc = range_of(t);
    EnergyPoly P(Y, jc);
    ok = false;
    for (int it = 0; it < 50; it++) {
      const int j = range_of(t);
      if (j != jc) { jc = j; P = EnergyPoly(Y, j); }
      const double dT = (P.e(t) + fma(R1, t, cf - h0)) * rcp3(P.cv(t) + R1);
      t = t - dT;
      if (!(t > 0.0)) break;
      if (fabs(dT) <= 1.0e-10 * t) { ok = true; break; }
    }
    if (ok) {
      const double r1 = p0 / (R1 * t);
      const int j = range_of(t);
      if (j != jc) P = EnergyPoly(Y, j);
      E = P.e(t) * r1;
#pragma unroll
      for (int k = 0; k < NS; k++) di[k] = Y[k] * r1;
      T = t;
    }
  }
  if (!ok) {
    cp_restore<NS>(di, E, h0, p0, nfail);
    T = 0.0;
  }
}

constexpr int TPB = 64;
#ifndef OCFD_MECHF_MINB
#define OCFD_MECHF_MINB 4
#endif
// Chemical_time_advance x nsub + comput_T_P on the flow cells (k_chem_cells)
__global__ void __launch_bounds__(TPB, OCFD_MECHF_MINB)
    k_cells(double* f, double* Et, double* T, double* p, double* di, double dt2, int nsub, int* nfail) {
  __shared__ double tab[E2_N], sp[SP_WORDS * TPB];
  exp2_tab_load(tab);
  __syncthreads();
  const unsigned t = blockIdx.x * TPB + threadIdx.x;
  const unsigned lanes = __ballot_sync(0xffffffffu, t < (unsigned)cC.N);
  if (t >= (unsigned)cC.N) return;
  const unsigned nx = (unsigned)cC.nx, ny = (unsigned)cC.ny;
  const unsigned jk = fast_div(t, nx, cC.mx, cC.sx), k = fast_div(jk, ny, cC.my, cC.sy);
  const int q = hidx((int)(t - jk * nx) + 1, (int)(jk - k * ny) + 1, (int)k + 1);
  double d[NS];
#pragma unroll
  for (int m = 0; m < NS; m++) d[m] = di[(size_t)m * cC.H + q];
  double e = Et[q], f5 = f[4 * cC.N + t], TT = T[q];
  bool zero = false;
  for (int s = 0; s < nsub; s++) {
    const double e0 = e;
    zero = step<TPB>(lanes, d, e, dt2, TT, nfail, sp + threadIdx.x, tab) || zero;
    f5 = f5 + (e - e0);
  }
  chem_check<NS>(d, e, zero, nfail);
#pragma unroll
  for (int m = 0; m < NS; m++) di[(size_t)m * cC.H + q] = d[m];
  Et[q] = e;
  f[4 * cC.N + t] = f5;
  if (!newton_T(d, e, TT)) TT = dev_T<NS>(d, e, nfail);
  T[q] = TT;
  p[q] = dev_P<NS>(d, TT);
}
// independent reactors as a work queue (k_chem_batch)
template <bool CP>
__global__ void __launch_bounds__(TPB, OCFD_MECHF_MINB)
    k_batch(int n, double* di, double* e, const double* dt, const int* nsub, const int* perm, int* counter, int* nfail) {
  __shared__ double tab[E2_N], sp[SP_WORDS * TPB];
  exp2_tab_load(tab);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (;;) {
    int base = 0;
    if (lane == 0) base = atomicAdd(counter, 32);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n) break;
    const int idx = base + lane;
    const int r = idx < n ? perm[idx] : -1;
    const int ks = r < 0 ? 0 : (nsub ? nsub[r] : 1);
    double d[NS], ee = 0.0, T = 0.0, h0 = 0.0, p0 = 0.0, dt2 = 0.0;
    if (r >= 0) {
      dt2 = dt[r] / ks;
#pragma unroll
      for (int m = 0; m < NS; m++) d[m] = di[(size_t)r * NS + m];
      ee = e[r];
      if (CP) cp_reference<NS>(d, ee, h0, p0, nfail);
    }
    bool zero = false;
    for (int s = 0;; s++) {
      const unsigned lanes = __ballot_sync(0xffffffffu, s < ks);
      if (lanes == 0) break;
      if (s < ks) {
        zero = step<TPB>(lanes, d, ee, dt2, T, nfail, sp + threadIdx.x, tab) || zero;
        if (CP) restore_p(d, ee, h0, p0, T, nfail);
      }
    }
    if (r >= 0) {
      chem_check<NS>(d, ee, zero, nfail);
#pragma unroll
      for (int m = 0; m < NS; m++) di[(size_t)r * NS + m] = d[m];
      e[r] = ee;
    }
  }
}
}  // namespace mech_fast
}  // namespace ocfd
#endif
