// Species viscous terms (du_scaler_viscous, OCFD_scaler_viscous.f90:4-79) and the species RK update
// (Scalar_time_adv_RK3, OCFD_Time_Adv.f90:134-166) on tensor-product grids, in their own translation
// unit. The cells at non-periodic faces and general grids keep k_scal_ev / k_scal_div (ocfd_flow.cuh).
#include <stdexcept>

#include "ocfd_flow.cuh"
#include "ocfd_launch.h"

namespace ocfd {

// A block is a 32 x SV_TY tile of cells of one plane, one cell per thread, every species in turn: the
// metric, the offsets and the stencil weights are formed once per cell, where the (cell, species)
// form spent 626 issued instructions per species and cell on them; 168 remain. The blocks of a slab
// of SV_SLAB tiles in j walk all k before the next slab, so that the z neighbours are read again while
// L2 still holds them. Bound by the latency of the loads (long_scoreboard at 16 warps per SM) at 2.5 to
// 3 TB/s of DRAM traffic. More warps per SM are slower, not faster: at 96 / 72 registers instead of
// 128 the pair of kernels took 8.3 instead of 6.8 ms per jet step, their rows evicting one another
// from L1; fewer (168 registers) 7.3; cp.async staging of the planes 8.1; two planes per thread 7.7.
// Measured with k_ci and the face cells, 9 species, ms per step, CD6 / CD8: contracted build 384x256x32
// 10.3 / 11.1 -> 6.8 / 7.6, 97x61x43 1.13 / 1.20 -> 0.85 / 0.94; exact build, whose face cells are three or
// four layers deep, 11.2 / 12.1 -> 7.7 / 8.7 and 1.21 / 1.30 -> 0.97 / 1.07.
constexpr int SV_TY = 4, SV_SLAB = 32 / SV_TY;
#ifndef OCFD_SE_MINB
#define OCFD_SE_MINB 4
#endif
#ifndef OCFD_SD_MINB
#define OCFD_SD_MINB 4
#endif

// the thread's cell; false when it has none
__device__ __forceinline__ bool sv_cell(int nbx, int& i, int& j, int& k) {
  const int bx = (int)blockIdx.x % nbx, bj = (int)blockIdx.x / nbx;
  i = bx * 32 + (int)threadIdx.x + 1;
  j = ((int)blockIdx.z * SV_SLAB + bj) * SV_TY + (int)threadIdx.y + 1;
  k = (int)blockIdx.y + 1;
  return i <= cC.nx && j <= cC.ny;
}
// A species' array is read through its base address, the same for every thread, and a 32-bit byte
// offset that is formed once per cell for all species (a halo array of several species is below
// 4 GB: the state, at least 50 such arrays, would not fit the device otherwise).
__device__ __forceinline__ double at(const double* base, unsigned off) {
  return __ldg(reinterpret_cast<const double*>(reinterpret_cast<const char*>(base) + off));
}
__device__ __forceinline__ void put(double* base, unsigned off, double v) {
  *reinterpret_cast<double*>(reinterpret_cast<char*>(base) + off) = v;
}
#if OCFD_FMA_BUILD
constexpr bool SV_WEIGHTS = true;
#else
constexpr bool SV_WEIGHTS = false;
#endif
// Derivative along one direction as a sum of weighted antisymmetric differences. Every closure of
// OCFD_dx0 but the one-sided form on the end planes has this shape with smaller reach (index 2:
// (f1 - f-1) / 2h; 3: the fourth-order form; CD8 at 4: CD6), so one straight-line code with weights
// per thread covers all cells but those planes, and no load waits behind a branch. Offsets beyond
// the domain are pulled in to the last point inside (their weight is zero). The exact build, which
// reproduces the closures' own operation order, takes this path for interior cells only.
template <int HZ>
struct Line {
  double w[HZ];
  unsigned p[HZ], m[HZ];  // byte offsets of the points up and down the line
  __device__ __forceinline__ Line(int dir, int ii, int n, int stride, int q) {
    // points on the nearer side (the exact build comes here with interior cells alone)
    const int dist = !SV_WEIGHTS || cC.iper[dir] ? HZ : min(ii - 1, n - ii);
#pragma unroll
    for (int r = 0; r < HZ; r++) {
      const int o = min(r + 1, dist) * stride;
      p[r] = (unsigned)(q + o) * 8u;
      m[r] = (unsigned)(q - o) * 8u;
    }
    if (HZ == 4 && dist >= 4) {
#pragma unroll
      for (int r = 0; r < HZ; r++) w[r] = cC.cd8[dir][r];
    } else {
      const double* a = cC.cd6[dir];  // outermost first
      const double h2 = 1.0 / cC.h2x[dir], h12 = 1.0 / cC.h12x[dir];
      w[0] = dist >= 3 ? a[2] : (dist == 2 ? 8.0 * h12 : h2);
      w[1] = dist >= 3 ? a[1] : (dist == 2 ? -h12 : 0.0);
      w[2] = dist >= 3 ? a[0] : 0.0;
      if (HZ == 4) w[HZ - 1] = 0.0;
    }
  }
  __device__ __forceinline__ void scale(double a) {
#pragma unroll
    for (int r = 0; r < HZ; r++) w[r] *= a;
  }
  // the reference's order of the interior sums: CD6 from the outermost pair in, CD8 from the inner out
  __device__ __forceinline__ void load(const double* f, double* v) const {
#pragma unroll
    for (int r = 0; r < HZ; r++) {
      v[2 * r] = at(f, p[r]);
      v[2 * r + 1] = at(f, m[r]);
    }
  }
  __device__ __forceinline__ double diff(const double* v) const {
    double d[HZ];
#pragma unroll
    for (int r = 0; r < HZ; r++) d[r] = v[2 * r] - v[2 * r + 1];
    if constexpr (HZ == 3) return w[2] * d[2] + w[1] * d[1] + w[0] * d[0];
    else return w[0] * d[0] + w[1] * d[1] + w[2] * d[2] + w[3] * d[3];
  }
};
__device__ __forceinline__ bool end_plane(int dir, int ii, int n) { return !cC.iper[dir] && (ii == 1 || ii == n); }
int face_layers(bool cd8) { return SV_WEIGHTS ? 1 : (cd8 ? 4 : 3); }
// whether a cell takes the straight-line path
__device__ __forceinline__ bool straight(int i, int j, int k) {
  if (SV_WEIGHTS) return !end_plane(0, i, cC.nx) && !end_plane(1, j, cC.ny) && !end_plane(2, k, cC.nz);
  return cdiff_interior(0, i, cC.nx) && cdiff_interior(1, j, cC.ny) && cdiff_interior(2, k, cC.nz);
}

// specific enthalpies h_k = R_k (c0 T + c1 T^2 / 2 + ... + Ect) as cubic-and-higher polynomials with
// the divisors folded in (contracted build; dev_hi evaluates the reference's expression)
constexpr int SV_NS = 9;
struct SpecConst {
  double h6[SV_NS][OCFD_NTCT_MAX][6];
};
__constant__ SpecConst cS;
cudaError_t species_setup(const DevConst& c, int ns) {
#if OCFD_FMA_BUILD
  SpecConst s{};
  for (int k = 0; k < ns && k < SV_NS; k++)
    for (int j = 0; j < OCFD_NTCT_MAX; j++) {
      if (c.realgas == 0) {
        s.h6[k][j][0] = 3.5 * c.Ri[k];
        continue;
      }
      for (int m = 0; m < 5; m++) s.h6[k][j][m] = (double)((long double)c.Ri[k] * c.cf[k][j][m] / (m + 1));
      s.h6[k][j][5] = c.Ri[k] * c.cf[k][j][7];
    }
  return cudaMemcpyToSymbol(cS, &s, sizeof(s));
#else
  (void)c; (void)ns;
  return cudaSuccess;
#endif
}
__device__ __forceinline__ double enthalpy(int k, int jc, double T) {
#if OCFD_FMA_BUILD
  if (T <= cC.tct_max || cC.realgas == 0) {
    const double* h = cS.h6[k][jc];
    return fma(T, fma(T, fma(T, fma(T, fma(T, h[4], h[3]), h[2]), h[1]), h[0]), h[5]);
  }
#endif
  return dev_hi(k, T);
}

// Diffusion fluxes of every species, e_d = d D_k grad(c_k) . A_d, and the enthalpy-flux sums Qp
// (species order), for the cells of the straight-line path: away from the end planes the metric
// matrix of a tensor-product grid is diagonal. The cells near the faces go to k_scal_ev.
template <int HZ>
__global__ void __launch_bounds__(32 * SV_TY, OCFD_SE_MINB)
    k_spec_ev(const double* __restrict__ ci, const double* __restrict__ d, const double* __restrict__ T,
              const double* __restrict__ amd, double* __restrict__ qpx, double* __restrict__ qpy,
              double* __restrict__ qpz, double* __restrict__ e1, double* __restrict__ e2, double* __restrict__ e3, Geo g,
              int ns, int nbx) {
  int i, j, k;
  if (!sv_cell(nbx, i, j, k)) return;
  if (!straight(i, j, k)) return;
  const long long H = cC.H, N = cC.N;
  const int q = hidx(i, j, k), nn = nidx(i, j, k);
  const double dq = d[q], Tq = T[q];
  double qx = 0.0, qy = 0.0, qz = 0.0;
  Line<HZ> lx(0, i, cC.nx, 1, q), ly(1, j, cC.ny, cC.HX, q), lz(2, k, cC.nz, cC.HX * cC.HY, q);
  double A[9], A1[9];
  metric_all<true>(g, i, j, k, q, A, A1);
#if OCFD_FMA_BUILD
  lx.scale(A[0]); ly.scale(A[4]); lz.scale(A[8]);  // the metric in the weights
  A[0] = A[4] = A[8] = 1.0;
#endif
  const int jc = trange(Tq);
  const unsigned qo = (unsigned)q * 8u, no = (unsigned)nn * 8u;
#pragma unroll 1
  for (int m = 0; m < ns; m++) {
    const double* c = ci + (size_t)m * H;
    double vx[2 * HZ], vy[2 * HZ], vz[2 * HZ];
    const double D = at(amd + (size_t)m * N, no);
    lx.load(c, vx);
    ly.load(c, vy);
    lz.load(c, vz);
    const double hi = enthalpy(m, jc, Tq);
    const double gx = lx.diff(vx), gy = ly.diff(vy), gz = lz.diff(vz);
    const double dD = dq * D;
    const double E1 = dD * (gx * A[0]), E2 = dD * (gy * A[4]), E3 = dD * (gz * A[8]);
    qx = qx + E1 * hi;
    qy = qy + E2 * hi;
    qz = qz + E3 * hi;
    put(e1 + (size_t)m * H, qo, E1 * A1[0]);
    put(e2 + (size_t)m * H, qo, E2 * A1[4]);
    put(e3 + (size_t)m * H, qo, E3 * A1[8]);
  }
  qpx[nn] = qx;
  qpy[nn] = qy;
  qpz[nn] = qz;
}

// Divergence of the diffusion fluxes added to Dus and, for KRK = 1..3, the species RK update on the
// finished value (Dus then stays in registers; nothing else reads it afterwards)
template <int HZ, int KRK>
__global__ void __launch_bounds__(32 * SV_TY, OCFD_SD_MINB)
    k_spec_div(const double* __restrict__ e1, const double* __restrict__ e2, const double* __restrict__ e3,
               double* __restrict__ dus, Geo g, double dt, const double* __restrict__ din, double* __restrict__ di,
               int ns, int nbx) {
  int i, j, k;
  if (!sv_cell(nbx, i, j, k)) return;
  if (!straight(i, j, k)) return;
  const double ra = KRK == 2 ? 3.0 / 4.0 : 1.0 / 3.0, rb = KRK == 2 ? 1.0 / 4.0 : 2.0 / 3.0;
  const long long H = cC.H, N = cC.N;
  const int q = hidx(i, j, k), nn = nidx(i, j, k);
  const double jac = metric_jac<true>(g, i, j, k, q);
  const unsigned qo = (unsigned)q * 8u, no = (unsigned)nn * 8u;
  const Line<HZ> lx(0, i, cC.nx, 1, q), ly(1, j, cC.ny, cC.HX, q), lz(2, k, cC.nz, cC.HX * cC.HY, q);
#pragma unroll 1
  for (int m = 0; m < ns; m++) {
    const size_t o = (size_t)m * H, on = (size_t)m * N;
    double vx[2 * HZ], vy[2 * HZ], vz[2 * HZ];
    const double du = dus[on + nn], dn = KRK == 0 ? 0.0 : at(din + on, no), dc = KRK <= 1 ? 0.0 : di[o + q];
    lx.load(e1 + o, vx);
    ly.load(e2 + o, vy);
    lz.load(e3 + o, vz);
    const double d1 = du + (lx.diff(vx) + ly.diff(vy) + lz.diff(vz)) * jac;
    if (KRK == 0) put(dus + on, no, d1);
    else if (KRK == 1) put(di + o, qo, dn + dt * d1);
    else put(di + o, qo, ra * dn + rb * (dc + dt * d1));
  }
}

namespace {
dim3 sv_grid(int nx, int ny, int nz, int& nbx) {
  auto nb = [](int n, int b) { return (n + b - 1) / b; };
  nbx = nb(nx, 32);
  const int nby = nb(ny, SV_TY);
  return dim3((unsigned)(nbx * SV_SLAB), (unsigned)nz, (unsigned)nb(nby, SV_SLAB));
}
template <int HZ>
void div_t(int ns, int krk, double dt, const SpecArgs& a, dim3 grid, int nbx, cudaStream_t st) {
  const dim3 block(32, SV_TY);
#define SD(K)                                                                                                     \
  case K:                                                                                                         \
    k_spec_div<HZ, K><<<grid, block, 0, st>>>(a.se[0], a.se[1], a.se[2], a.dus, a.g, dt, a.din, a.di, ns, nbx);    \
    break;
  switch (krk) { SD(0) SD(1) SD(2) SD(3) default: throw std::runtime_error("RK stage"); }
#undef SD
}
}  // namespace

void launch_spec_ev(int ns, bool cd8, const SpecArgs& a, cudaStream_t st) {
  int nbx;
  const dim3 grid = sv_grid(a.nx, a.ny, a.nz, nbx), block(32, SV_TY);
  (cd8 ? k_spec_ev<4> : k_spec_ev<3>)<<<grid, block, 0, st>>>(a.ci, a.d, a.T, a.amd, a.qp[0], a.qp[1], a.qp[2], a.se[0],
                                                            a.se[1], a.se[2], a.g, ns, nbx);
}
void launch_spec_div(int ns, bool cd8, int krk, double dt, const SpecArgs& a, cudaStream_t st) {
  int nbx;
  const dim3 grid = sv_grid(a.nx, a.ny, a.nz, nbx);
  if (cd8) div_t<4>(ns, krk, dt, a, grid, nbx, st);
  else div_t<3>(ns, krk, dt, a, grid, nbx, st);
}
}  // namespace ocfd
