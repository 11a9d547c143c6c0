// cns_turb.cu -- the turbulence-transport terms of the reference: the
// diffusion coefficients of the transport equations (met_fludc.f90 for
// k-epsilon, met_fludcsa.f90 for Spalart-Allmaras), the TVD Roe dissipation
// of the two transport variables (met_roe2o.f90, with Harten's entropy fix
// met_roe2oh.f90), the Spalart-Allmaras eddy viscosity (met_samut.f90) and
// the transport equations' explicit balance (sch_turb.f90).
//
// The transport state t and the dissipation d are the reference's (ld, 7)
// arrays (columns 6 and 7: the transport variables).  FP64, --fmad=false,
// reference expression order: bit-identical.
#include "cns_kernels.cuh"

namespace cns {

namespace {

inline int grid_of(const Space& s) { return s.ntiles; }

// met_fludc.f90:72-85 over the flat range [n0, n1]
__global__ void __launch_bounds__(256) k_fludc(long long n0, long long n1,
                                              const double* __restrict__ mu,
                                              const double* __restrict__ mut, double* fd5x,
                                              double* fd5y, double* fd5z, double* fd6x,
                                              double* fd6y, double* fd6z, double alfak,
                                              double alfae) {
  pdl_sync();
  const long long n = n0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n > n1) return;
  const double m = mu[n], mt = mut[n];
  fd5x[n] = (m + mt / alfak) * fd5x[n];
  fd5y[n] = (m + mt / alfak) * fd5y[n];
  fd5z[n] = (m + mt / alfak) * fd5z[n];
  fd6x[n] = (m + mt / alfae) * fd6x[n];
  fd6y[n] = (m + mt / alfae) * fd6y[n];
  fd6z[n] = (m + mt / alfae) * fd6z[n];
}

// met_fludcsa.f90:92-104 over the flat range [n0, n1]; s6 = s(:,6)
__global__ void __launch_bounds__(256) k_fludcsa(long long n0, long long n1,
                                                const double* __restrict__ s6,
                                                const double* __restrict__ mu, double* fd5x,
                                                double* fd5y, double* fd5z, double* fd6x,
                                                double* fd6y, double* fd6z, double sigma1) {
  pdl_sync();
  const long long n = n0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n > n1) return;
  const double smutot = sigma1 * (mu[n] + s6[n]);
  fd5x[n] = smutot * fd5x[n];
  fd5y[n] = smutot * fd5y[n];
  fd5z[n] = smutot * fd5z[n];
  fd6x[n] = 0.;
  fd6y[n] = 0.;
  fd6z[n] = 0.;
}

// met_roe2o.f90:288-296
__device__ __forceinline__ double amimd(double a, double b) {
  const double s = copysign(1.0, a);
  return s * fmax(0., fmin(fabs(a), b * s));
}
__device__ __forceinline__ double fi1(double x, double y, double z) {
  return amimd(x, amimd(y, z));
}
// met_roe2oh.f90:318-323
__device__ __forceinline__ double psi_h(double aa, double eps) {
  return 0.5 * (1. + copysign(1.0, fabs(aa) - eps)) * fabs(aa) +
         0.25 * (1. - copysign(1.0, fabs(aa) - eps)) * (aa * aa + eps * eps) / eps;
}

// dissipation coefficient of the face between the cells n (upper) and n1
// (met_roe2o.f90:89-101; met_roe2oh.f90 with harten): the half velocities
// rho u / (2 rho) are half the primitive ones, exactly
__device__ __forceinline__ double roe2o_coef(int harten, double epsroe, double gam, double gam1,
                                             const double* __restrict__ t,
                                             const double* __restrict__ prim, long long ld,
                                             long long n, long long n1, double s1, double s2,
                                             double s3) {
  const double u = 0.5 * prim[n] + 0.5 * prim[n1];
  const double v = 0.5 * prim[ld + n] + 0.5 * prim[ld + n1];
  const double w = 0.5 * prim[2 * ld + n] + 0.5 * prim[2 * ld + n1];
  if (!harten) return 0.5 * fabs(u * s1 + v * s2 + w * s3);
  const double etot = t[4 * ld + n] / (2 * t[n]) + t[4 * ld + n1] / (2 * t[n1]);
  const double q2 = 0.5 * (u * u + v * v + w * w);
  const double c = sqrt(gam * gam1 * (etot - q2));
  const double cnds = sqrt(s1 * s1 + s2 * s2 + s3 * s3);
  const double rlam = (u * s1 + v * s2 + w * s3) / cnds;
  return 0.5 * psi_h(rlam, epsroe * c) * cnds;
}

// TVD Roe dissipation d(:,6:7) of every cell of i 0..ni, j 0..nj, k 0..nk
// (met_roe2o.f90:89-114 and the j, i twins): per direction (k, j, i) the
// lower face subtracts, the upper face adds, where the face exists (the other
// two indices real); the ghost rows receive their one face.  The slope
// differences are extended past the ends (met_roe2o.f90:75-88: face 0 = face
// 1, face nd+1 = face nd).  A cell evaluates both its faces of a direction
// (its neighbour forms the same values), which costs less than writing the
// faces out and reading them back: 254 -> 127 us on a 2.1M-cell
// plate (cold, four launches before).
__global__ void __launch_bounds__(kTile) k_roe2o_cell(const Blk* __restrict__ blks, Space sp,
                                                      int harten, double epsroe, double gam,
                                                      double gam1, const double* __restrict__ t,
                                                      const double* __restrict__ prim,
                                                      long long ld,
                                                      const double* __restrict__ sn,
                                                      double* __restrict__ d) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  --i;
  --j;
  --k;
  const long long n = cell_index(B, i, j, k);
  double acc[2] = {0., 0.};
  const int idx[3] = {i, j, k};
  const int lim[3] = {B.ni, B.nj, B.nk};
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    const int dir = 2 - o;
    const int d1 = (dir + 1) % 3, d2 = (dir + 2) % 3;
    if (idx[d1] < 1 || idx[d1] > lim[d1] - 1 || idx[d2] < 1 || idx[d2] > lim[d2] - 1) continue;
    const int p = idx[dir], nd = lim[dir];
    const long long inc = ninc_of(B, dir);
    const double *s0 = sn_ptr(sn, B, dir, 0), *s1 = sn_ptr(sn, B, dir, 1),
                 *s2 = sn_ptr(sn, B, dir, 2);
    double cl = 0., cu = 0.;
    if (p >= 1)
      cl = roe2o_coef(harten, epsroe, gam, gam1, t, prim, ld, n, n - inc, s0[n], s1[n], s2[n]);
    if (p + 1 <= nd)
      cu = roe2o_coef(harten, epsroe, gam, gam1, t, prim, ld, n + inc, n, s0[n + inc],
                      s1[n + inc], s2[n + inc]);
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const double* tc = t + (5 + a) * ld + n;
      // slope differences of the faces p - 1 .. p + 2
      double del[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int f = min(max(p - 1 + q, 1), nd) - p;
        del[q] = tc[f * inc] - tc[(f - 1) * inc];
      }
      if (p >= 1) acc[a] = acc[a] - cl * (del[1] - fi1(del[0], del[1], del[2]));
      if (p + 1 <= nd) acc[a] = acc[a] + cu * (del[2] - fi1(del[1], del[2], del[3]));
    }
  }
  d[5 * ld + n] = acc[0];
  d[6 * ld + n] = acc[1];
}

// met_samut.f90:35-46 on the real cells: mut = v6 fv1 (x**3 as x*x*x)
__global__ void __launch_bounds__(kTile) k_samut(const Blk* __restrict__ blks, Space sp,
                                                 const double* __restrict__ v6,
                                                 const double* __restrict__ mu,
                                                 double* __restrict__ mut, double cv13) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const long long n = cell_index(blks[b], i, j, k);
  const double xkhi = v6[n] / mu[n];
  const double xkhi3 = xkhi * xkhi * xkhi;
  const double fv1 = xkhi3 / (xkhi3 + cv13);
  mut[n] = v6[n] * fv1;
}

// centred cell fluxes of the transport variables (sch_turb.f90:84-93)
__device__ __forceinline__ void turb_cell_flux(const double* __restrict__ v,
                                               const double* __restrict__ prim, long long ld,
                                               long long n, const double* const fd[6],
                                               double F[6]) {
  const double qx = prim[n], qy = prim[ld + n], qz = prim[2 * ld + n];
  const double t6 = v[5 * ld + n], t7 = v[6 * ld + n];
  F[0] = t6 * qx - fd[0][n];
  F[1] = t6 * qy - fd[1][n];
  F[2] = t6 * qz - fd[2][n];
  F[3] = t7 * qx - fd[3][n];
  F[4] = t7 * qy - fd[4][n];
  F[5] = t7 * qz - fd[5][n];
}

struct FdPtrs {
  const double* p[6];
};

// the explicit balance of sch_turb.f90:95-287 per real cell: interior faces
// sum the two cells' fluxes, boundary faces take twice the ghost cell's; the
// six faces in the reference's order, then u6 = 0.5 u6 - vol ts6 - d6 and the
// same for 7.  Each cell evaluates its own six faces from seven cells' fluxes
// (products of stored velocities), with no face buffer written and read back:
// 299 -> 140 us on a 2.1M-cell plate (cold, four launches before).
__global__ void __launch_bounds__(kTile) k_turb_cell(const Blk* __restrict__ blks, Space sp,
                                                     const double* __restrict__ v,
                                                     const double* __restrict__ prim,
                                                     long long ld, FdPtrs fdp,
                                                     const double* __restrict__ sn,
                                                     const double* __restrict__ vol,
                                                     const double* __restrict__ ts6,
                                                     const double* __restrict__ ts7,
                                                     const double* __restrict__ d,
                                                     double* __restrict__ u) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  const long long n = cell_index(B, i, j, k);
  double F0[6], acc[2] = {0., 0.};
  turb_cell_flux(v, prim, ld, n, fdp.p, F0);
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const long long inc = ninc_of(B, dir);
    const int nd = nd_of(B, dir);
    const int p = dir == 0 ? i : (dir == 1 ? j : k);
    const bool upper_first = (p == 1) && nd >= 3;
    const double *s0 = sn_ptr(sn, B, dir, 0), *s1 = sn_ptr(sn, B, dir, 1),
                 *s2 = sn_ptr(sn, B, dir, 2);
    double Fl[6], Fu[6];
    turb_cell_flux(v, prim, ld, n - inc, fdp.p, Fl);
    turb_cell_flux(v, prim, ld, n + inc, fdp.p, Fu);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      Fl[q] = p >= 2 ? F0[q] + Fl[q] : 2. * Fl[q];
      Fu[q] = p + 1 <= nd - 1 ? Fu[q] + F0[q] : 2. * Fu[q];
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const double gl = Fl[3 * a] * s0[n] + Fl[3 * a + 1] * s1[n] + Fl[3 * a + 2] * s2[n];
      const double gu = Fu[3 * a] * s0[n + inc] + Fu[3 * a + 1] * s1[n + inc] +
                        Fu[3 * a + 2] * s2[n + inc];
      if (upper_first) {
        acc[a] = acc[a] + gu;
        acc[a] = acc[a] - gl;
      } else {
        acc[a] = acc[a] - gl;
        acc[a] = acc[a] + gu;
      }
    }
  }
  u[5 * ld + n] = 0.5 * acc[0] - vol[n] * ts6[n] - d[5 * ld + n];
  u[6 * ld + n] = 0.5 * acc[1] - vol[n] * ts7[n] - d[6 * ld + n];
}

}  // namespace

cudaError_t launch_fludc(long long n0, long long n1, const double* mu, const double* mut,
                         double* const fd[6], double alfak, double alfae, cudaStream_t st) {
  if (n1 >= n0)
    pdl(k_fludc, (int)((n1 - n0 + 256) / 256), 256, 0, st)(n0, n1, mu, mut, fd[0], fd[1], fd[2],
                                                          fd[3], fd[4], fd[5], alfak, alfae);
  return cudaGetLastError();
}

cudaError_t launch_fludcsa(long long n0, long long n1, const double* s6, const double* mu,
                           double* const fd[6], double sigma, cudaStream_t st) {
  const double sigma1 = 1. / sigma;
  if (n1 >= n0)
    pdl(k_fludcsa, (int)((n1 - n0 + 256) / 256), 256, 0, st)(n0, n1, s6, mu, fd[0], fd[1],
                                                            fd[2], fd[3], fd[4], fd[5], sigma1);
  return cudaGetLastError();
}

cudaError_t launch_samut(const Blk* blks, Space cells, const double* v6, const double* mu,
                         double* mut, cudaStream_t st) {
  const double cv1 = 7.1;  // atlecdon.f90:200
  if (cells.ntiles > 0)
    pdl(k_samut, grid_of(cells), kTile, 0, st)(blks, cells, v6, mu, mut, cv1 * cv1 * cv1);
  return cudaGetLastError();
}

cudaError_t launch_sch_turb(const Blk* blks, Space cells, const double* v, const double* prim,
                            long long ld, const double* const fd[6], const double* ts6,
                            const double* ts7, const double* d, const double* sn,
                            const double* vol, double* u, cudaStream_t st) {
  FdPtrs fdp;
  for (int q = 0; q < 6; ++q) fdp.p[q] = fd[q];
  if (cells.ntiles > 0)
    pdl(k_turb_cell, grid_of(cells), kTile, 0, st)(blks, cells, v, prim, ld, fdp, sn, vol, ts6,
                                                   ts7, d, u);
  return cudaGetLastError();
}

cudaError_t launch_roe2o(const Blk* blks, Space cells_ext, int harten, double epsroe, double gam,
                         double gam1, const double* t, const double* prim, long long ld,
                         const double* sn, double* d, cudaStream_t st) {
  if (cells_ext.ntiles > 0)
    pdl(k_roe2o_cell, grid_of(cells_ext), kTile, 0, st)(blks, cells_ext, harten, epsroe, gam,
                                                        gam1, t, prim, ld, sn, d);
  return cudaGetLastError();
}

}  // namespace cns
