// cns_flow.cu -- per-iteration kernels of the CodeNS hot path on sm_100a:
// thermodynamics (zpres, zvismo), local time step (chronos), boundary
// conditions and coincident halos (rbord, rbte, rbtc), viscous gradients and
// stresses (zgrad2 + zfluto), Roe-MUSCL face fluxes (sch_roe_euler, sch_roe
// with the in-place limiter recurrence), the face-owned accumulation of the
// residual, the matrix-free point-Jacobi implicit phase (implimf_eu,
// implimf_3d) and the residual norms (residu, rscpsv).
//
// Residual accumulation is face-owned, not atomic: each face flux is computed
// once into a face buffer, then every cell sums its six faces in exactly the
// order in which the reference's loops add them (interior faces in ascending
// order, then the lower and the upper boundary face), which keeps the FP64
// result bit-identical.
#include <math_constants.h>

#include "cns_kernels.cuh"
#include "cns_pmath.h"
#include "cns_hot.cuh"

namespace cns {

namespace {

inline int grid_of(const Space& s) { return s.ntiles; }

// ---------------------------------------------------------------------------
// thermodynamics
// ---------------------------------------------------------------------------

// zpres.f90:66-79 and, for the Navier-Stokes equations, zvismo.f90:77-104,
// of cell n; returns c (and mu through *mu_n when with_mu)
__device__ __forceinline__ double zpres_cell(Phys ph, int with_mu,
                                             const double* __restrict__ v, long long ld,
                                             long long n, double* ps, double* temp,
                                             double* cson, double* mu, int* status,
                                             double* mu_n) {
  const double v1 = v[n], v2 = v[ld + n], v3 = v[2 * ld + n], v4 = v[3 * ld + n],
               v5 = v[4 * ld + n];
  const double rhoe = v5 - 0.5 * (sq(v2) + sq(v3) + sq(v4)) / v1;
  const double p = ph.gam1 * (rhoe - ph.pinfl);
  const double t = ph.gam * p / v1;
  ps[n] = p;
  temp[n] = t;
  const double c = sqrt(t);
  cson[n] = c;
  if (with_mu) {
    // the reference aborts on T <= 0 (zvismo.f90:123-127); here the status
    // word records it and the host turns it into an error code
    double m;
    if (t <= 0.) {
      m = 0.;
      atomicOr(status, 1);
    } else {
      const double usrey = 1. / ph.reynz, a = ph.suth_a;
      m = usrey * t * sqrt(t) * (1. + a) / (t + a);
    }
    mu[n] = m;
    *mu_n = m;
  }
  return c;
}

__global__ void __launch_bounds__(kTile) k_zpres(const Blk* __restrict__ blks,
                                                 Space sp, Phys ph, int with_mu,
                                                 const double* __restrict__ v,
                                                 long long ld, double* ps,
                                                 double* temp, double* cson,
                                                 double* mu, int* status) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const long long n = cell_index(blks[b], i, j, k);
  double m;
  (void)zpres_cell(ph, with_mu, v, ld, n, ps, temp, cson, mu, status, &m);
}

// zvismo.f90:77-104 alone (temperature already known)
__global__ void __launch_bounds__(kTile) k_zvismo(const Blk* __restrict__ blks,
                                                  Space sp, Phys ph, double* mu,
                                                  const double* __restrict__ temp,
                                                  int* status) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const long long n = cell_index(blks[b], i, j, k);
  const double t = temp[n];
  if (t <= 0.) {
    mu[n] = 0.;
    atomicOr(status, 1);
  } else {
    const double usrey = 1. / ph.reynz, a = ph.suth_a;
    mu[n] = usrey * t * sqrt(t) * (1. + a) / (t + a);
  }
}

// primitive velocities u = rho u / rho (and v, w) of every cell of a flat
// range, once per iteration after the boundary conditions: the face fluxes,
// the limiter ratios, the gradients and the implicit phase all use these very
// quotients (the reference recomputes them at every use, with identical
// results), so sharing them changes no bit
template <bool SHADOW>
__global__ void __launch_bounds__(256) k_prim(long long n0, long long n1,
                                             const double* __restrict__ v,
                                             long long ld, double* __restrict__ prim,
                                             const double* __restrict__ ps, PrimShadow sh) {
  pdl_sync();
  const long long n = n0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n1) return;
  const double r = v[n];
  const double q0 = v[ld + n] / r, q1 = v[2 * ld + n] / r, q2 = v[3 * ld + n] / r;
  prim[n] = q0;
  prim[ld + n] = q1;
  prim[2 * ld + n] = q2;
  if (SHADOW) {
    // the single-precision copies (PrimShadow)
    const float r32 = (float)r, e32 = (float)v[4 * ld + n], p32 = (float)ps[n];
    const float u32 = (float)q0, w1 = (float)q1, w2 = (float)q2;
    const Blk* __restrict__ blks = sh.blks;
    const int nblk = sh.nblk;
    float* __restrict__ st32 = sh.st32;
    sh.cq32[n] = make_float4(u32, w1, w2, (float)sh.cson[n]);
    sh.cv32[n] = make_float2(
        (float)sh.vol[n],
        sh.eu ? 0.f : (sh.gp * (float)sh.mu[n] + sh.gpt * (float)sh.mut[n]) / r32);
    if (sh.v32) {
      sh.prim32[n] = u32;
      sh.prim32[ld + n] = w1;
      sh.prim32[2 * ld + n] = w2;
      sh.v32[n] = r32;
#pragma unroll
      for (int a = 1; a < 4; ++a) sh.v32[a * ld + n] = (float)v[a * ld + n];
      sh.v32[4 * ld + n] = e32;
      sh.ps32[n] = p32;
    }
    if (st32) {
      // the cell's block (blocks in increasing npc) and (i, j, k) in it
      int lo = 0, hi = nblk - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (blks[mid].npc <= n) lo = mid;
        else hi = mid - 1;
      }
      const Blk& B = blks[lo];
      const long long q = n - B.npc;
      if (q < B.nnn) {
        // (i, j, k) by 32-bit divisions (a block holds fewer than 2^31 cells)
        const unsigned q32 = (unsigned)q, nijd = (unsigned)B.nijd, nid = (unsigned)B.nid;
        const unsigned k = q32 / nijd, rem = q32 - k * nijd;
        const unsigned j = rem / nid, i = rem - j * nid;
        const long long pn = pad_index(B, i, j, k);
        st32[pn] = r32;
        st32[B.pld + pn] = e32;
        st32[2 * B.pld + pn] = p32;
        st32[3 * B.pld + pn] = u32;
        st32[4 * B.pld + pn] = w1;
        st32[5 * B.pld + pn] = w2;
      }
    }
  }
}

// the length of cell nc: volume by face area (chronos.f90:110-130)
__device__ __forceinline__ double chronos_length(const Blk& B, long long nc,
                                                 const double* __restrict__ sn,
                                                 const double* __restrict__ vol) {
  double sf[3][2];
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const long long inc = ninc_of(B, dir);
    const double *s0 = sn_ptr(sn, B, dir, 0), *s1 = sn_ptr(sn, B, dir, 1),
                 *s2 = sn_ptr(sn, B, dir, 2);
    sf[dir][0] = s0[nc] * s0[nc] + s1[nc] * s1[nc] + s2[nc] * s2[nc];
    sf[dir][1] = s0[nc + inc] * s0[nc + inc] + s1[nc + inc] * s1[nc + inc] +
                 s2[nc + inc] * s2[nc + inc];
  }
  const double simax = fmax(sf[0][1], sf[0][0]);
  const double sjmax = fmax(sf[1][1], sf[1][0]);
  const double skmax = fmax(sf[2][1], sf[2][0]);
  const double smoy = sqrt(simax + sjmax + skmax);
  return vol[nc] / smoy;
}

// the local time step of cell nc (chronos.f90:110-194, kprec = 0) from its
// state t (rho, rho u, rho v, rho w), length, sound speed c and viscosities
__device__ __forceinline__ double chronos_cell(const Blk& B, Phys ph, Scheme sc,
                                               const double* __restrict__ t, long long ld,
                                               long long nc, double dism, double c, double mu_c,
                                               double mut_c) {
  const double ro = t[nc];
  const double qq = (sq(t[ld + nc]) + sq(t[2 * ld + nc]) + sq(t[3 * ld + nc])) / sq(ro);
  const double q = sqrt(qq);
  const double dte = dism / (q + c);
  double d = B.eta * dte;
  if (sc.ns) {
    const double rv1 = ph.gam * (mu_c / ph.pr + mut_c / ph.prt) / t[nc];
    const double rv = fmax(rv1, 4. / 3. * (mu_c + mut_c) / t[nc]);
    const double dtv = B.eta * 0.25 * sq(dism) / rv;
    d = fmin(d, dtv);
  }
  return d;
}

__global__ void __launch_bounds__(kTile) k_chronos(
    const Blk* __restrict__ blks, Space sp, Phys ph, Scheme sc,
    const double* __restrict__ mu, const double* __restrict__ mut,
    const double* __restrict__ t, long long ld, double* dt,
    const double* __restrict__ sn, const double* __restrict__ vol,
    const double* __restrict__ cson) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  const long long nc = cell_index(B, i, j, k);
  dt[nc] = chronos_cell(B, ph, sc, t, ld, nc, chronos_length(B, nc, sn, vol), cson[nc],
                        sc.ns ? mu[nc] : 0., sc.ns ? mut[nc] : 0.);
}

// zpres (+ zvismo) and chronos of each real cell in one pass: the time step
// takes the sound speed and viscosity just computed (the values the separate
// kernels store and re-read)
__global__ void __launch_bounds__(kTile) k_zpres_chronos(
    const Blk* __restrict__ blks, Space sp, Phys ph, Scheme sc, const double* __restrict__ v,
    long long ld, double* ps, double* temp, double* cson, double* mu,
    const double* __restrict__ mut, double* dt, const double* __restrict__ sn,
    const double* __restrict__ vol, int* status) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  const long long n = cell_index(B, i, j, k);
  double m = 0.;
  const double mt = sc.ns ? mut[n] : 0.;
  // first, so that its loads go with the state's: 151 -> 142 us on 4.4M cells
  const double dism = chronos_length(B, n, sn, vol);
  const double c = zpres_cell(ph, sc.ns, v, ld, n, ps, temp, cson, mu, status, &m);
  dt[n] = chronos_cell(B, ph, sc, v, ld, n, dism, c, m, mt);
}

// ---------------------------------------------------------------------------
// boundary conditions (rbord.f90:137-429)
// ---------------------------------------------------------------------------

// one list entry of a coincident, extrapolation, adiabatic-wall or
// outlet-pressure boundary; injection boundaries are handled by
// k_clidd_count and k_clidd_apply.
// rbvc runs before and after the physical conditions in the reference; every
// ghost cell depends on interior cells only, so one pass gives the same values.
// An entry is a chain of latencies (the lists, then its cells): it loads all
// its cells' values before the first store, which may not pass a load of the
// same array (with k_tau_ghosts and the time step's loads an iteration of
// 64x32x32 limited Navier-Stokes cells 144.5 -> 140.0 us, of 16x12x8 Euler 66.7 ->
// 65.3).
__global__ void __launch_bounds__(256) k_rbord(Bnd bd, Phys ph, double* v,
                                              long long ld, double* ps,
                                              double* temp, double* cson,
                                              unsigned* idd_work) {
  pdl_sync();
  // the injection boundaries' work starts at zero (k_clidd_count follows)
  if (blockIdx.x == 0)
    for (int q = threadIdx.x; q < 3 * bd.nbnd + 1; q += blockDim.x) idd_work[q] = 0u;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= bd.nlist) return;
  const int bb = bd.ent_bnd[e];
  const int kind = bd.type[bb];
  const long long nd = bd.ncbd[e], ni = bd.ncin[e];
  if (kind == BC_RC) {  // rbvc.f90:40-92
    const int p = bd.partner[bb];
    const long long nc = bd.ncin[bd.mpb[p] + (e - bd.mpb[bb])];
    const double c = bd.cosr[p], s = bd.sinr[p];
    const double b0 = v[nc], b1 = v[ld + nc];
    const double b2 = v[2 * ld + nc] * c + v[3 * ld + nc] * s;
    const double b3 = v[3 * ld + nc] * c - v[2 * ld + nc] * s;
    const double b4 = v[4 * ld + nc];
    const double b5 = ps[nc], b6 = temp[nc], b7 = cson[nc];
    const double a0 = v[ni], a1 = v[ld + ni], a2 = v[2 * ld + ni], a3 = v[3 * ld + ni],
                 a4 = v[4 * ld + ni], a5 = ps[ni], a6 = temp[ni], a7 = cson[ni];
    v[nd] = 0.5 * (a0 + b0);
    v[ld + nd] = 0.5 * (a1 + b1);
    v[2 * ld + nd] = 0.5 * (a2 + b2);
    v[3 * ld + nd] = 0.5 * (a3 + b3);
    v[4 * ld + nd] = 0.5 * (a4 + b4);
    ps[nd] = 0.5 * (a5 + b5);
    temp[nd] = 0.5 * (a6 + b6);
    cson[nd] = 0.5 * (a7 + b7);
  } else if (kind == BC_EXTR) {  // clextr.f90:23-37
    double x[5];
#pragma unroll
    for (int a = 0; a < 5; ++a) x[a] = v[a * ld + ni];
    const double p = ps[ni], tt = temp[ni], c = cson[ni];
#pragma unroll
    for (int a = 0; a < 5; ++a) v[a * ld + nd] = x[a];
    ps[nd] = p;
    temp[nd] = tt;
    cson[nd] = c;
  } else if (kind == BC_PARA || kind == BC_LP2) {  // clpara.f90:24-40 (rbord.f90:374-388)
    const double v1 = v[ni], v2 = v[ld + ni], v3 = v[2 * ld + ni], v4 = v[3 * ld + ni];
    const double p = ps[ni], tt = temp[ni], c = cson[ni];
    const double rhoe1 = v[4 * ld + ni] - 0.5 * (sq(v2) + sq(v3) + sq(v4)) / v1;
    v[nd] = v1;
    v[ld + nd] = 0.;
    v[2 * ld + nd] = 0.;
    v[3 * ld + nd] = 0.;
    v[4 * ld + nd] = rhoe1;
    ps[nd] = p;
    temp[nd] = tt;
    cson[nd] = c;
  } else if (kind == BC_PRD) {  // rbve.f90 then clprd.f90:31-59
    const double gam = ph.gam, gam1 = ph.gam1, pinfl = ph.pinfl;
    const double pres = bd.bceqt[e];
    const double r1 = v[ni];
    const double qxs = v[ld + ni] / r1, qys = v[2 * ld + ni] / r1, qzs = v[3 * ld + ni] / r1;
    const double p = gam1 * (v[4 * ld + ni] - 0.5 * r1 * (sq(qxs) + sq(qys) + sq(qzs)) - pinfl);
    const double cs2 = gam * p / r1;
    const double roc0 = sqrt(gam * p * r1);
    const double dqn = (pres - p) / roc0;
    const double qx = qxs + dqn * bd.nxn[e];
    const double qy = qys + dqn * bd.nyn[e];
    const double qz = qzs + dqn * bd.nzn[e];
    const double drho = (pres - p) / cs2;
    const double rho = r1 + drho;
    v[nd] = rho;
    v[ld + nd] = rho * qx;
    v[2 * ld + nd] = rho * qy;
    v[3 * ld + nd] = rho * qz;
    v[4 * ld + nd] = pres / gam1 + pinfl + 0.5 * rho * (sq(qx) + sq(qy) + sq(qz));
    ps[nd] = pres;
    const double tt = gam * pres / rho;
    temp[nd] = tt;
    cson[nd] = sqrt(tt);
  }
}

// utidd.f90 + rbve.f90 + clidd.f90:50-170: injection at imposed total
// pressure, total temperature and flow direction.  The reference iterates a
// Newton method on the normal velocity of every boundary cell, sweep after
// sweep, until the largest relative update over the whole boundary is at most
// 1e-7 (at most 20 sweeps).  Each cell's iterate depends on that cell only;
// only the number of sweeps is global.  So k_clidd_count takes every cell to
// the first sweep t whose update is small and keeps the boundary's largest t
// (every earlier sweep has that cell's large update).  A cell of reversed flow
// counts as small whatever its update (clidd.f90:113 divides by the signed
// velocity) and may be large again once it turns, so such a cell records all
// its sweeps: the boundary stops at the first sweep from t on that no reversed
// cell holds open.  k_clidd_apply replays that many sweeps and looks at each
// cell's last update again: should a forward cell be large there (in a rotating
// frame the derivative may vanish beside its iterate), its last CTA redoes the
// boundary from the record of all 20 sweeps.  The same values as the sequential
// loop.  Latency of the dependent
// sweeps (a real power each) bounds both: recording all 20 sweeps of every cell
// takes 28 us on a 5.5k-cell inlet, the count 12 us.  With the redo for the
// reversed cells too, ghosts with 5% of them took 8.2 ms on a 16k-cell inlet
// (40 us without any), with their record 57 us.
// work (unsigned): nbnd largest sweeps (then sweep masks of a redo), nbnd masks
// of the reversed cells' large sweeps, nbnd redo flags, a counter of finished
// CTAs; k_rbord clears it.
struct IddCell {
  double usdn, usdn2, un, qn, roc0, am0, rpi, rti;
};

__device__ __forceinline__ void idd_setup(const Bnd& bd, const Phys& ph,
                                          const double* __restrict__ v,
                                          long long ld, long long e, IddCell& c) {
  const long long nl = bd.nlist, ni = bd.ncin[e];
  const double d0x = bd.bceqt[2 * nl + e], d0y = bd.bceqt[3 * nl + e],
               d0z = bd.bceqt[4 * nl + e];
  const double nx = bd.nxn[e], ny = bd.nyn[e], nz = bd.nzn[e];
  c.rpi = bd.bceqt[e];
  c.rti = bd.bceqt[nl + e];
  c.usdn = 1. / (d0x * nx + d0y * ny + d0z * nz);
  c.usdn2 = sq(c.usdn);
  c.un = ph.omg * (bd.ym[e] * nz - bd.zm[e] * ny);
  // the ghost cell holds the interior state (rbve) when clidd reads it
  const double r1 = v[ni], r2 = v[ld + ni], r3 = v[2 * ld + ni], r4 = v[3 * ld + ni];
  const double qxs = r2 / r1, qys = r3 / r1, qzs = r4 / r1;
  c.qn = qxs * nx + qys * ny + qzs * nz;
  const double p = ph.gam1 * (v[4 * ld + ni] - 0.5 * (qxs * r2 + qys * r3 + qzs * r4) - ph.pinfl);
  c.roc0 = -sqrt(ph.gam * p * r1);
  c.am0 = p + c.roc0 * c.qn;
}

// one Newton sweep of clidd.f90:96-113 on one cell; returns resi
__device__ __forceinline__ double idd_sweep(const Phys& ph, IddCell& c) {
  const double gam6 = ph.gam / ph.gam1;
  const double gamt = ph.gam / sq(ph.aa1);
  const double gam2t = 0.5 * ph.gam1 / sq(ph.aa1);
  const double b = 1. / (1. + gam2t / c.rti * c.usdn2 * sq(c.qn + c.un));
  const double p = ph.pa1 * c.rpi * cns_pow(b, gam6);
  const double ro = gamt * p / (b * c.rti);
  const double f = p + c.roc0 * c.qn - c.am0;
  const double df = c.roc0 - ro * (c.qn + c.un) * c.usdn2;
  const double dqn = -f / df;
  const double resi = fabs(dqn) / c.qn;
  c.qn = c.qn + dqn;
  return resi;
}

constexpr double kIddTol = 0.0000001;

__global__ void __launch_bounds__(64) k_clidd_count(Bnd bd, Phys ph, const long long* ents,
                                                   long long nent, const double* v,
                                                   long long ld, unsigned* work) {
  pdl_sync();
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nent) return;
  const long long e = ents[q];
  IddCell c;
  idd_setup(bd, ph, v, ld, e, c);
  const int b = bd.ent_bnd[e];
  unsigned t = 0;
  double resi = 0.;
  while (t < 20 && (resi = idd_sweep(ph, c)) > kIddTol) ++t;
  atomicMax(&work[b], t);
  if (t < 20 && resi < 0.) {
    unsigned late = 0u;
    while (++t < 20)
      if (idd_sweep(ph, c) > kIddTol) late |= 1u << t;
    if (late) atomicOr(&work[bd.nbnd + b], late);
  }
}

// nsweep sweeps of entry e, then its ghost state; returns the last update
__device__ __forceinline__ double idd_apply(const Bnd& bd, const Phys& ph, long long e,
                                            int nsweep, double* v, long long ld, double* ps_,
                                            double* temp, double* cson) {
  const long long nl = bd.nlist, nc = bd.ncbd[e];
  IddCell c;
  idd_setup(bd, ph, v, ld, e, c);
  double resi = 0.;
  for (int t = 0; t < nsweep; ++t) resi = idd_sweep(ph, c);
  const double gam = ph.gam, gam1 = ph.gam1, pinfl = ph.pinfl, omg = ph.omg;
  const double gam6 = gam / gam1;
  const double gamt = gam / sq(ph.aa1);
  const double gam2t = 0.5 * gam1 / sq(ph.aa1);
  const double d0x = bd.bceqt[2 * nl + e], d0y = bd.bceqt[3 * nl + e],
               d0z = bd.bceqt[4 * nl + e];
  const double ym = bd.ym[e], zm = bd.zm[e];
  const double b = 1. / (1. + gam2t / c.rti * c.usdn2 * sq(c.qn + c.un));
  const double p = ph.pa1 * c.rpi * cns_pow(b, gam6);
  const double ro = gamt * p / (b * c.rti);
  const double wn = c.qn + c.un;
  const double w = wn * c.usdn;
  const double m2 = ro * (w * d0x);
  const double m3 = ro * (w * d0y + zm * omg);
  const double m4 = ro * (w * d0z - ym * omg);
  v[nc] = ro;
  v[ld + nc] = m2;
  v[2 * ld + nc] = m3;
  v[3 * ld + nc] = m4;
  v[4 * ld + nc] = p / gam1 + pinfl + 0.5 * (sq(m2) + sq(m3) + sq(m4)) / ro;
  ps_[nc] = p;
  const double tt = gam * p / ro;
  temp[nc] = tt;
  cson[nc] = sqrt(tt);
  return resi;
}

__global__ void __launch_bounds__(64) k_clidd_apply(Bnd bd, Phys ph, const long long* ents,
                                                   long long nent, double* v, long long ld,
                                                   double* ps, double* temp, double* cson,
                                                   unsigned* work) {
  pdl_sync();
  const unsigned* late = work + bd.nbnd;
  unsigned *flag = work + 2 * bd.nbnd, *count = work + 3 * bd.nbnd;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < nent) {
    const long long e = ents[q];
    const int b = bd.ent_bnd[e];
    // the first sweep from work[b] on that no reversed cell holds open (or 20)
    const int m = __ffs((int)(~late[b] >> work[b])) - 1 + (int)work[b];
    const double resi = idd_apply(bd, ph, e, m < 20 ? m + 1 : 20, v, ld, ps, temp, cson);
    if (m < 20 && resi > kIddTol) atomicOr(&flag[b], 1u);
  }
  __shared__ unsigned last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ int redo;
  if (threadIdx.x == 0) redo = 0;
  __syncthreads();
  for (int b = threadIdx.x; b < bd.nbnd; b += blockDim.x)
    if (__ldcg(&flag[b])) {
      work[b] = 0u;
      redo = 1;
    }
  __threadfence();
  __syncthreads();
  if (!redo) return;
  for (long long r = threadIdx.x; r < nent; r += blockDim.x) {
    const long long e = ents[r];
    const int b = bd.ent_bnd[e];
    if (!__ldcg(&flag[b])) continue;
    IddCell c;
    idd_setup(bd, ph, v, ld, e, c);
    unsigned bits = 0u;
    for (int t = 0; t < 20; ++t)
      if (idd_sweep(ph, c) > kIddTol) bits |= 1u << t;
    atomicOr(&work[b], bits);
  }
  __threadfence();
  __syncthreads();
  for (long long r = threadIdx.x; r < nent; r += blockDim.x) {
    const long long e = ents[r];
    const int b = bd.ent_bnd[e];
    if (!__ldcg(&flag[b])) continue;
    const unsigned clear = ~__ldcg(&work[b]) & 0xfffffu;
    (void)idd_apply(bd, ph, e, clear ? __ffs((int)clear) : 20, v, ld, ps, temp, cson);
  }
}

// rbte.f90:15-31 (non-coincident boundaries: copy of the interior cell) and
// rbtc.f90:30-100 (coincident: average with the rotated partner)
__global__ void __launch_bounds__(256) k_tau_ghosts(Bnd bd, double* tau, long long ld) {
  pdl_sync();
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= bd.nlist) return;
  const int bb = bd.ent_bnd[e];
  const long long nd = bd.ncbd[e], ndm = bd.ncin[e];
  if (bd.type[bb] != BC_RC) {
    double x[9];
#pragma unroll
    for (int a = 0; a < 9; ++a) x[a] = tau[a * ld + ndm];
#pragma unroll
    for (int a = 0; a < 9; ++a) tau[a * ld + nd] = x[a];
    return;
  }
  const int p = bd.partner[bb];
  const long long nc = bd.ncin[bd.mpb[p] + (e - bd.mpb[bb])];
  const double sr = -bd.sinr[p], cr = bd.cosr[p];
  const double txx = tau[nc], txy = tau[ld + nc], txz = tau[2 * ld + nc],
               tyy = tau[3 * ld + nc], tyz = tau[4 * ld + nc], tzz = tau[5 * ld + nc];
  double bf[9];
  bf[0] = txx;
  bf[1] = cr * txy - sr * txz;
  bf[2] = cr * txz + sr * txy;
  bf[3] = cr * cr * tyy - 2. * cr * sr * tyz + sr * sr * tzz;
  bf[4] = -cr * sr * (tzz - tyy) + (2. * cr * cr - 1.) * tyz;
  bf[5] = sr * sr * tyy + 2. * cr * sr * tyz + cr * cr * tzz;
  bf[6] = tau[6 * ld + nc];
  bf[7] = cr * tau[7 * ld + nc] - sr * tau[8 * ld + nc];
  bf[8] = cr * tau[8 * ld + nc] + sr * tau[7 * ld + nc];
  double x[9];
#pragma unroll
  for (int a = 0; a < 9; ++a) x[a] = tau[a * ld + ndm];
#pragma unroll
  for (int a = 0; a < 9; ++a) tau[a * ld + nd] = 0.5 * (x[a] + bf[a]);
}

// ---------------------------------------------------------------------------
// viscous gradients and stresses: zgrad2.f90 (unit weights, inivec.f90:110)
// then zfluto.f90:38-57, per real cell
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kTile) k_grad(const Blk* __restrict__ blks,
                                                Space sp, Phys ph,
                                                const double* __restrict__ s,
                                                const double* __restrict__ prim,
                                                long long ld,
                                                const double* __restrict__ mu,
                                                const double* __restrict__ mut,
                                                double* __restrict__ tau,
                                                const double* __restrict__ sn,
                                                const double* __restrict__ vol,
                                                const double* __restrict__ temp,
                                                double* __restrict__ rv) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  const long long n = cell_index(B, i, j, k);
  double g[12];
#pragma unroll
  for (int a = 0; a < 12; ++a) g[a] = 0.;
  const double fc[4] = {prim[n], prim[ld + n], prim[2 * ld + n], temp[n]};
  // directions in the reference's order: k faces, then j, then i
#pragma unroll
  for (int oi = 0; oi < 3; ++oi) {
    const int dir = 2 - oi;
    const long long inc = ninc_of(B, dir);
    const int nd = nd_of(B, dir);
    const int p = dir == 0 ? i : (dir == 1 ? j : k);
    const double *s0 = sn_ptr(sn, B, dir, 0), *s1 = sn_ptr(sn, B, dir, 1),
                 *s2 = sn_ptr(sn, B, dir, 2);
    const long long nl = n - inc, nu = n + inc;
    const double fl[4] = {prim[nl], prim[ld + nl], prim[2 * ld + nl], temp[nl]};
    const double fu[4] = {prim[nu], prim[ld + nu], prim[2 * ld + nu], temp[nu]};
    const double sl[3] = {s0[n], s1[n], s2[n]};
    const double su[3] = {s0[nu], s1[nu], s2[nu]};
    const bool lower_bnd = (p == 1), upper_bnd = (p + 1 == nd);
    const bool upper_first = lower_bnd && nd >= 3;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const bool do_upper = (pass == 0) == upper_first;
      if (!do_upper) {  // lower face of the cell
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (lower_bnd)
              g[3 * a + c] = g[3 * a + c] - sl[c] * 2 * fl[a];
            else
              g[3 * a + c] = g[3 * a + c] - (fc[a] + fl[a]) * sl[c];
          }
      } else {  // upper face
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (upper_bnd)
              g[3 * a + c] = g[3 * a + c] + su[c] * 2 * fu[a];
            else
              g[3 * a + c] = g[3 * a + c] + (fu[a] + fc[a]) * su[c];
          }
      }
    }
  }
  const double eps = 0.00001, ds3 = 2. / 3.;
  const double vn = vol[n];
  const double ts = copysign(0.5, -vn);
  const double vols = (0.5 + ts) * eps + (0.5 - ts) * vn;
  const double c0 = .5 / (vols + 2.2250738585072014e-308);
#pragma unroll
  for (int a = 0; a < 12; ++a) g[a] = g[a] * c0;
  const double dvxx = g[0], dvxy = g[1], dvxz = g[2], dvyx = g[3], dvyy = g[4],
               dvyz = g[5], dvzx = g[6], dvzy = g[7], dvzz = g[8];
  const double m = mu[n] + mut[n];
  tau[n] = ds3 * m * (2 * dvxx - dvyy - dvzz);
  tau[3 * ld + n] = ds3 * m * (2 * dvyy - dvxx - dvzz);
  tau[5 * ld + n] = ds3 * m * (2 * dvzz - dvxx - dvyy);
  tau[ld + n] = m * (dvxy + dvyx);
  tau[2 * ld + n] = m * (dvxz + dvzx);
  tau[4 * ld + n] = m * (dvyz + dvzy);
  const double kd = mu[n] / ph.pr + mut[n] / ph.prt;
  const double kq = ph.cp * kd;
  tau[6 * ld + n] = kq * g[9];
  tau[7 * ld + n] = kq * g[10];
  tau[8 * ld + n] = kq * g[11];
  // the viscous spectral factor of the implicit phase (k_impl_rv)
  if (rv) rv[n] = ph.gam * kd / s[n];
}

// the viscous spectral factor rv of a real cell (implimf_3d.f90:95-105), for
// the calls that do not run k_grad before the implicit phase
__global__ void __launch_bounds__(kTile) k_impl_rv(const Blk* __restrict__ blks, Space sp,
                                                   Phys ph, const double* __restrict__ v,
                                                   const double* __restrict__ mu,
                                                   const double* __restrict__ mut, double* rv) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const long long n = cell_index(blks[b], i, j, k);
  rv[n] = ph.gam * (mu[n] / ph.pr + mut[n] / ph.prt) / v[n];
}

// spectral radius of one face (implimf_eu.f90:141-159, implimf_3d.f90:110-190)
// from its two cells q = (u, v, w, c, rv, vol) (Euler: u, v, w from the
// reciprocal density); every sum of the two cells is symmetric, so both cells
// of a face form the same value
template <bool EU>
__device__ __forceinline__ double face_radius(const double a[6], const double b[6], double sx,
                                              double sy, double sz) {
  const double cnds = sx * sx + sy * sy + sz * sz;
  const double cc = 0.5 * (a[3] + b[3]);
  const double uu = 0.5 * (a[0] + b[0]), vv = 0.5 * (a[1] + b[1]), ww = 0.5 * (a[2] + b[2]);
  const double vn = uu * sx + vv * sy + ww * sz;
  if (EU) return 0.5 * (fabs(vn)) + sqrt(cnds) * cc;
  return 0.5 * (fabs(vn) + sqrt(cnds) * cc) + (a[4] + b[4]) * cnds / (a[5] + b[5]);
}

// the flux increments of the iterate d of cell n (the reference expressions)
template <bool EU>
__device__ __forceinline__ void point_df(const double* __restrict__ v,
                                         const double* __restrict__ prim,
                                         const double* __restrict__ ps, long long ld,
                                         long long n, double gam1, double pinfl, int qfix,
                                         const double d[5], double f[9]) {
  jacobi_df<double, EU>(d, v[n], v[ld + n], v[2 * ld + n], v[3 * ld + n], v[4 * ld + n], ps[n],
                        EU ? 0. : prim[n], EU ? 0. : prim[ld + n], EU ? 0. : prim[2 * ld + n],
                        gam1, pinfl, qfix, f);
}

// (d, f) of cell n of the point sweeps' packed iterate; zero unless in
__device__ __forceinline__ void point_load(const double2* __restrict__ p, long long ld,
                                           long long n, bool in, double d[5], double f[9]) {
  double2 x[7];
#pragma unroll
  for (int q = 0; q < 7; ++q) x[q] = in ? p[q * ld + n] : make_double2(0., 0.);
  d[0] = x[0].x, d[1] = x[0].y, d[2] = x[1].x, d[3] = x[1].y, d[4] = x[2].x;
  f[0] = x[2].y, f[1] = x[3].x, f[2] = x[3].y, f[3] = x[4].x, f[4] = x[4].y;
  f[5] = x[5].x, f[6] = x[5].y, f[7] = x[6].x, f[8] = x[6].y;
}

__device__ __forceinline__ void point_store(double2* __restrict__ p, long long ld, long long n,
                                            const double d[5], const double f[9]) {
  p[n] = make_double2(d[0], d[1]);
  p[ld + n] = make_double2(d[2], d[3]);
  p[2 * ld + n] = make_double2(d[4], f[0]);
  p[3 * ld + n] = make_double2(f[1], f[2]);
  p[4 * ld + n] = make_double2(f[3], f[4]);
  p[5 * ld + n] = make_double2(f[5], f[6]);
  p[6 * ld + n] = make_double2(f[7], f[8]);
}

template <bool EU>
__device__ __forceinline__ void radius_cell(const double* __restrict__ v,
                                            const double* __restrict__ prim, long long ld,
                                            const double* __restrict__ vol,
                                            const double* __restrict__ cson,
                                            const double* __restrict__ rv, long long n,
                                            double q[6]) {
  if (EU) {
    const double norm = 1. / v[n];
    q[0] = v[ld + n] * norm;
    q[1] = v[2 * ld + n] * norm;
    q[2] = v[3 * ld + n] * norm;
    q[4] = q[5] = 0.;
  } else {
    q[0] = prim[n];
    q[1] = prim[ld + n];
    q[2] = prim[2 * ld + n];
    q[4] = rv[n];
    q[5] = vol[n];
  }
  q[3] = cson[n];
}

// The implicit coefficients of a real cell and its first Jacobi iterate, in
// one pass: the spectral radii of the cell's six faces (implimf_eu.f90:141-159,
// implimf_3d.f90:110-190; the lower faces stored, and the upper face at the
// end of each line), the diagonal in the reference's left-to-right chain --
// vol/dt, or for the Euler form vol*(1.5/dtpas + 1/dt), then the faces
// (implimf_eu.f90:82-85, 161-170, implimf_3d.f90:192-203), then 1.5*vol/dtpas
// for the Navier-Stokes form (implimf_3d.f90:213-224; dtpas > 0: dual time
// stepping) -- and d1 = -u / cd, the first sweep from a zero iterate, whose
// face terms are all zero (-u + 0.: +0 for u = 0, as those terms leave it).
// Bound by the loads of the seven cells (L1 and L2 hits); each interior face
// is evaluated by both its cells, which costs less than the launches and the
// re-reads of a seed, a face pass per direction, a diagonal and a first-sweep
// kernel (one launch instead of six): 10 us less of a 170 us iteration on
// 64x32x32 Euler cells, 13 us less of 263 us with Navier-Stokes, 15 us less
// of 2.33 ms on a 1.07M-cell Navier-Stokes channel.
// With p1 given (the point sweeps) the iterate goes there together with its
// flux increments instead.  ACC (the FP64 iteration): u is formed here from
// the face fluxes G, V (accumulate_cell) and stored, in place of a launch and a
// re-read: an iteration of 16x12x8 Euler cells 77.1 -> 74.6 us, of 64x32x32
// cells 121.0 -> 117.7 (Euler) and 159.1 -> 155.7 (limited Navier-Stokes), of
// 1.07M cells 2025 -> 2023.  With a
// cell's loads issued together (accumulate_cell) the FP32 coefficient kernel
// does the same.
template <bool EU, bool ACC>
__global__ void __launch_bounds__(kTile) k_impl_coefs(
    const Blk* __restrict__ blks, Space sp, double dtpas, const double* __restrict__ v,
    const double* __restrict__ prim, long long ld, const double* __restrict__ sn,
    const double* __restrict__ vol, const double* __restrict__ cson,
    const double* __restrict__ rv, const double* __restrict__ dt,
    const double* __restrict__ u, double* __restrict__ coefe, double* __restrict__ coefdiag,
    double* __restrict__ d1, double2* __restrict__ p1, const double* __restrict__ ps, Phys ph,
    int qfix, const double* __restrict__ G, const double* __restrict__ V,
    double* __restrict__ u_out) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  const long long n = cell_index(B, i, j, k);
  double d[5];
  if (ACC) {
    if (V)
      accumulate_cell<true>(B, i, j, k, n, G, V, ld, d);
    else
      accumulate_cell<false>(B, i, j, k, n, G, V, ld, d);
  }
  double q0[6];
  radius_cell<EU>(v, prim, ld, vol, cson, rv, n, q0);
  const double vn = vol[n];
  double c;
  if (EU)
    c = vn * ((dtpas > 0. ? 1.5 / dtpas : 0.) + 1. / dt[n]);
  else
    c = vn / dt[n];
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const long long inc = ninc_of(B, dir);
    const int p = dir == 0 ? i : (dir == 1 ? j : k);
    const double *s0 = sn_ptr(sn, B, dir, 0), *s1 = sn_ptr(sn, B, dir, 1),
                 *s2 = sn_ptr(sn, B, dir, 2);
    double ql[6], qu[6];
    radius_cell<EU>(v, prim, ld, vol, cson, rv, n - inc, ql);
    radius_cell<EU>(v, prim, ld, vol, cson, rv, n + inc, qu);
    const double cl = face_radius<EU>(q0, ql, s0[n], s1[n], s2[n]);
    const double cu = face_radius<EU>(qu, q0, s0[n + inc], s1[n + inc], s2[n + inc]);
    coefe[(long long)dir * ld + n] = cl;
    if (p == nd_of(B, dir) - 1) coefe[(long long)dir * ld + n + inc] = cu;
    c = c + cl;
    c = c + cu;
  }
  if (!EU && dtpas > 0.) c = c + 1.5 * vn / dtpas;
  coefdiag[n] = c;
  if (ACC) {
#pragma unroll
    for (int a = 0; a < 5; ++a) u_out[a * ld + n] = d[a];
  }
  if (!d1 && !p1) return;
#pragma unroll
  for (int a = 0; a < 5; ++a) d[a] = (-(ACC ? d[a] : u[a * ld + n]) + 0.) / c;
  if (d1) {
#pragma unroll
    for (int a = 0; a < 5; ++a) d1[a * ld + n] = d[a];
  } else {
    double f[9];
    point_df<EU>(v, prim, ps, ld, n, ph.gam1, ph.pinfl, qfix, d, f);
    point_store(p1, ld, n, d, f);
  }
}

// ---------------------------------------------------------------------------
// Point sweep: the Jacobi sweep of grids small enough for every array of the
// sweeps to stay in L2 (kPointEuler64 in cns_kernels.cuh has the lines and
// both sides' figures).  One thread per cell reads its own and its six
// neighbours' iterate and flux increment (d, f), evaluates the six faces and
// the new iterate with the expressions and order of the 2.5D sweep, then the
// new iterate's increment once, for the next sweep: no tile prologue, no
// plane-by-plane chain, every load of a cell independent of the others.  (On
// a large grid the stored increments would cost 72 B more a cell and sweep,
// and the k neighbours come from HBM again: the 2.5D sweep stays.)  Same
// inputs through the same operations as the 2.5D sweep: the same bits.
// (d, f) is packed as seven double2 [d0 d1][d2 d3][d4 f0][f1 f2][f3 f4]
// [f5 f6][f7 f8], component-major: a warp's loads are whole lines.
// ---------------------------------------------------------------------------
template <bool EU, bool LAST>
__global__ void __launch_bounds__(kTile) k_jacobi_point(
    const Blk* __restrict__ blks, Space sp, Phys ph, int qfix, long long ld,
    const double* __restrict__ u, const double* __restrict__ v,
    const double* __restrict__ prim, const double* __restrict__ ps,
    const double* __restrict__ sn, const double* __restrict__ coefe,
    const double* __restrict__ coefdiag, const double2* __restrict__ p_in,
    double2* __restrict__ p_out, double* __restrict__ d_out) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const Blk& B = blks[b];
  const long long n = cell_index(B, i, j, k);
  double d0[5], f0[9], w[5];
  point_load(p_in, ld, n, true, d0, f0);
#pragma unroll
  for (int a = 0; a < 5; ++a) w[a] = -u[a * ld + n];
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const long long inc = ninc_of(B, dir);
    const int p = dir == 0 ? i : (dir == 1 ? j : k);
    const double *s0 = sn_ptr(sn, B, dir, 0), *s1 = sn_ptr(sn, B, dir, 1),
                 *s2 = sn_ptr(sn, B, dir, 2);
    const double* ce = coefe + (long long)dir * ld;
    double dl[5], fl[9], du[5], fu[9], tl[5], tu[5];
    point_load(p_in, ld, n - inc, p > 1, dl, fl);
    point_load(p_in, ld, n + inc, p < nd_of(B, dir) - 1, du, fu);
    face_tn<double, EU>(d0, dl, f0, fl, s0[n], s1[n], s2[n], tl);
    face_tn<double, EU>(du, d0, fu, f0, s0[n + inc], s1[n + inc], s2[n + inc], tu);
    const double cel = ce[n], ceu = ce[n + inc];
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      w[a] = w[a] + tl[a] + cel * dl[a] + ceu * du[a];
      w[a] = w[a] - tu[a];
    }
  }
  const double cd = coefdiag[n];
  double d[5];
#pragma unroll
  for (int a = 0; a < 5; ++a) d[a] = w[a] / cd;
  if (LAST) {
#pragma unroll
    for (int a = 0; a < 5; ++a) d_out[a * ld + n] = d[a];
  } else {
    double f[9];
    point_df<EU>(v, prim, ps, ld, n, ph.gam1, ph.pinfl, qfix, d, f);
    point_store(p_out, ld, n, d, f);
  }
}

// standalone residual partials from stored arrays (rscpsv.f90 called with u0)
__global__ void __launch_bounds__(kTile) k_norm_partials(
    const Blk* __restrict__ blks, Space sp, long long ld,
    const double* __restrict__ u0, const double* __restrict__ v,
    const double* __restrict__ dt, double* normpart) {
  int b, i, j, k;
  const bool valid = space_elem_sync(sp, threadIdx.x, b, i, j, k);
  double res[5] = {0., 0., 0., 0., 0.};
  if (valid) {
    const long long n = cell_index(blks[b], i, j, k);
#pragma unroll
    for (int a = 0; a < 5; ++a) res[a] = (v[a * ld + n] - u0[a * ld + n]) / dt[n];
  }
  norm_tile_reduce(res, valid, normpart + (long long)(sp.tile0 + blockIdx.x) * 15);
}

// Sums of the tile partials in a fixed order, and the rscpsv.f90:79-150
// combination over blocks, in one launch.  CTA (x, y) sums the tiles
// x * kNormChunk .. of block y: 32 rows of 15 lanes walk the partials
// [tile][15] (consecutive threads read consecutive values), then, turned round
// in shared memory, a tree over the rows of column q in warp q; the last CTA to
// finish combines the blocks the same way and resets the counter.  Latency
// bound (a megabyte of partials on a million cells): 13 -> 8.5 us on 64x32x32
// cells, 30 -> 10 us on 1.07M cells in three blocks, against one CTA a block
// and a combining kernel (cold).  The trees are shuffles: with one barrier in
// place of eighteen and the partials' own tree (norm_tile_reduce) an iteration
// of 16x12x8 cells takes 74.6 -> 71.5 us.
constexpr int kNormRows = 32;

// tree over the lanes (rows) of column q; the result is lane 0's
__device__ __forceinline__ double norm_tree(int q, double x) {
#pragma unroll
  for (int s = kNormRows / 2; s > 0; s >>= 1)
    x = norm_add(q, x, __shfl_down_sync(0xffffffffu, x, s));
  return x;
}

__global__ void __launch_bounds__(kNormRows * 15) k_norms(
    const Blk* __restrict__ blks, const int* __restrict__ blk_tile0,
    const double* __restrict__ normpart, double* __restrict__ chunksum, int* counter,
    double* norms) {
  __shared__ double red[kNormRows * 15];
  __shared__ int last;
  const int t1 = blk_tile0[blockIdx.y + 1];
  const int c0 = blk_tile0[blockIdx.y] + (int)blockIdx.x * kNormChunk;
  const int c1 = min(c0 + kNormChunk, t1);
  pdl_sync();
  double x = 0.;
#pragma unroll 8
  for (int t = c0 + (int)threadIdx.x / 15; t < c1; t += kNormRows)
    x = norm_add(threadIdx.x % 15, x, normpart[(long long)t * 15 + threadIdx.x % 15]);
  red[threadIdx.x] = x;
  __syncthreads();
  const int q = threadIdx.x / 32, row = threadIdx.x % 32;
  x = norm_tree(q, red[row * 15 + q]);
  const int ctas = gridDim.x * gridDim.y;
  if (ctas > 1) {
    const long long chunk = (long long)blockIdx.y * gridDim.x + blockIdx.x;
    if (row == 0) {
      chunksum[chunk * 15 + q] = x;
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1) == ctas - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) *counter = 0;
  }
  // blocks row, row + 32, ... (rscpsv.f90: nmax * norm1, nmax * norm2^2, max)
  double g = 0., npts = 0.;
  for (int b = row; b < (int)gridDim.y; b += kNormRows) {
    const Blk& B = blks[b];
    const double nmax = (double)((long long)(B.ni - 1) * (B.nj - 1) * (B.nk - 1));
    const double coef = 1. / nmax;
    double s = 0.;
    if (ctas == 1) s = x;
    else
      for (int c = 0; c < (int)gridDim.x; ++c)
        s = norm_add(q, s, __ldcg(chunksum + ((long long)b * gridDim.x + c) * 15 + q));
    if (q < 5)
      s = nmax * (coef * s);
    else if (q < 10)
      s = nmax * sq(sqrt(coef * s));
    g = norm_add(q, g, s);
    npts += nmax;
  }
  const double tot = norm_tree(q, g), n = norm_tree(0, npts);
  if (row == 0) norms[q] = q < 5 ? tot / n : (q < 10 ? sqrt(tot / n) : tot);
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

cudaError_t launch_zpres(const Blk* blks, Space sp, Phys ph, int with_mu,
                         const double* v, long long ld, double* ps, double* temp,
                         double* cson, double* mu, int* status, cudaStream_t st) {
  if (sp.ntiles > 0)
    pdl(k_zpres, grid_of(sp), kTile, 0, st)(blks, sp, ph, with_mu, v, ld, ps, temp,
                                           cson, mu, status);
  return cudaGetLastError();
}

cudaError_t launch_zvismo(const Blk* blks, Space sp, Phys ph, double* mu,
                          const double* temp, int* status, cudaStream_t st) {
  if (sp.ntiles > 0)
    pdl(k_zvismo, grid_of(sp), kTile, 0, st)(blks, sp, ph, mu, temp, status);
  return cudaGetLastError();
}

cudaError_t launch_prim(long long n0, long long n1, const double* v, long long ld,
                        double* prim, cudaStream_t st) {
  if (n1 > n0)
    pdl(k_prim<false>, (int)((n1 - n0 + 255) / 256), 256, 0, st)(n0, n1, v, ld, prim, nullptr,
                                                                PrimShadow{});
  return cudaGetLastError();
}

cudaError_t launch_prim_shadow(long long ncells, const double* v, long long ld, double* prim,
                               const double* ps, const PrimShadow& sh, cudaStream_t st) {
  if (ncells > 0)
    pdl(k_prim<true>, (int)((ncells + 255) / 256), 256, 0, st)(0, ncells, v, ld, prim, ps, sh);
  return cudaGetLastError();
}

// chrono.f90:113-151 (kdtl = 0): the smallest local time step over the real
// cells of every block, min(dt1min, it) everywhere, and the reference's stop
// when it is below dt1min as status bit 2.  Min is exact in any order.
__global__ void __launch_bounds__(kTile) k_dt_partials(const Blk* __restrict__ blks, Space sp,
                                                       const double* __restrict__ dt,
                                                       double* __restrict__ part) {
  pdl_sync();
  int b, i, j, k;
  double x = CUDART_INF;
  if (space_elem(sp, threadIdx.x, b, i, j, k)) x = dt[cell_index(blks[b], i, j, k)];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmin(x, __shfl_xor_sync(0xffffffffu, x, o));
  __shared__ double wm[kTile / 32];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = wm[0];
    for (int q = 1; q < kTile / 32; ++q) m = fmin(m, wm[q]);
    part[blockIdx.x] = m;
  }
}

__global__ void __launch_bounds__(256) k_dt_reduce(const double* __restrict__ part, int n,
                                                  double dt1min, double* __restrict__ out,
                                                  int* status) {
  pdl_sync();
  double x = CUDART_INF;
  for (int q = threadIdx.x; q < n; q += blockDim.x) x = fmin(x, part[q]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmin(x, __shfl_xor_sync(0xffffffffu, x, o));
  __shared__ double wm[8];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = wm[0];
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) m = fmin(m, wm[q]);
    const double dtmin = fmin(dt1min, m);
    if (dtmin < dt1min) atomicOr(status, 2);
    *out = dtmin;
  }
}

__global__ void __launch_bounds__(256) k_dt_set(long long ncells, const double* __restrict__ v,
                                               double* __restrict__ dt) {
  pdl_sync();
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n < ncells) dt[n] = *v;
}

cudaError_t launch_chronos(const Blk* blks, Space sp, Phys ph, Scheme sc,
                           const double* mu, const double* mut, const double* v,
                           long long ld, double* dt, const double* sn,
                           const double* vol, const double* cson, cudaStream_t st) {
  if (sp.ntiles > 0)
    pdl(k_chronos, grid_of(sp), kTile, 0, st)(blks, sp, ph, sc, mu, mut, v, ld, dt,
                                             sn, vol, cson);
  return cudaGetLastError();
}

cudaError_t launch_zpres_chronos(const Blk* blks, Space sp, Phys ph, Scheme sc,
                                 const double* v, long long ld, double* ps, double* temp,
                                 double* cson, double* mu, const double* mut, double* dt,
                                 const double* sn, const double* vol, int* status,
                                 cudaStream_t st) {
  if (sp.ntiles > 0)
    pdl(k_zpres_chronos, grid_of(sp), kTile, 0, st)(blks, sp, ph, sc, v, ld, ps, temp, cson, mu,
                                                   mut, dt, sn, vol, status);
  return cudaGetLastError();
}

cudaError_t launch_dt_global(const Blk* blks, Space cells, long long ncells, double dt1min,
                             double* dt, double* part, double* scalar, int* status,
                             cudaStream_t st) {
  if (cells.ntiles == 0) return cudaSuccess;
  pdl(k_dt_partials, grid_of(cells), kTile, 0, st)(blks, cells, dt, part);
  pdl(k_dt_reduce, 1, 256, 0, st)(part, cells.ntiles, dt1min, scalar, status);
  pdl(k_dt_set, (int)((ncells + 255) / 256), 256, 0, st)(ncells, scalar, dt);
  return cudaGetLastError();
}

cudaError_t launch_rbord(const Bnd& bd, Phys ph, double* v, long long ld,
                         double* ps, double* temp, double* cson, long long n_idd_ent,
                         const long long* idd_ents, unsigned* idd_work, cudaStream_t st) {
  if (bd.nlist > 0)
    pdl(k_rbord, (int)((bd.nlist + 255) / 256), 256, 0, st)(bd, ph, v, ld, ps, temp, cson,
                                                            idd_work);
  if (n_idd_ent > 0) {
    const int g = (int)((n_idd_ent + 63) / 64);
    pdl(k_clidd_count, g, 64, 0, st)(bd, ph, idd_ents, n_idd_ent, v, ld, idd_work);
    pdl(k_clidd_apply, g, 64, 0, st)(bd, ph, idd_ents, n_idd_ent, v, ld, ps, temp, cson,
                                     idd_work);
  }
  return cudaGetLastError();
}

cudaError_t launch_tau_ghosts(const Bnd& bd, double* tau, long long ld,
                              cudaStream_t st) {
  if (bd.nlist > 0)
    pdl(k_tau_ghosts, (int)((bd.nlist + 255) / 256), 256, 0, st)(bd, tau, ld);
  return cudaGetLastError();
}

cudaError_t launch_grad(const Blk* blks, Space sp, Phys ph, const double* v,
                        const double* prim, long long ld, const double* mu,
                        const double* mut, double* tau, const double* sn,
                        const double* vol, const double* temp, double* rv,
                        cudaStream_t st) {
  if (sp.ntiles > 0)
    pdl(k_grad, grid_of(sp), kTile, 0, st)(blks, sp, ph, v, prim, ld, mu, mut, tau, sn,
                                          vol, temp, rv);
  return cudaGetLastError();
}

template <>
cudaError_t launch_ratio_t<double>(const Blk* blks, const SpaceBuf* lines, int l0,
                                   const double* v, const double* prim, long long ld,
                                   const double* ps, double* R, cudaStream_t st) {
  return ratio_launch<double>(blks, lines, l0, v, prim, ld, ps, R, st);
}

cudaError_t launch_residual_fused(const Blk* blks, Tiles tl, Phys ph, Scheme sc, const double* v,
                                  const double* prim, long long ld, const double* ps,
                                  const double* tau, const double* sn, const double* R,
                                  double* u, float* u32, cudaStream_t st) {
  return residual_fused_dispatch<double>(blks, tl, ph, sc, v, prim, ld, ps, tau, sn, R, u, u32,
                                         st);
}

template <>
cudaError_t launch_face_flux_t<double>(const Blk* blks, const SpaceBuf* faces, int l0,
                                       Phys ph, Scheme sc, const double* v,
                                       const double* prim, long long ld,
                                       const double* ps, const double* tau,
                                       const double* sn, const double* R, double* G,
                                       cudaStream_t st, double* V) {
  return face_flux_dispatch(blks, faces, l0, ph, sc, v, prim, ld, ps, tau, sn, R, G, V, st);
}

template <>
cudaError_t launch_accumulate_t<double>(const Blk* blks, Space sp, const double* G,
                                        long long ld, const double* corr, double* u,
                                        float* u32, cudaStream_t st, const double* V) {
  if (sp.ntiles > 0)
    pdl(k_accumulate<double>, grid_of(sp), kTile, 0, st)(blks, sp, G, ld, corr, u, u32, V);
  return cudaGetLastError();
}

template <>
cudaError_t launch_jacobi_25d_t<double>(const Blk* blks, Tiles tl, Phys ph, int qfix, int eu,
                                        long long ld, const double* u, const double* v,
                                        const double* prim, const double* ps, const double* sn,
                                        const double* coefe, const double* coefdiag,
                                        const double* d_in, double* d_out, cudaStream_t st) {
  return jacobi_25d_dispatch<double>(blks, tl, ph, qfix, eu, ld, u, v, prim, ps, sn, coefe,
                                        coefdiag, d_in, d_out, st);
}

int jacobi_25d_blocks_per_sm(int ti, int tj, int eu) {
  int n = 0;
#define CNS_OCC1(A, B, E)                                                                   \
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_jacobi_25d<double, E, A, B>, A * B, \
                                                jacobi_25d_smem<A, B, double, E>())
#define CNS_OCC(A, B)                                  \
  if (ti == A && tj == B) {                            \
    if (eu) CNS_OCC1(A, B, true);                      \
    else CNS_OCC1(A, B, false);                        \
    return n;                                          \
  }
  CNS_OCC(32, 4)
  CNS_OCC(32, 8)
  CNS_OCC(16, 8)
  CNS_OCC(16, 16)
#undef CNS_OCC
#undef CNS_OCC1
  return 0;
}

cudaError_t init_jacobi_25d() {
  cudaError_t e = jacobi_25d_attr<double>();
  if (e == cudaSuccess) e = init_jacobi_25d_float();
  return e;
}

// the FP64 sweeps after the first, whose iterate the coefficient kernel
// writes into dpp[0]: 2.5D-blocked with the increments evaluated by the
// reference expressions (bit-identical to storing them,
// implimf_3d.f90:222-466)
template <>
cudaError_t launch_sweeps_t<double>(const Blk* blks, Tiles tl, Phys ph, Scheme sc, int eu,
                                    int lmx, long long ld, const double* u, const double* v,
                                    const double* prim, const double* ps, const double* sn,
                                    const double* coefe, const double* coefdiag,
                                    double* const dpp[2], int* cur_out, cudaStream_t st) {
  int cur = 0;
  if (lmx == 0) {
    cudaError_t e0 = cudaMemsetAsync(dpp[0], 0, sizeof(double) * 5 * ld, st);
    if (e0 != cudaSuccess) return e0;
  }
  const int q = eu ? sc.qfix_dfez : 0;
  for (int ls = 2; ls <= lmx; ++ls) {
    cudaError_t e1 = launch_jacobi_25d_t<double>(blks, tl, ph, q, eu, ld, u, v, prim, ps, sn,
                                                 coefe, coefdiag, dpp[cur], dpp[1 - cur], st);
    if (e1 != cudaSuccess) return e1;
    cur = 1 - cur;
  }
  *cur_out = cur;
  return cudaGetLastError();
}

template <>
cudaError_t launch_update_t<double>(const Blk* blks, Space cells, long long ld,
                                    const double* d, double* v, const double* dt,
                                    double* d_out, double* normpart, cudaStream_t st) {
  if (cells.ntiles > 0)
    pdl(k_update<double>, grid_of(cells), kTile, 0, st)(blks, cells, ld, d, v, dt, d_out,
                                                       normpart);
  return cudaGetLastError();
}

cudaError_t launch_implicit_coefficients(const Blk* blks, Space cells, Phys ph, int eu,
                                         double dtpas, const double* dt, const double* v,
                                         const double* prim, const double* mu,
                                         const double* mut, const double* sn,
                                         const double* vol, const double* cson, double* u,
                                         int sum_faces, const double* V, int rv_done,
                                         double* d1, double2* p1, const double* ps, int qfix,
                                         Work& w, cudaStream_t st) {
  if (cells.ntiles == 0) return cudaSuccess;
  const int g = grid_of(cells);
  if (!eu && !rv_done) pdl(k_impl_rv, g, kTile, 0, st)(blks, cells, ph, v, mu, mut, w.rv);
  auto run = [&](auto kernel) {
    pdl(kernel, g, kTile, 0, st)(blks, cells, dtpas, v, prim, w.ld, sn, vol, cson, w.rv, dt, u,
                                 w.coefe, w.coefdiag, d1, p1, ps, ph, qfix, w.G, V, u);
  };
  if (sum_faces)
    eu ? run(k_impl_coefs<true, true>) : run(k_impl_coefs<false, true>);
  else
    eu ? run(k_impl_coefs<true, false>) : run(k_impl_coefs<false, false>);
  return cudaGetLastError();
}

// sweeps 2..lmx of a small grid (the first iterate is in w.point_iterate(0));
// the final iterate in w.dpp[0]
static cudaError_t point_sweeps64(const Blk* blks, Space cells, Phys ph, int qfix, int eu,
                                  int lmx, const double* u, const double* v, const double* ps,
                                  const double* sn, Work& w, cudaStream_t st) {
  const int g = grid_of(cells);
  auto run = [&](auto kernel, const double2* in, double2* out) {
    pdl(kernel, g, kTile, 0, st)(blks, cells, ph, qfix, w.ld, u, v, w.prim, ps, sn, w.coefe,
                                w.coefdiag, in, out, w.dpp[0]);
  };
  for (int ls = 2; ls <= lmx; ++ls) {
    const double2* in = w.point_iterate(ls & 1);
    double2* out = w.point_iterate((ls & 1) ^ 1);
    if (eu)
      ls < lmx ? run(k_jacobi_point<true, false>, in, out)
               : run(k_jacobi_point<true, true>, in, out);
    else
      ls < lmx ? run(k_jacobi_point<false, false>, in, out)
               : run(k_jacobi_point<false, true>, in, out);
  }
  return cudaGetLastError();
}

cudaError_t launch_implicit(const Blk* blks, Space cells, Tiles tl, Phys ph, Scheme sc, int eu,
                            int lmx, double* u, int sum_faces, const double* V, const double* dt,
                            double* v, double* d_out, const double* mu, const double* mut,
                            const double* sn, const double* vol, const double* ps,
                            const double* cson, int rv_done, Work& w, int want_norms,
                            cudaStream_t st) {
  const long long ld = w.ld;
  if (cells.ntiles == 0) return cudaSuccess;
  const int qfix = eu ? sc.qfix_dfez : 0;
  const bool point = (eu ? w.point_eu : w.point_ns) && lmx >= 2;
  // dtpas > 0: dual time stepping with physical step dtpas
  cudaError_t e = launch_implicit_coefficients(
      blks, cells, ph, eu, sc.kfmg == 3 ? sc.dt1min : 0., dt, v, w.prim, mu, mut, sn, vol, cson,
      u, sum_faces, V, rv_done, lmx >= 1 && !point ? w.dpp[0] : nullptr,
      point ? w.point_iterate(0) : nullptr, ps, qfix, w, st);
  int cur = 0;
  if (e == cudaSuccess && point)
    e = point_sweeps64(blks, cells, ph, qfix, eu, lmx, u, v, ps, sn, w, st);
  else if (e == cudaSuccess)
    e = launch_sweeps_t<double>(blks, tl, ph, sc, eu, lmx, ld, u, v, w.prim, ps, sn, w.coefe,
                                w.coefdiag, w.dpp, &cur, st);
  if (e == cudaSuccess)
    e = launch_update_t<double>(blks, cells, ld, w.dpp[cur], v, dt, d_out,
                                want_norms ? w.normpart : nullptr, st);
  return e;
}

// sch_dual.f90:18-52 / sch_dual2.f90:18-52: u += vol*dti*(fact*v + ptdual)
// on the real cells (the physical time term of dual time stepping); u32:
// the single-precision copy of u the FP32 sweeps read, refreshed
__global__ void __launch_bounds__(kTile) k_dual(const Blk* __restrict__ blks, Space sp,
                                                long long ld, double fact, double dti,
                                                const double* __restrict__ v,
                                                const double* __restrict__ vol,
                                                const double* __restrict__ ptdual,
                                                double* __restrict__ u, float* __restrict__ u32) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const long long n = cell_index(blks[b], i, j, k);
  const double c0 = vol[n] * dti;
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    const double r = u[a * ld + n] + c0 * (fact * v[a * ld + n] + ptdual[a * ld + n]);
    u[a * ld + n] = r;
    if (u32) u32[a * ld + n] = (float)r;
  }
}

// the physical-step arrays on the real cells: mode 0 = sch_duin.f90 after
// utinia.f90:140-160 (vdual = vdual1 = vdual2 = v, ptdual = -vdual); mode 1
// = sch_duup.f90 (vdual1 = vdual, vdual = v, ptdual = -2 vdual + 0.5 vdual1);
// mode 2 = sch_duup2.f90 (vdual2 = vdual1, vdual1 = vdual, vdual = v,
// ptdual = -3 vdual + 1.5 vdual1 - vdual2/3)
__global__ void __launch_bounds__(kTile) k_dual_update(const Blk* __restrict__ blks, Space sp,
                                                       long long ld, int mode,
                                                       const double* __restrict__ v,
                                                       double* ptdual, double* vdual,
                                                       double* vdual1, double* vdual2) {
  int b, i, j, k;
  if (!space_elem_sync(sp, threadIdx.x, b, i, j, k)) return;
  const long long n = cell_index(blks[b], i, j, k);
  const double c13 = 1. / 3.;
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    const long long q = a * ld + n;
    if (mode == 0) {
      vdual[q] = v[q];
      vdual1[q] = v[q];
      vdual2[q] = v[q];
      ptdual[q] = -vdual[q];
    } else if (mode == 1) {
      vdual1[q] = vdual[q];
      vdual[q] = v[q];
      ptdual[q] = -2. * vdual[q] + 0.5 * vdual1[q];
    } else {
      vdual2[q] = vdual1[q];
      vdual1[q] = vdual[q];
      vdual[q] = v[q];
      ptdual[q] = -3. * vdual[q] + 1.5 * vdual1[q] - c13 * vdual2[q];
    }
  }
}

cudaError_t launch_dual(const Blk* blks, Space cells, long long ld, double fact, double dti,
                        const double* v, const double* vol, const double* ptdual, double* u,
                        float* u32, cudaStream_t st) {
  if (cells.ntiles > 0)
    pdl(k_dual, cells.ntiles, kTile, 0, st)(blks, cells, ld, fact, dti, v, vol, ptdual, u, u32);
  return cudaGetLastError();
}

cudaError_t launch_dual_update(const Blk* blks, Space cells, long long ld, int mode,
                               const double* v, double* ptdual, double* vdual, double* vdual1,
                               double* vdual2, cudaStream_t st) {
  if (cells.ntiles > 0)
    pdl(k_dual_update, cells.ntiles, kTile, 0, st)(blks, cells, ld, mode, v, ptdual, vdual,
                                                  vdual1, vdual2);
  return cudaGetLastError();
}

cudaError_t launch_norm_partials(const Blk* blks, Space cells, long long ld,
                                 const double* u0, const double* v,
                                 const double* dt, double* normpart,
                                 cudaStream_t st) {
  if (cells.ntiles > 0)
    pdl(k_norm_partials, cells.ntiles, kTile, 0, st)(blks, cells, ld, u0, v, dt, normpart);
  return cudaGetLastError();
}

cudaError_t launch_norm_finalize(const Blk* blks, const int* blk_tile0_dev, int nblk, int chunks,
                                 const double* normpart, double* chunksum, int* counter,
                                 double* norms, cudaStream_t st) {
  pdl(k_norms, dim3(chunks, nblk), kNormRows * 15, 0, st)(blks, blk_tile0_dev, normpart, chunksum,
                                                         counter, norms);
  return cudaGetLastError();
}

}  // namespace cns
