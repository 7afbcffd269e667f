// hy_core.cuh -- device arithmetic of the unsplit hydro update.
//
// Templated on the reconstruction/flux type R (double for the FP64 paths,
// float for the mixed path).  The expressions keep the evaluation order of
// the Fortran they restate (paths inside mbdevpl/FLASH5,
// source/physics/Hydro/HydroMain/unsplit unless stated), so that the FP64
// variant compiled without FMA contraction reproduces an IEEE evaluation of
// the reference arithmetic.  The hydro eigenvectors are sparse
// (OnlyHydro/hy_eigenVector.F90:114-151); the dot products below add only
// their non-zero terms, in index order, which gives the same values as the
// dense sums (the skipped terms are exact zeros).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "exact_rs.cuh"

namespace fhy {

// primitive slots of UHD.h:374-383 (HY_DENS..HY_EINT), 0-based
enum { HD = 0, HVX = 1, HVY = 2, HVZ = 3, HP = 4, HGC = 5, HGE = 6, HEI = 7 };
// flux slots of OnlyHydro/Config:6-13, 0-based
enum { FDENS = 0, FXMOM, FYMOM, FZMOM, FENER, FPRES, FEINT, FVOLU, NFLX = 8 };

// status bits (include/flash_hy.h)
constexpr unsigned ST_NEG_SOUND = 1u << 0;
constexpr unsigned ST_NEWTON = 1u << 2;
constexpr unsigned ST_NAN = 1u << 3;

struct DevParams {
  int ndim;
  int nbx, nby, nbz;          // blocks per axis of the uniform level
  int bc[6];
  int use_flattening, use_steepening, char_limiting, limiter, use_aux_eint, use_ctu;
  int riemann;                // 4 = HLLC, 100 = exact
  int learned;                // exact solver: MLP initial guess
  double lim_beta, gamma, gam1inv, ggprodinv, abar, smalle, smlrho, eswitch, tiny, cfl;
  double del[3];
  double dt;
  const double *dt_dev;       // when set, dt is read from device memory (graph-replayed steps)
  const int *blk_at;          // block index at block coordinates
  const int *blk_nbr;         // uniform grids: face neighbours of each block [b][x-, x+, y-, y+, z-, z+]
                              // (-1 beyond a non-periodic boundary or absent from the grid)
  const int *blk_coord;       // 3 ints per block
  const int *blk_list;        // optional list of blocks to update (NULL = all)
  const double *s_in[5];      // dens, velx, vely, velz, eint (block-major SoA)
  double *s_out[5];
  unsigned *status;
  const void *mlp;            // learned-guess network, xrs::MlpPacked (exact solver; NULL = off)
  double *harvest;            // optional face-state sample, [7][harvest_cap] (dl,ul,pl,dr,ur,pr,gamma)
  unsigned long long *harvest_n;
  long long harvest_cap;
  unsigned harvest_mask;      // a face is kept when its hash & mask == 0
  double rs_tol;              // exact solver: relative tolerance of p*
  int rs_max_iter;
  // AMR hierarchy (blk_level == NULL: one uniform level)
  const int *blk_level;       // level of each node
  const int *leaf;            // 1 for the leaves
  const int *parent;          // parent node, -1 on level 1
  const int *slot;            // leaf slot (guard buffer, sig scratch, flux register) / parent slot (halo)
  const int *at;              // node by (level, block coordinates), -1 where the level is not refined
  int at_off[17];
  int at_ext[17][3];
  double *lh;                 // leaf guard cells after the EOS: [slot][5][(N+8)^d]
  double *gp;                 // parent guard-inclusive blocks: [slot][6][(N+8)^d] (rho, v, e, E)
  double *pe;                 // parents' restricted specific total energy [node * NCB + cell]
  double *freg;               // fine-face fluxes at fine/coarse faces: [leaf slot][2 ndim][faces][8]
  // split step (hy_computeFluxes with Uout disassociated, hy_updateSolution):
  // 0 = fused step, 1 = store the fluxes and update, 2 = store the fluxes
  // only, 3 = update from the stored fluxes
  int fmode;
  double *fstore;             // [block][ndim][8 x faces (FLASH flx order) + n+1/2 pressure sum per cell]
  // species and mass scalars (nsp > 0; the first nspec are renormalised):
  // [nsp][ncells] block-major SoA interiors, double-buffered like s_in/s_out.
  // The hydro direction kernels leave for them, per launch slot and
  // direction in the line-cell order of DirGeom, the face mass flux
  // (sp_mf), whether the 3D CTU stage fell back to first order (sp_fb) and
  // the flattening coefficient (sp_flat).
  int nsp, nspec;
  const double *sp_in;
  double *sp_out;
  double *sp_mf;
  unsigned char *sp_fb;
  double *sp_flat;            // flattening coefficient of each line cell (same layout)
  // species on AMR hierarchies: guard cells of the leaves [leaf slot][nsp]
  // [halo], guard-inclusive copies of the parents [parent slot][nsp][halo],
  // the species flux register [nsp][leaf slot][2 ndim][faces]
  double *sp_lh, *sp_gp, *sp_freg;
  size_t sp_ncells;           // stride of the species arrays
  size_t sp_freg_stride;      // doubles per species in sp_freg
  // split step: species face fluxes F_dens * X per block, direction and
  // species, in the face order of the hydro flux store [block][dir][nsp][faces]
  double *sp_fstore;
  // the exact Riemann solver's gas constants (xrs::gas_of(gamma), host-side)
  xrs::Gas gas;
};

// Cell sizes of block b: level-1 deltas scaled by 2^(1-level) (exact).
__device__ __forceinline__ void blk_deltas(const DevParams &P, int b, double del[3]) {
  const double s = P.blk_level ? ldexp(1.0, 1 - P.blk_level[b]) : 1.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) del[d] = d < P.ndim ? P.del[d] * s : P.del[d];
}

__device__ __forceinline__ int at_node(const DevParams &P, int l, int x, int y, int z) {
  return P.at[P.at_off[l] + (z * P.at_ext[l][1] + y) * P.at_ext[l][0] + x];
}

template <class R> __device__ __forceinline__ R rmax(R a, R b) { return a > b ? a : b; }
template <class R> __device__ __forceinline__ R rmin(R a, R b) { return a < b ? a : b; }

// x / b rounded to nearest, from rb = RN(1 / b) (Markstein's theorem,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34 (1990): q0 = RN(x rb) is within an ulp of
// x / b, the remainder x - q0 b is exact with an FMA, and
// RN(q0 + (x - q0 b) rb) = RN(x / b)).  Outside the exponent range where
// the remainder cannot underflow or the product overflow (zeros,
// subnormals, infinities and NaN included) it divides.  Equal to x / b in
// every bit: a CPU test checks the method on random and special operands,
// and the FP64 GPU parity tests compare the kernels that use it with the
// oracle's divisions.
__device__ __forceinline__ double div_rn(double x, double b, double rb) {
  const double q0 = x * rb;
  const double a = fabs(q0), ax = fabs(x);
  if (a > 0x1p-960 && a < 0x1p1000 && ax > 0x1p-960 && ax < 0x1p1000) return fma(fma(-q0, b, x), rb, q0);
  return x / b;
}

// ---------------------------------------------------------------------------
// Branch-free correctly rounded FP64 division for the direction kernels: the
// compiler's division ends its basic block (a call for operands outside the
// fast path), which keeps the scheduler from overlapping the forty divisions
// of a cell.  From the mathematics of Newton's iteration and Markstein's
// theorems (IBM J. Res. Dev. 34 (1990)):
//   y1 = y0 (1 + e + e^2), e = 1 - b y0, from the 20-bit seed of
//        rcp.approx.ftz.f64: within an ulp of 1 / b;
//   y  = y1 + y1 (1 - b y1) with exact residual: RN(1 / b) unless the
//        significand of b is all ones;
//   q0 = RN(x y); q = q0 - y (q0 b - x) with exact residual: RN(x / b), and
//        for b > 0 the sign of a zero x (the residual's sign is chosen so).
// They hold where nothing leaves the normal numbers: `bad` is raised unless
// b and x (or x = 0) lie in [2^-500, 2^500) in magnitude, and for a divisor
// of all ones; the caller then evaluates the cell again with plain
// divisions.  tests/test_div_rn.py checks the method against IEEE division.
// ---------------------------------------------------------------------------
struct Rcp { double b, r; };               // divisor (> 0) and RN(1 / b)
// plain (Fast = false): the compiler's divisions
template <bool Fast> struct Arith;
template <> struct Arith<true> {
  bool bad = false;
  __device__ __forceinline__ void check(double x, bool when = true) {            // x = 0 or in range
    const unsigned u = (unsigned)__double2hiint(x) & 0x7fffffffu;
    bad |= u - 0x20B00000u >= 0x3E800000u && (u | (unsigned)__double2loint(x)) != 0u && when;
  }
  __device__ __forceinline__ Rcp rcp(double b, bool when = true) {
    const unsigned hi = (unsigned)__double2hiint(b), u = hi & 0x7fffffffu;
    bad |= (u - 0x20B00000u >= 0x3E800000u || (((hi | 0xfff00000u) & (unsigned)__double2loint(b)) == 0xffffffffu)) && when;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;\n" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return Rcp{b, fma(y, fma(-b, y, 1.0), y)};
  }
  __device__ __forceinline__ double by(double x, const Rcp &d, bool when = true) {
    check(x, when);
    const double q0 = x * d.r;
    return fma(-fma(q0, d.b, -x), d.r, q0);
  }
  __device__ __forceinline__ double div(double x, double b, bool when = true) { return by(x, rcp(b, when), when); }
  // x / B for a small integer constant
  template <int B> __device__ __forceinline__ double byc(double x) { return by(x, Rcp{(double)B, 1.0 / B}); }
};
template <> struct Arith<false> {
  static constexpr bool bad = false;
  __device__ __forceinline__ Rcp rcp(double b, bool = true) { return Rcp{b, 1.0 / b}; }
  __device__ __forceinline__ double by(double x, const Rcp &d, bool = true) { return x / d.b; }
  __device__ __forceinline__ double div(double x, double b, bool = true) { return x / b; }
  template <int B> __device__ __forceinline__ double byc(double x) { return x / (double)B; }
};
__device__ __forceinline__ double rsign(double a, double b) { return copysign(fabs(a), b); }
__device__ __forceinline__ float rsign(float a, float b) { return copysignf(fabsf(a), b); }
__device__ __forceinline__ double rabs(double a) { return fabs(a); }
__device__ __forceinline__ float rabs(float a) { return fabsf(a); }
__device__ __forceinline__ double rsqrt_(double a) { return sqrt(a); }
__device__ __forceinline__ float rsqrt_(float a) { return sqrtf(a); }

// velocity slots of the normal / first / second transverse direction
// (hy_eigenVector.F90:75-89)
template <int DIR> struct Slots;
template <> struct Slots<1> { static constexpr int v1 = HVX, v2 = HVY, v3 = HVZ; };
template <> struct Slots<2> { static constexpr int v1 = HVY, v2 = HVZ, v3 = HVX; };
template <> struct Slots<3> { static constexpr int v1 = HVZ, v2 = HVX, v3 = HVY; };

// ---------------------------------------------------------------------------
// slope limiters, hy_slopeLimiters.F90:38-60; hy_TVDslope.F90:213-245
// ---------------------------------------------------------------------------
template <class R> __device__ __forceinline__ R lim_vanleer(R a, R b) {
  if (a * b <= R(0)) return R(0);
  return R(2) * a * b / (a + b);
}
template <class R> __device__ __forceinline__ R lim_mc(R a, R b) {
  R m = rabs(a), t = R(.25) * rabs(a + b);
  if (t < m) m = t;
  if (rabs(b) < m) m = rabs(b);
  return (rsign(R(1), a) + rsign(R(1), b)) * m;
}
template <class R> __device__ __forceinline__ R lim_minmod(R a, R b) {
  R m = rabs(a) < rabs(b) ? rabs(a) : rabs(b);
  return R(.5) * (rsign(R(1), a) + rsign(R(1), b)) * m;
}
template <class R> __device__ __forceinline__ R limit2(int lim, R beta, R d1, R d2) {
  switch (lim) {
    case 1: return lim_minmod(d1, d2);
    case 2: return lim_mc(d1, d2);
    case 4: return lim_vanleer(d1, d2);
    case 5:
      if (d2 > R(0)) return rmax(R(0), rmax(rmin(beta * d1, d2), rmin(d1, beta * d2)));
      return rmin(R(0), rmin(rmax(beta * d1, d2), rmax(d1, beta * d2)));
  }
  return R(0);
}

// ---------------------------------------------------------------------------
// eigen system in primitive variables: hy_eigenParameters.F90:71-89,
// hy_eigenValue.F90:46-50, OnlyHydro/hy_eigenVector.F90:95-152
// ---------------------------------------------------------------------------
template <class R> struct Eig {
  R lam[5];
  R cf, ahinv, a2inv, lp, rho, rp;
};

// wave speeds along DIR of a cell with sound speed e.cf
template <class R, int DIR>
__device__ __forceinline__ void speeds(const R *V, Eig<R> &e) {
  const R un = V[Slots<DIR>::v1];
  e.lam[0] = un - e.cf; e.lam[1] = un; e.lam[2] = un; e.lam[3] = un; e.lam[4] = un + e.cf;
}

template <class R, int DIR>
__device__ __forceinline__ void eigen(const R *V, Eig<R> &e, unsigned &st) {
  R a2 = V[HGC] * V[HP] / V[HD];
  if (a2 <= R(0)) st |= ST_NEG_SOUND;
  R cf = rsqrt_(a2);
  e.cf = cf;
  speeds<R, DIR>(V, e);
  R dinv = R(1) / V[HD];
  R a2e = cf * cf;
  e.a2inv = R(1) / a2e;
  e.ahinv = R(0.5) / cf;
  R Na = R(0.5) * e.a2inv;
  e.lp = dinv * Na;
  e.rho = V[HD];
  e.rp = V[HD] * a2e;
}
// the same bits: g p / rho and 1 / rho share their divisor, halving is exact
template <int DIR, class A>
__device__ __forceinline__ void eigen64(const double *V, Eig<double> &e, A &ar, unsigned &st) {
  const Rcp d = ar.rcp(V[HD]);
  const double a2 = ar.by(V[HGC] * V[HP], d);
  if (a2 <= 0.) st |= ST_NEG_SOUND;
  const double cf = sqrt(a2);
  e.cf = cf;
  speeds<double, DIR>(V, e);
  const double a2e = cf * cf;
  e.a2inv = ar.rcp(a2e).r;
  e.ahinv = 0.5 * ar.rcp(cf).r;
  e.lp = d.r * (0.5 * e.a2inv);
  e.rho = V[HD];
  e.rp = V[HD] * a2e;
}

// left eigenvector k (column k of LeftEigvec) dotted with d[0..4]
template <class R, int DIR>
__device__ __forceinline__ R ldot(const Eig<R> &e, int k, const R *d) {
  constexpr int v1 = Slots<DIR>::v1, v2 = Slots<DIR>::v2, v3 = Slots<DIR>::v3;
  switch (k) {
    case 0: return (-e.ahinv) * d[v1] + e.lp * d[HP];
    case 1: return d[v2];
    case 2: return d[HD] + (-e.a2inv) * d[HP];
    case 3: return d[v3];
    default: return e.ahinv * d[v1] + e.lp * d[HP];
  }
}

// right-eigenvector projection sum_k reig(v,k) db(k) (PPM.F90:528-570)
template <class R, int DIR>
__device__ __forceinline__ void rproject(const Eig<R> &e, const R db[5], R t[5]) {
  constexpr int v1 = Slots<DIR>::v1, v2 = Slots<DIR>::v2, v3 = Slots<DIR>::v3;
  t[HD] = e.rho * db[0] + db[2] + e.rho * db[4];
  t[v1] = (-e.cf) * db[0] + e.cf * db[4];
  t[v2] = db[1];
  t[v3] = db[3];
  t[HP] = e.rp * db[0] + e.rp * db[4];
}

// ---------------------------------------------------------------------------
// hy_TVDslope.F90:76-246; slots 5,6 (gamc, game) are never used downstream
// under FLASH_EOS_GAMMA (PPM.F90:733-736) and are not computed.
// ---------------------------------------------------------------------------
template <class R, int DIR>
__device__ __forceinline__ void tvd_slope_d(const DevParams &P, const R *dL, const R *dR, R dLe, R dRe,
                                            const Eig<R> &e, R db[8]) {
  const int lim = P.limiter;
  const R beta = R(P.lim_beta);
  if (P.char_limiting) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      R a = ldot<R, DIR>(e, k, dL), b = ldot<R, DIR>(e, k, dR);
      int lk = lim == 3 ? (k == 2 ? 2 : 1) : lim;
      db[k] = limit2(lk, beta, a, b);
    }
    db[HEI] = limit2(lim == 3 ? 2 : lim, beta, dLe, dRe);
    R t[5];
    rproject<R, DIR>(e, db, t);
#pragma unroll
    for (int n = 0; n < 5; ++n) db[n] = t[n];
  } else {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      int lk = lim == 3 ? (k == HD ? 2 : 1) : lim;
      db[k] = limit2(lk, beta, dL[k], dR[k]);
    }
    db[HEI] = lim == 3 ? R(0) : limit2(lim, beta, dLe, dRe);   // hybrid: EINT is in neither case list, slope 0
  }
  db[HGC] = R(0); db[HGE] = R(0);
}

// FP64 with the division of the van Leer limiter through ar; the other
// limiters have none
template <int DIR, class A>
__device__ __forceinline__ void tvd_slope64(const DevParams &P, const double *VL, const double *V0, const double *VR,
                                            const Eig<double> &e, A &ar, double db[8]) {
  double dL[5], dR[5];
#pragma unroll
  for (int n = 0; n < 5; ++n) { dL[n] = V0[n] - VL[n]; dR[n] = VR[n] - V0[n]; }
  const double dLe = V0[HEI] - VL[HEI], dRe = VR[HEI] - V0[HEI];
  if (P.limiter == 4 && P.char_limiting) {
    auto vanleer = [&](double a, double b) {
      const bool on = !(a * b <= 0.);
      // a and b have one sign: take the quotient with a positive divisor
      const double num = 2. * a * b, s = a + b;
      const double q = ar.div(num, fabs(s), on);
      return on ? (s < 0. ? -q : q) : 0.;
    };
    double d[5], t[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) d[k] = vanleer(ldot<double, DIR>(e, k, dL), ldot<double, DIR>(e, k, dR));
    db[HEI] = vanleer(dLe, dRe);
    rproject<double, DIR>(e, d, t);
#pragma unroll
    for (int n = 0; n < 5; ++n) db[n] = t[n];
  } else {
    tvd_slope_d<double, DIR>(P, dL, dR, dLe, dRe, e, db);
  }
}

// ---------------------------------------------------------------------------
// hy_upwindTransverseFlux.F90:75-207 (transOrder = 1), sparse reig terms
// ---------------------------------------------------------------------------
template <class R, int DIR>
__device__ __forceinline__ void upwind_tflux_d(const DevParams &P, const R *dl, const R *dr, R dle, R dre,
                                               const Eig<R> &e, R sig[8]) {
  constexpr int v1 = Slots<DIR>::v1, v2 = Slots<DIR>::v2, v3 = Slots<DIR>::v3;
  R dn[5];
#pragma unroll
  for (int n = 0; n < 5; ++n) dn[n] = ldot<R, DIR>(e, n, e.lam[n] > R(0) ? dl : dr);
  const R *lam = e.lam;
  sig[HD] = (lam[0] * e.rho) * dn[0] + lam[2] * dn[2] + (lam[4] * e.rho) * dn[4];
  sig[v1] = (lam[0] * (-e.cf)) * dn[0] + (lam[4] * e.cf) * dn[4];
  sig[v2] = lam[1] * dn[1];
  sig[v3] = lam[3] * dn[3];
  sig[HP] = (lam[0] * e.rp) * dn[0] + (lam[4] * e.rp) * dn[4];
  sig[HGC] = R(0); sig[HGE] = R(0);
  sig[HEI] = P.use_aux_eint ? lam[2] * (lam[2] > R(0) ? dle : dre) : R(0);
}

// upwind differences dl = vc0 - vm1, dr = vp1 - vc0 of the three cells
template <class R, int DIR>
__device__ __forceinline__ void upwind_tflux(const DevParams &P, const R *vm1, const R *vc0, const R *vp1,
                                             const Eig<R> &e, R sig[8]) {
  R dl[5], dr[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) { dl[v] = vc0[v] - vm1[v]; dr[v] = vp1[v] - vc0[v]; }
  upwind_tflux_d<R, DIR>(P, dl, dr, vc0[HEI] - vm1[HEI], vp1[HEI] - vc0[HEI], e, sig);
}

// ---------------------------------------------------------------------------
// flattening of hy_getRiemannState.F90:356-454 for the cell at stencil
// position 3 of p[0..6] (pressures at c-3..c+3) and u[0..6] (normal vel.)
// ---------------------------------------------------------------------------
template <class A>
__device__ __forceinline__ double flat_tilde(A &ar, double pm2, double pm1, double pp1, double pp2, double um1,
                                             double up1) {
  const double dp1 = pp1 - pm1, dp2 = pp2 - pm2, dv1 = up1 - um1;
  const bool on = fabs(dp2) > 1.e-15;
  const double q = ar.div(dp1, fabs(dp2), on);
  const double Sp = on ? (dp2 < 0. ? -q : q) - 0.75 : 0.;
  double ft = rmax(0.0, rmin(1.0, 10.0 * Sp));
  if ((ar.div(fabs(dp1), rmin(pm1, pp1)) < 1. / 3.) || dv1 > 0.) ft = 0.;
  return ft;
}

}  // namespace fhy
