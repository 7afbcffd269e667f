// hy_dir64.cuh -- the FP64 direction kernel (k_dir).
//
// One direction of the unsplit update, in the expression order of the
// Fortran it restates, so that the build without FMA contraction stays
// bit-identical to an IEEE evaluation of the reference.  What the reference
// evaluates three times per cell (its own and its neighbours' eigensystems,
// limited slopes and flattening switches,
// hy_DataReconstructNormalDir_PPM.F90:438-441) is evaluated once per cell
// and shared through shared memory: the same expressions on the same
// operands, hence the same bits.  Divisions are branch-free and share
// reciprocals (Arith, hy_core.cuh), with the bits of IEEE division; a cell
// whose operands leave the range where that is proven is evaluated again
// with plain divisions.
#pragma once
#include <type_traits>
#include "hy_kernels.cuh"
#include "hy_launch.h"
#include "hy_tma.cuh"

namespace fhy {

// ---------------------------------------------------------------------------
// Geometry of a CTA: the lines along DIR of part `part` of a block's
// cross-section (the slower transverse axis split into Q parts), over one
// block or over a run of K blocks that follow one another along DIR.
// Positions x of a line: staged cells [-4, N+3], slope cells [-2, N+1], line
// cells [-1, N], faces [0, N] (face x between cells x - 1 and x).
// ---------------------------------------------------------------------------
template <int NDIM, int NX, int NY, int NZ, int DIR, int Q, int K>
struct Dir64 {
  static constexpr int N0 = DIR == 1 ? NX : (DIR == 2 ? NY : NZ);     // block extent along DIR
  static constexpr int N = K * N0;                                    // line interior
  static constexpr int T1 = DIR == 1 ? NY : NX;                       // faster transverse axis
  static constexpr int T2 = NDIM > 2 ? (DIR == 3 ? NY : NZ) : 1;      // slower one, split
  static_assert(T2 % Q == 0, "the slower transverse axis is split evenly");
  static constexpr int T2Q = T2 / Q;
  static_assert(K == 1 || T2Q == 1, "a run's tiles hold one layer of lines");
  static constexpr int C = T1 * T2Q;                                  // lines
  static constexpr int L4 = N + 8, LS = N + 4, LC = N + 2;
  static constexpr int SA = L4 * C, SB = LS * C, SC = LC * C;
  static constexpr int step = DIR == 1 ? 1 : C;                       // +1 along the line (slope and line cells)
  __device__ static __forceinline__ int at(int x, int l, int L, int o) {
    return DIR == 1 ? l * L + (x + o) : (x + o) * C + l;
  }
  __device__ static __forceinline__ void dec(int s, int L, int o, int &x, int &l) {
    if (DIR == 1) { l = s / L; x = s % L - o; }
    else { l = s % C; x = s / C - o; }
  }
  // staged cells: the line layout, or, for a run along x, the tiles as they
  // are copied (slab below, the blocks, slab above, each x fastest; along y
  // and z the tiles follow one another in the line layout)
  __device__ static __forceinline__ int sidx(int x, int l) {
    if (K == 1 || DIR != 1) return at(x, l, L4, 4);
    if (x < 0) return l * 4 + (x + 4);
    if (x >= N) return (4 + N) * C + l * 4 + (x - N);
    return 4 * C + (x / N0) * (N0 * C) + l * N0 + x % N0;
  }
  // block of the run at position x (the end blocks for the guard positions);
  // x becomes relative to it
  __device__ static __forceinline__ int blk_of(int &x) {
    if (K == 1) return 0;
    const int m = x < 0 ? 0 : (x >= N ? K - 1 : x / N0);
    x -= m * N0;
    return m;
  }
  __device__ static __forceinline__ void cell(int x, int l, int part, int &i, int &j, int &k) {
    const int t1 = l % T1, t2 = l / T1 + part * T2Q;
    i = DIR == 1 ? x : t1;
    j = DIR == 1 ? t1 : (DIR == 2 ? x : t2);
    k = DIR == 3 ? x : (NDIM > 2 ? t2 : 0);
  }
  // shared memory (doubles): the staged primitives rho, u, v, w, e, later
  // the 8 face fluxes; the 6 limited slopes and the flattening switch; the
  // 6 + 6 face-state slots and the cell's game; runs: the staging barrier
  // and the slack that aligns the tiles to 128 bytes
  static constexpr int NQ = 5 * SA > NFLX * SC ? 5 * SA : NFLX * SC;
  static constexpr int ND = 7 * SB, NW = 13 * SC;
  static constexpr size_t smem_bytes() { return (size_t)(NQ + ND + NW) * sizeof(double) + (K > 1 ? 16 + 128 : 0); }
};

// Parts of a block's cross-section per direction launch: one-block CTAs of
// 3D grids are halved (75 KB of shared memory), so that two fit an SM.
// Quarters at 192 threads and four CTAs per SM: the same time (a 3D
// hierarchy's step 4.34 against 4.37 ms).
template <int NDIM> constexpr int dir64_parts() { return NDIM == 3 ? 2 : 1; }

// Launch bounds (threads, CTAs per SM).  The kernel is bound by dependent
// FP64 latency, so warps in flight decide: runs hold 27 warps at 72
// registers with spills to L1 (128^3 step 1.33 ms) against 18 at 96 (1.48)
// and 16 at 128 (1.9); one-block 3D CTAs 20 warps at 96.  2D 8^2 blocks: 24
// warps at 80 registers, best from 256^2 to 2048^2 zones (step 0.042 / 1.65 ms;
// 20 warps at 102 registers 0.054 / 1.85, 32 at 64 0.044 / 1.68).  2D 16^2: 20
// warps at 96 (0.040 / 1.55; 10 warps 0.056 / 2.42; 30 at 64 registers 0.044 /
// 1.44: better from 1024^2 on, worse below).
template <int NDIM, int NX, int K> struct Dir64Bounds {
  static constexpr int threads = K > 1 ? 288 : (NDIM == 3 || NX == 16 ? 320 : 128);
  static constexpr int ctas = K > 1 ? 3 : (NDIM == 3 || NX == 16 ? 2 : 6);
};

// ---------------------------------------------------------------------------
// hy_DataReconstructNormalDir_PPM.F90:485-842 for one cell from the limited
// slopes of the cell and its neighbours (HLL-type characteristic tracing).
// Vm, Vc, Vp: slots rho, u, v, w, p and (HEI) e; db(n, s): limited slope of
// variable n (5 = e) at the cell (s = 0) and its neighbours (s = -1, 1);
// rho2(s), and the cell's game for the steepening; flat: the flattening
// coefficient, 0 without flattening.  e comes first and leaves through
// eint(Wm, Wp), so that its values hold no registers during the tracing;
// the others in Wm, Wp (slots 0..4).
// ---------------------------------------------------------------------------
template <int DIR, class A, class Slope, class Rho2, class EintOut>
__device__ __forceinline__ void ppm_states(const DevParams &P, A &ar, const double *Vm, const double *Vc, const double *Vp,
                                           Slope db, Rho2 rho2, double game, double flat, double dtn, double delta,
                                           const Eig<double> &e0, double Wp[5], double Wm[5], EintOut eint) {
  constexpr int v1 = Slots<DIR>::v1, v2 = Slots<DIR>::v2, v3 = Slots<DIR>::v3;
  const double hdtn = 0.5 * dtn;
  constexpr int NS = 6;
  double delW[5], W6[5];
#pragma unroll
  for (int r = 0; r < NS; ++r) {
    const int q = r == 0 ? 5 : r - 1, n = q < 5 ? q : HEI;
    const double dN = db(q, -1), d0 = db(q, 0), dP = db(q, 1);
    double vl = 0.5 * (Vc[n] + Vm[n]) - ar.template byc<6>(d0 - dN);
    double vr = 0.5 * (Vc[n] + Vp[n]) - ar.template byc<6>(dP - d0);
    if (n == HD && P.use_steepening) {                            // PPM.F90:639-670
      const double eta1 = 20.E0, eta2 = 0.05E0, epsln = 0.01E0, K0 = 0.1E0;
      const double temp1 = Vp[HD] - Vm[HD];
      if (fabs(temp1) > P.tiny) {
        const double del2rhoR = (rho2(2) - 2. * Vp[HD] + Vc[HD]) / (6. * delta * delta);
        const double del2rhoL = (Vc[HD] - 2. * Vm[HD] + rho2(-2)) / (6. * delta * delta);
        double eta_steep = (del2rhoL - del2rhoR) * (delta * delta) / temp1;
        if (del2rhoR * del2rhoL >= 0.) eta_steep = 0.;
        if (epsln * rmin(Vp[HD], Vm[HD]) - fabs(Vp[HD] - Vm[HD]) >= 0.) eta_steep = 0.;
        eta_steep = rmax(0., rmin(1., eta1 * (eta_steep - eta2)));
        const double temp2 = fabs(Vp[HP] - Vm[HP]) / rmin(Vp[HP], Vm[HP]);
        const double temp3 = fabs(Vp[HD] - Vm[HD]) / rmin(Vp[HD], Vm[HD]);
        if (game * K0 * temp3 - temp2 < 0.0) eta_steep = 0.;
        vl = vl * (1. - eta_steep) + (Vm[HD] + 0.5 * dN) * eta_steep;
        vr = vr * (1. - eta_steep) + (Vp[HD] - 0.5 * dP) * eta_steep;
      }
    }
    if (flat != 0.) {                                             // PPM.F90:676-679 (the identity where flat = 0)
      vl = flat * Vc[n] + (1.0 - flat) * vl;
      vr = flat * Vc[n] + (1.0 - flat) * vr;
    }
    // PPM.F90:686-706: the second test repeats the first one's operands
    // unless that one moved the left value
    if ((vr - Vc[n]) * (Vc[n] - vl) <= 0.) { vl = Vc[n]; vr = Vc[n]; }
    double d = vr - vl, m = Vc[n] - 0.5 * (vl + vr);
    if (6. * d * m > d * d) {
      vl = 3. * Vc[n] - 2. * vr;
      d = vr - vl;
      m = Vc[n] - 0.5 * (vl + vr);
    }
    if (6. * d * m < -(d * d)) {
      vr = 3. * Vc[n] - 2. * vl;
      d = vr - vl;
      m = Vc[n] - 0.5 * (vr + vl);
    }
    if (n == HEI) {                           // entropy-wave traced initial guess (PPM.F90:715-727)
      const double w6 = 6. * m, lmax = rmax(e0.lam[2], 0.), lmin = -rmin(e0.lam[2], 0.);
      eint(vl + lmin * hdtn * (d + (1.0 - ar.template byc<3>(lmin * hdtn * 4.)) * w6),
           vr - lmax * hdtn * (d - (1.0 - ar.template byc<3>(lmax * hdtn * 4.)) * w6));
    } else {
      delW[q] = d;
      W6[q] = 6. * m;
    }
  }
  // characteristic tracing, all waves into both sides (PPM.F90:753-800)
  double mW6[5];
#pragma unroll
  for (int n = 0; n < 5; ++n) mW6[n] = -W6[n];
  double sigL[5], sigR[5];
  const double f43 = 4. / 3.;
#pragma unroll
  for (int n = 0; n < 5; ++n) {
    const double cA = ldot<double, DIR>(e0, n, delW);
    const double cB = ldot<double, DIR>(e0, n, mW6);
    const double lam = e0.lam[n];
    const double x = dtn * lam;
    const double AL = .5 * (-1. - dtn * lam);
    const double BL = .25 * (1. + 2. * dtn * lam + f43 * (x * x));
    const double AR = .5 * (1. - dtn * lam);
    const double BR = .25 * (1. - 2. * dtn * lam + f43 * (x * x));
    // non-zero entries of column n of RightEigvec
    if (n == 0 || n == 4) {
      const double rv = n == 0 ? -e0.cf : e0.cf;
      const double tL_d = AL * e0.rho * cA + BL * e0.rho * cB, tR_d = AR * e0.rho * cA + BR * e0.rho * cB;
      const double tL_v = AL * rv * cA + BL * rv * cB, tR_v = AR * rv * cA + BR * rv * cB;
      const double tL_p = AL * e0.rp * cA + BL * e0.rp * cB, tR_p = AR * e0.rp * cA + BR * e0.rp * cB;
      if (n == 0) {
        sigL[HD] = tL_d; sigR[HD] = tR_d; sigL[v1] = tL_v; sigR[v1] = tR_v; sigL[HP] = tL_p; sigR[HP] = tR_p;
      } else {
        sigL[HD] = sigL[HD] + tL_d; sigR[HD] = sigR[HD] + tR_d;
        sigL[v1] = sigL[v1] + tL_v; sigR[v1] = sigR[v1] + tR_v;
        sigL[HP] = sigL[HP] + tL_p; sigR[HP] = sigR[HP] + tR_p;
      }
    } else {
      const double tL = AL * cA + BL * cB, tR = AR * cA + BR * cB;       // reig entry 1
      if (n == 1) { sigL[v2] = tL; sigR[v2] = tR; }
      else if (n == 2) { sigL[HD] = sigL[HD] + tL; sigR[HD] = sigR[HD] + tR; }
      else { sigL[v3] = tL; sigR[v3] = tR; }
    }
  }
#pragma unroll
  for (int n = 0; n < 5; ++n) {                                   // PPM.F90:841-842
    const double c = Vc[n] + ar.template byc<12>(W6[n]);
    Wm[n] = c + sigL[n];
    Wp[n] = c + sigR[n];
  }
}

// ---------------------------------------------------------------------------
// hy_prim2con.F90:37-54, hy_prim2flx.F90:49-123, hy_HLLC.F90:94-311, and the
// auxiliary volume flux F_dens / rho of the upwind side
// (hy_getFaceFlux.F90:433-442).  Only the side whose flux (and star state)
// the solver returns is evaluated; the star state's five divisions share
// their divisor.  With branch-free arithmetic the solver's early exits
// (vanishing densities or pressures, a negative squared sound speed) raise
// `bad` instead.
// ---------------------------------------------------------------------------
template <int DIR, class A>
__device__ __forceinline__ void hllc64(const DevParams &P, A &ar, const double *Vm, const double *Vp, double Fs[6],
                                       double &fv, unsigned &st) {
  constexpr int v1 = Slots<DIR>::v1;
  const double tiny = P.tiny;
  const double velNL = Vm[v1], velNR = Vp[v1];
  const Rcp rL = ar.rcp(Vm[HD]), rR = ar.rcp(Vp[HD]);
  const double aL2 = ar.by(Vm[HGC] * Vm[HP], rL);
  const double aR2 = ar.by(Vp[HGC] * Vp[HP], rR);
  const bool vanish = (Vm[HD] < tiny && Vm[HD] > 0.) || (Vp[HD] < tiny && Vp[HD] > 0.) ||
                      (Vm[HP] < tiny && Vm[HP] > 0.) || (Vp[HP] < tiny && Vp[HP] > 0.);
  const bool neg = aL2 < 0. || aR2 < 0.;
  if constexpr (std::is_same<A, Arith<true>>::value) {
    ar.bad |= vanish || neg;
  } else if (vanish || neg) {
    if (!vanish) st |= ST_NEG_SOUND;
#pragma unroll
    for (int n = 0; n < 6; ++n) Fs[n] = 0.;
    fv = 0. / Vp[HD];
    return;
  }
  const double cfL = sqrt(aL2), cfR = sqrt(aR2);
  const double SL = rmin(velNL - cfL, velNR - cfR);
  const double SR = rmax(velNL + cfL, velNR + cfR);
  const double pL = Vm[HP], pR = Vp[HP];
  // the wave speeds bound the velocities (SL <= uL, uR <= SR): a positive divisor
  const double qStar = ar.div(Vp[HD] * velNR * (SR - velNR) - Vm[HD] * velNL * (SL - velNL) + pL - pR - 0. * 0. + 0. * 0.,
                              Vp[HD] * (SR - velNR) - Vm[HD] * (SL - velNL));
  const double pStar = Vm[HD] * (SL - velNL) * (qStar - velNL) + pL;
  const bool useL = SL >= 0. || ((SL < 0.) && (qStar >= 0.));
  const bool star = useL ? !(SL >= 0.) : ((qStar < 0.) && (SR >= 0.));
  double V[8];
#pragma unroll
  for (int n = 0; n < 5; ++n) V[n] = useL ? Vm[n] : Vp[n];
  const double ge = useL ? Vm[HGE] : Vp[HGE], S = useL ? SL : SR;
  const double velN = V[v1], p = V[HP];
  const double u2 = V[HVX] * V[HVX] + V[HVY] * V[HVY] + V[HVZ] * V[HVZ];
  const double E = 0.5 * V[HD] * u2 + ar.div(p, ge - 1.);
  double F[5];
  F[0] = V[HD] * velN;
  F[1] = F[0] * V[HVX];
  F[2] = F[0] * V[HVY];
  F[3] = F[0] * V[HVZ];
  F[DIR] = F[DIR] + 1.0 * p;                     // hy_fPresInMomFlux = 1
  F[4] = (E + p) * velN;
  Fs[5] = p;
  const double U[5] = {V[HD], V[HD] * V[HVX], V[HD] * V[HVY], V[HD] * V[HVZ], E + 0.5 * 0.};
  // numerator and divisor negated on the left: a positive divisor
  const double numer = useL ? velN - S : S - velN;
  const Rcp denom = ar.rcp(useL ? qStar - S : S - qStar, star);
  const double work = pStar * qStar - p * velN;
  const double dStar = ar.by(U[0] * numer, denom, star);
  double UC[5];
  UC[0] = dStar;
  UC[4] = ar.by(U[4] * numer, denom, star) + ar.by(useL ? -work : work, denom, star);
#pragma unroll
  for (int m = 1; m <= 3; ++m) UC[m] = (m == DIR) ? dStar * qStar : ar.by(U[m] * numer, denom, star);
#pragma unroll
  for (int n = 0; n < 5; ++n) Fs[n] = star ? F[n] + S * (UC[n] - U[n]) : F[n];
  const bool up = Fs[0] > 0.;
  fv = ar.by(Fs[0], up ? rL : rR);
}

// ---------------------------------------------------------------------------
// k_dir: one direction of the unsplit update for one part of a block per CTA.
// Bound by dependent FP64 latency.  What it measured (B200, KH 128^3 step,
// k_sig included, HLLC): 2.99 ms with one kernel body that evaluated three
// slopes per cell (150 registers, 10 warps per SM); 1.97 with the phases
// below (96 registers); 1.92 with the bulk L2 prefetch; 1.85 on runs of four
// blocks; 1.50 with branch-free divisions; 1.33 with three run CTAs per SM
// and the traced e parked in shared memory.  2D Sod 256^2: 0.090 -> 0.044 ms.
//   stage    the line stencils (cp.async through the neighbour table; runs:
//            TMA tile copies)
//   slopes   eigensystem, limited slopes and flattening switch of the cells
//            [-2, N+1] of every line
//   states   face states W-/W+ of the cells [-1, N]: PPM
//            (hy_dataReconstOneStep.F90:485-716), transverse corrections
//            (:918-951), last negativity check (:1120-1154), 3D full-CTU
//            cross terms and positivity fallback
//            (hy_getRiemannState.F90:956-1313)
//   faces    HLLC (RS = 0) or the exact solver (RS = 1) at the N+1 faces of
//            every line plus the auxiliary internal-energy and volume fluxes
//            (hy_getFaceFlux.F90:283-442)
//   update   accumulation of the conservative update in direction order
//            x, y, z (updateConservedVariable, hy_unsplitUpdate.F90:1187-
//            1242); the last direction finishes the cell: internal-energy
//            update with the n+1/2 pressure (:657-672, hy_getFaceFlux.F90:
//            551-557 and y/z analogues), hy_energyFix (:188-253), the EOS
//            and the CFL reduction (Hydro_computeDt.F90:186-290).
// ---------------------------------------------------------------------------
// slots stored for the face states: dens, velx, vely, velz, pres, eint
__device__ __forceinline__ int wslot(int q) { return q < 5 ? q : HEI; }

template <int NDIM, int NX, int NY, int NZ, int DIR, bool FIRST, bool LAST, int VAR, int RS, int Q, int K>
__global__ void __launch_bounds__(Dir64Bounds<NDIM, NX, K>::threads, Dir64Bounds<NDIM, NX, K>::ctas)
k_dir(const DevParams P, const double *__restrict__ SIG, double *__restrict__ ACC, double *__restrict__ AUX,
      size_t ncells, CflPart *part, CflCand *cflq, const __grid_constant__ TmaLine tm) {
  using G = Dir64<NDIM, NX, NY, NZ, DIR, Q, K>;
  using B = Box<NDIM, NX, NY, NZ>;
  using DG = DirGeom<NDIM, NX, NY, NZ, double, DIR>;
  constexpr int NCB = NX * NY * NZ;
  constexpr int v1 = Slots<DIR>::v1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char *smem = smem_raw;
  if constexpr (K > 1) smem += (128u - (smem_u32(smem_raw) & 127u)) & 127u;
  double *sQ = reinterpret_cast<double *>(smem);       // [5][SA] rho, u, v, w, e
  double *sF = sQ;                                      // [8][SC], over the stencil once the states are done
  double *sDb = sQ + G::NQ;                             // [6][SB] limited slopes, [SB] flattening switches
  double *sWp = sDb + G::ND;                            // [6][SC]
  double *sWm = sWp + 6 * G::SC;                        // [6][SC]
  double *sGe = sWm + 6 * G::SC;                        // [SC] game
  if (K > 1 && threadIdx.x < 10) prefetch_tensormap(threadIdx.x < 5 ? &tm.intr[threadIdx.x] : &tm.slab[threadIdx.x - 5]);
  const int launch_slot = Q == 1 ? (int)blockIdx.x : (int)(blockIdx.x / Q);
  const int qtr = Q == 1 ? 0 : (int)(blockIdx.x % Q);
  // the CTA's block, or the K blocks of its run and the neighbours below
  // and above it (-1: none)
  int blk[K], nbs[2] = {-1, -1};
  if constexpr (K == 1) {
    blk[0] = P.blk_list ? P.blk_list[launch_slot] : launch_slot;
  } else {
    const int *run = tm.runs + (size_t)launch_slot * (K + 2);
#pragma unroll
    for (int m = 0; m < K; ++m) blk[m] = run[m];
    nbs[0] = run[K];
    nbs[1] = run[K + 1];
  }
  const int b = blk[0];
  const int slot = P.slot ? P.slot[b] : launch_slot;      // one-block CTAs: where the block's sig lies
  const int3 bc = blk_coords(P, b);
  unsigned st = 0;
  const double dt = P.dt_dev ? *P.dt_dev : P.dt;
  double del[3];
  blk_deltas(P, b, del);
  const double delta = del[DIR - 1];
  auto fidx = [](int along, int t1, int t2) { return G::at(along, t1 + G::T1 * t2, G::LC, 1); };   // t2 within the part
  const double *sigb = SIG + (size_t)(K == 1 ? slot : b) * NDIM * 6 * B::n;
  // what is read from global memory after the staging (the other
  // directions' sig, the accumulators and, in the last direction, the aux
  // rows) is fetched into L2 meanwhile, one bulk request per contiguous range
  static_assert((6 * B::n * 8) % 16 == 0 && (NCB * 8) % 16 == 0, "bulk prefetch sizes are multiples of 16 bytes");
  // (the first CTAs of a run take a block each)
  if (threadIdx.x < 32 && qtr < K) {
    const int ln = threadIdx.x;
    const int pb = K == 1 ? b : tm.runs[(size_t)launch_slot * (K + 2) + qtr];
    const double *ps = SIG + (size_t)(K == 1 ? slot : pb) * NDIM * 6 * B::n;
    if (ln < NDIM && ln != DIR - 1 && P.fmode != 3) bulk_prefetch_l2(ps + (size_t)ln * 6 * B::n, 6u * B::n * 8u);
    if (!FIRST && ln >= 4 && ln < 9) bulk_prefetch_l2(ACC + (ln - 4) * ncells + (size_t)pb * NCB, NCB * 8u);
    if (LAST && ln >= 12 && ln < 12 + 3 * (NDIM - 1))
      bulk_prefetch_l2(AUX + (ln - 12) * ncells + (size_t)pb * NCB, NCB * 8u);
  }

  // where the species pass finds line cell y of block m on line l
  auto sp_line = [&](int m, int y, int l) {
    int i, j, k;
    G::cell(y, l, qtr, i, j, k);
    return sp_line_base<NDIM, NX, NY, NZ, DIR>(K == 1 ? slot : pick(blk, m)) + DG::idx(i, j, k);
  };
  if (K > 1 || P.fmode != 3) {
  // ---- stage
  if constexpr (K == 1) {
    __shared__ int sNb[NDIM > 2 ? 27 : 9];
    if (P.lh == nullptr) {
      neighbour_table<NDIM, NX, NY, NZ>(P, bc, sNb);
      __syncthreads();
    }
    stage_prims<NDIM, NX, NY, NZ>(P, b, bc, slot, sNb, sQ, G::SA, [=](int c, int &i, int &j, int &k) {
      int x, l;
      G::dec(c, G::L4, 4, x, l);
      G::cell(x, l, qtr, i, j, k);
      return true;
    });
  } else {
    // a run: the blocks' layers and the neighbours' slabs by TMA tile
    // copies, one per lane of warp 0; slabs beyond a non-periodic boundary
    // through load_prim; then the copied guard cells' EOS in place
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(sGe + G::SC);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    constexpr int NOPS = 5 * (K + 2);
    static_assert(NOPS <= 32, "one copy per lane of warp 0");
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0)
        mbar_expect_tx(bar, 5u * 8u * (unsigned)G::C * (unsigned)(G::N + (nbs[0] >= 0 ? 4 : 0) + (nbs[1] >= 0 ? 4 : 0)));
      __syncwarp();
      if (threadIdx.x < NOPS) {
        const int v = threadIdx.x / (K + 2), r = threadIdx.x % (K + 2);
        double *dst = sQ + v * G::SA;
        if (r < K) {
          const int bl = tm.runs[(size_t)launch_slot * (K + 2) + r];
          tma_load_3d(dst + (4 + r * G::N0) * G::C, &tm.intr[v], 0, DIR == 3 ? qtr : 0, bl * NZ + (DIR == 3 ? 0 : qtr), bar);
        } else if (r == K) {
          if (nbs[0] >= 0)
            tma_load_3d(dst, &tm.slab[v], DIR == 1 ? NX - 4 : 0, DIR == 2 ? NY - 4 : (DIR == 3 ? qtr : 0),
                        nbs[0] * NZ + (DIR == 3 ? NZ - 4 : qtr), bar);
        } else if (nbs[1] >= 0) {
          tma_load_3d(dst + (4 + G::N) * G::C, &tm.slab[v], 0, DIR == 3 ? qtr : 0,
                      nbs[1] * NZ + (DIR == 3 ? 0 : qtr), bar);
        }
      }
    }
    for (int g = threadIdx.x; g < 8 * G::C; g += blockDim.x) {
      const int side = g >= 4 * G::C, r = g - side * 4 * G::C;
      if (nbs[side] >= 0) continue;
      const int x = side ? G::N + r / G::C : r / G::C - 4, l = r % G::C, q = G::sidx(x, l);
      int xl = x, i, j, k;
      const int bm = blk[side ? K - 1 : 0];
      G::blk_of(xl);
      G::cell(xl, l, qtr, i, j, k);
      double V[8];
      load_prim<NDIM, NX, NY, NZ, false>(P, bm, blk_coords(P, bm), i, j, k, V);
      sQ[q] = V[HD]; sQ[G::SA + q] = V[HVX]; sQ[2 * G::SA + q] = V[HVY]; sQ[3 * G::SA + q] = V[HVZ];
      sQ[4 * G::SA + q] = V[HEI];
    }
    if (!tma_wait(bar, P.status)) return;
    for (int g = threadIdx.x; g < 8 * G::C; g += blockDim.x) {
      const int side = g >= 4 * G::C, r = g - side * 4 * G::C;
      if (nbs[side] < 0) continue;
      const int x = side ? G::N + r / G::C : r / G::C - 4, q = G::sidx(x, r % G::C);
      const double vx = sQ[G::SA + q], vy = sQ[2 * G::SA + q], vz = sQ[3 * G::SA + q];
      const double ekin = 0.5 * (vx * vx + vy * vy + vz * vz);
      const double ener = sQ[4 * G::SA + q] + ekin;
      if (ener - ekin > rmax(P.smalle, P.eswitch * ekin)) sQ[4 * G::SA + q] = ener - ekin;
    }
  }
  __syncthreads();
  const double gam1inv = P.gam1inv;
  // slots rho, u, v, w, p (and e in HEI) of staged cell s
  auto prim = [&](int s, double V[8]) {
    const double rho = sQ[s], e = sQ[4 * G::SA + s];
    V[HD] = rho; V[HVX] = sQ[G::SA + s]; V[HVY] = sQ[2 * G::SA + s]; V[HVZ] = sQ[3 * G::SA + s];
    V[HP] = rho * e * gam1inv; V[HGC] = P.gamma; V[HGE] = 0.; V[HEI] = e;
  };
  auto pres = [&](int s) { return sQ[s] * sQ[4 * G::SA + s] * gam1inv; };

  // ---- slopes
  auto slopes = [&](auto &ar, int q) {
    int x, l;
    G::dec(q, G::LS, 2, x, l);
    double Vm[8], Vc[8], Vp[8], db[8];
    prim(G::sidx(x - 1, l), Vm);
    prim(G::sidx(x, l), Vc);
    prim(G::sidx(x + 1, l), Vp);
    Eig<double> e;
    eigen64<DIR>(Vc, e, ar, st);
    tvd_slope64<DIR>(P, Vm, Vc, Vp, e, ar, db);
    double ft = 0.;
    if (P.use_flattening)
      ft = flat_tilde(ar, pres(G::sidx(x - 2, l)), Vm[HP], Vp[HP], pres(G::sidx(x + 2, l)), Vm[v1], Vp[v1]);
#pragma unroll
    for (int n = 0; n < 5; ++n) sDb[n * G::SB + q] = db[n];
    sDb[5 * G::SB + q] = db[HEI];
    sDb[6 * G::SB + q] = ft;
  };
  // (each phase runs with branch-free divisions; where any cell of the CTA
  // needs plain ones, the CTA takes the phase again with those, and the
  // status bits of the first attempt go)
  Arith<true> ar;
  Arith<false> plain;
  unsigned st0 = st;
  for (int q = threadIdx.x; q < G::SB; q += blockDim.x) slopes(ar, q);
  if (__syncthreads_or(ar.bad)) {
    st = st0;
    for (int q = threadIdx.x; q < G::SB; q += blockDim.x) slopes(plain, q);
    __syncthreads();
  }

  // ---- states
  const double dtn = dt / delta;
  const double hdtx = 0.5 * dt / del[0], hdty = 0.5 * dt / del[1], hdtz = 0.5 * dt / del[2];
  auto states = [&](auto &ar, int t) {
    int x, l, i, j, k;
    G::dec(t, G::LC, 1, x, l);
    int xl = x;
    const int mb = G::blk_of(xl);                // block of the run: its sig box covers xl in [-1, N0]
    G::cell(xl, l, qtr, i, j, k);
    const double *sigc = K == 1 ? sigb : SIG + (size_t)pick(blk, mb) * NDIM * 6 * B::n;
    const int q = G::at(x, l, G::LS, 2);
    double Vc[8];
    Eig<double> e0;
    auto cell_state = [&] {                                        // first order: the cell's own values
#pragma unroll
      for (int qq = 0; qq < 6; ++qq) sWm[qq * G::SC + t] = sWp[qq * G::SC + t] = Vc[wslot(qq)];
    };
    const int bi = B::idx(i, j, k);
    {
      double Vm[8], Vp[8], Wm[5], Wp[5];
      prim(G::sidx(x - 1, l), Vm);
      prim(G::sidx(x, l), Vc);
      prim(G::sidx(x + 1, l), Vp);
      Vc[HGE] = ar.div(Vc[HP], Vc[HEI] * Vc[HD]) + 1;         // Eos_putData.F90:105-106
      sGe[t] = Vc[HGE];
      double flat = 0.;
      if (P.use_flattening) {
        const double t0 = sDb[6 * G::SB + q], dp1 = Vp[HP] - Vm[HP];
        if (dp1 < 0.0) flat = rmax(t0, sDb[6 * G::SB + q + G::step]);
        else if (dp1 == 0.) flat = t0;
        else flat = rmax(t0, sDb[6 * G::SB + q - G::step]);
      }
      if (P.sp_flat)
        seam_blocks<K, G::N0, false>(x, [&](int m, int y) { P.sp_flat[sp_line(m, y, l)] = flat; });
      eigen64<DIR>(Vc, e0, ar, st);
      ppm_states<DIR>(P, ar, Vm, Vc, Vp, [&](int n, int o) { return sDb[n * G::SB + q + o * G::step]; },
                      [&](int o) { return sQ[G::sidx(x + o, l)]; }, Vc[HGE], flat, dtn, delta, e0, Wp, Wm,
                      [&](double wm, double wp) { sWm[5 * G::SC + t] = wm; sWp[5 * G::SC + t] = wp; });
      // transverse corrections with the sig of the other directions (same cell)
      constexpr int d1 = DIR == 1 ? 1 : 0, d2 = DIR == 3 ? 1 : 2;
      const double hdt1 = d1 == 0 ? hdtx : hdty, hdt2 = d2 == 1 ? hdty : hdtz;
      bool bad = false;
#pragma unroll
      for (int qq = 0; qq < 6; ++qq) {
        double wm = qq < 5 ? Wm[qq] : sWm[5 * G::SC + t], wp = qq < 5 ? Wp[qq] : sWp[5 * G::SC + t];
        const double c1 = hdt1 * sigc[(d1 * 6 + qq) * B::n + bi];
        wm = wm - c1;
        wp = wp - c1;
        if (NDIM == 3) {
          const double c2 = hdt2 * sigc[(d2 * 6 + qq) * B::n + bi];
          wm = wm - c2;
          wp = wp - c2;
        }
        if (qq == HD || qq == HP) bad |= wm < 0. || wp < 0.;
        sWm[qq * G::SC + t] = wm;
        sWp[qq * G::SC + t] = wp;
      }
      if (bad) cell_state();
    }
    if (NDIM == 3 && P.use_ctu) {
      // axis / sig direction pairs of hy_getRiemannState.F90:999-1022,
      // 1101-1124, 1204-1227; the eigensystem differs from the line's only
      // in its wave speeds
      constexpr int A1 = DIR == 1 ? 2 : (DIR == 2 ? 3 : 1), S1 = DIR == 1 ? 3 : (DIR == 2 ? 1 : 2);
      constexpr int A2 = DIR == 1 ? 3 : (DIR == 2 ? 1 : 2), S2 = DIR == 1 ? 2 : (DIR == 2 ? 3 : 1);
      const double fac = dt * dt / (6. * (DIR == 1 ? del[1] : (DIR == 2 ? del[2] : del[0])) *
                                    (DIR == 1 ? del[2] : (DIR == 2 ? del[0] : del[1])));
      double T1[8], T2[8];
      {
        double sm[8], s0[8], sp[8];
        const double *base = sigc + (size_t)(S1 - 1) * 6 * B::n + bi;
        constexpr int o = A1 == 1 ? 1 : (A1 == 2 ? B::bx : B::bx * B::by);
        load_sig(base - o, B::n, sm);
        load_sig(base, B::n, s0);
        load_sig(base + o, B::n, sp);
        Eig<double> e = e0;
        speeds<double, A1>(Vc, e);
        upwind_tflux<double, A1>(P, sm, s0, sp, e, T1);
      }
      {
        double sm[8], s0[8], sp[8];
        const double *base = sigc + (size_t)(S2 - 1) * 6 * B::n + bi;
        constexpr int o = A2 == 1 ? 1 : (A2 == 2 ? B::bx : B::bx * B::by);
        load_sig(base - o, B::n, sm);
        load_sig(base, B::n, s0);
        load_sig(base + o, B::n, sp);
        Eig<double> e = e0;
        speeds<double, A2>(Vc, e);
        upwind_tflux<double, A2>(P, sm, s0, sp, e, T2);
      }
      bool fb = false;
#pragma unroll
      for (int qq = 0; qq < 6; ++qq) {
        const double c = (T1[wslot(qq)] + T2[wslot(qq)]) * fac;
        const double wp = sWp[qq * G::SC + t] + c, wm = sWm[qq * G::SC + t] + c;
        if (qq == HD || qq == HP) fb |= wp <= 0. || wm <= 0.;
        sWp[qq * G::SC + t] = wp;
        sWm[qq * G::SC + t] = wm;
      }
      if (fb) cell_state();
      if (P.sp_fb) seam_blocks<K, G::N0, false>(x, [&](int m, int y) { P.sp_fb[sp_line(m, y, l)] = fb; });
    }
  };
  ar.bad = false;
  st0 = st;
  for (int t = threadIdx.x; t < G::SC; t += blockDim.x) states(ar, t);
  if (__syncthreads_or(ar.bad)) {
    st = st0;
    for (int t = threadIdx.x; t < G::SC; t += blockDim.x) states(plain, t);
    __syncthreads();
  }

  // ---- faces (exact solver: again, the pairs out of its range alone, after
  // the loop, so that it holds no call)
  bool redo = false;
  auto faces = [&](auto &ar, int t, auto again) {
    int x, l;
    G::dec(t, G::LC, 1, x, l);
    if (x < 0) return;
    double VL[8], VR[8];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      VL[wslot(q)] = sWp[q * G::SC + t - G::step];
      VR[wslot(q)] = sWm[q * G::SC + t];
    }
    VL[HGE] = sGe[t - G::step]; VR[HGE] = sGe[t];
    VL[HGC] = P.gamma; VR[HGC] = P.gamma;
    if constexpr (decltype(again)::value) {
      if (xrs::fast_pair(xrs::Side{VL[HD], 0., VL[HP]}, xrs::Side{VR[HD], 0., VR[HP]})) return;
    }
    double F[6], fv, fe;
    if constexpr (RS == 1) {
      if constexpr (decltype(again)::value) exact_face_any<DIR>(P, P.gas, VL, VR, F, st);
      else redo |= exact_face<DIR>(P, P.gas, VL, VR, F, st);
      fv = F[FDENS] / (F[FDENS] > 0. ? VL[HD] : VR[HD]);
    } else {
      hllc64<DIR>(P, ar, VL, VR, F, fv, st);
    }
#pragma unroll
    for (int n = 0; n < 6; ++n) sF[n * G::SC + t] = F[n];
    fe = F[FDENS] * (F[FDENS] > 0. ? VL[HEI] : VR[HEI]);         // hy_getFaceFlux.F90:433-442
    if (!P.use_aux_eint) fv = fe = 0.;
    sF[FEINT * G::SC + t] = fe;
    sF[FVOLU * G::SC + t] = fv;
    if (P.sp_mf)
      seam_blocks<K, G::N0, true>(x, [&](int m, int y) { P.sp_mf[sp_line(m, y, l)] = F[FDENS]; });
  };
  ar.bad = false;
  for (int t = threadIdx.x; t < G::SC; t += blockDim.x) faces(ar, t, std::false_type());
  if constexpr (RS == 1) {
    if (redo)
      for (int t = threadIdx.x; t < G::SC; t += blockDim.x) faces(ar, t, std::true_type());
  }
  if (__syncthreads_or(ar.bad)) {
    for (int t = threadIdx.x; t < G::SC; t += blockDim.x) faces(plain, t, std::false_type());
    __syncthreads();
  }
  if (K == 1 && P.freg) {       // AMR: fine/coarse faces
    flux_register<NDIM, NX, NY, NZ, DIR, Q>(P, b, bc, qtr, sF, G::SC, fidx);
    __syncthreads();
  }

  } else {
    // replay: the stored fluxes, and the stored pressure sums in place of
    // the face-state sum N05 + P05 of the update
    flux_load<NDIM, NX, NY, NZ, DIR, Q>(P, b, qtr, sF, G::SC, fidx, [&](int t, double sp) {
      sWm[4 * G::SC + t] = sp;
      sWp[4 * G::SC + t] = 0.;
    });
    __syncthreads();
  }
  if (K == 1 && (P.fmode == 1 || P.fmode == 2)) {
    flux_store<NDIM, NX, NY, NZ, DIR, Q>(P, b, qtr, sF, G::SC, fidx,
                                         [&](int t) { return sWm[4 * G::SC + t] + sWp[4 * G::SC + t]; });
    if (P.fmode == 2) {
      if (st) atomicOr(P.status, st);
      return;
    }
  }

  // ---- update
  const double dtd = dt / delta;
  CflCand cand[K];                         // per block of the run
#pragma unroll
  for (int m = 0; m < K; ++m) { cand[m].key = 0.0; cand[m].val = 0.0; cand[m].idx = 0x7fffffff; }
  for (int t = threadIdx.x; t < G::SC; t += blockDim.x) {
    int x, l, i, j, k;
    G::dec(t, G::LC, 1, x, l);
    if (x < 0 || x >= G::N) continue;
    const int mb = G::blk_of(x);
    G::cell(x, l, qtr, i, j, k);
    const int loc = (k * NY + j) * NX + i;
    const size_t off = (size_t)pick(blk, mb) * NCB + loc;
    double U[5];
    if (FIRST) {
      const double rho = P.s_in[0][off], vx = P.s_in[1][off], vy = P.s_in[2][off], vz = P.s_in[3][off],
                   e = P.s_in[4][off];
      const double ekin = 0.5 * (vx * vx + vy * vy + vz * vz);
      U[0] = rho; U[1] = vx * rho; U[2] = vy * rho; U[3] = vz * rho; U[4] = rho * (e + ekin);
    } else {
#pragma unroll
      for (int n = 0; n < 5; ++n) U[n] = ACC[n * ncells + off];
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) U[n] = U[n] - dtd * (sF[n * G::SC + t + G::step] - sF[n * G::SC + t]);
    const double ea = sF[FEINT * G::SC + t] - sF[FEINT * G::SC + t + G::step];
    const double eb = sF[FVOLU * G::SC + t] - sF[FVOLU * G::SC + t + G::step];
    const double sp = sWm[4 * G::SC + t] + sWp[4 * G::SC + t];   // N05 + P05
    if (!LAST) {
#pragma unroll
      for (int n = 0; n < 5; ++n) ACC[n * ncells + off] = U[n];
      double *ax = AUX + (size_t)(DIR - 1) * 3 * ncells;
      ax[off] = ea; ax[ncells + off] = eb; ax[2 * ncells + off] = sp;
    } else {
#pragma unroll
      for (int n = 0; n < 5; ++n) U[n] = U[n] + 0.0;       // + dt*(Sgeo + Sphys), both +0 here
      const double rho0 = P.s_in[0][off], e0 = P.s_in[4][off];
      double IntEner = 0.0;
      if (P.use_aux_eint) {
        // n+1/2 pressure: scrch_Ptr(1) of hy_getFaceFlux.F90:551-557 and the
        // y/z averages
        double pb;
        const double sx = AUX[2 * ncells + off];
        if (NDIM == 2) {
          pb = (0.5 * sx) * 0.5 + sp * 0.25;
        } else {
          const double sy = AUX[3 * ncells + 2 * ncells + off];
          pb = ((0.5 * sx) * 0.5 + sy * 0.25) * 4.0;
          pb = (pb + sp) / 6.0;
        }
        IntEner = rho0 * e0;
        IntEner = IntEner + dt / del[0] * (AUX[off] + pb * AUX[ncells + off]);
        if (NDIM == 2) {
          IntEner = IntEner + dt / del[1] * (ea + pb * eb);
        } else {
          const double *ay = AUX + 3 * ncells;
          IntEner = IntEner + dt / del[1] * (ay[off] + pb * ay[ncells + off]);
          IntEner = IntEner + dt / del[2] * (ea + pb * eb);
        }
        IntEner = IntEner + dt * 0.;
      }
      // hy_unsplitUpdate.F90:811-893
      const double dens = rmax(U[0], P.smlrho);
      Arith<true> au;
      const Rcp rd = au.rcp(dens);
      double vx = au.by(U[1], rd), vy = au.by(U[2], rd), vz = au.by(U[3], rd);
      double ener = au.by(U[4], rd), eaux = au.by(IntEner, rd);
      if (au.bad) { vx = U[1] / dens; vy = U[2] / dens; vz = U[3] / dens; ener = U[4] / dens; eaux = IntEner / dens; }
      // hy_energyFix.F90:188-253
      const double ekin = 0.5 * (vx * vx + vy * vy + vz * vz);
      const double eint = ener - ekin - 0.0;
      double newE;
      if (!P.use_aux_eint || eint > P.eswitch * (ekin + 0.0)) newE = rmax(P.smalle, eint);
      else newE = rmax(P.smalle, eaux);
      ener = newE + ekin;
      // Eos_wrapped(MODE_DENS_EI)
      double e = newE;
      if (ener - ekin > rmax(P.smalle, P.eswitch * ekin)) e = ener - ekin;
      P.s_out[0][off] = dens; P.s_out[1][off] = vx; P.s_out[2][off] = vy; P.s_out[3][off] = vz;
      P.s_out[4][off] = e;
      if (!(isfinite(dens) && isfinite(vx) && isfinite(vy) && isfinite(vz) && isfinite(e))) st |= ST_NAN;
      // CFL: Hydro_computeDt.F90:260-284 on the new state
      const double pn = dens * e * P.gam1inv;
      const double cs = sqrt(P.gamma * pn / dens);
      double dtl = (fabs(vx - 0.) + cs) * (1.0 / del[0]);
      if (NDIM > 1) dtl = rmax(dtl, (fabs(vy - 0.) + cs) * (1.0 / del[1]));
      if (NDIM > 2) dtl = rmax(dtl, (fabs(vz - 0.) + cs) * (1.0 / del[2]));
      CflCand c; c.key = dtl * P.cfl; c.val = dtl; c.idx = loc;
#pragma unroll
      for (int m = 0; m < K; ++m)
        if (m == mb) cfl_merge(cand[m], c);
    }
  }
  if (LAST) {
    if constexpr (Q == 1) cfl_block_reduce<NX, NY, NZ>(cand[0], b, P.cfl, part);
    else cfl_parts_reduce<K>(cand, [&](int m) { return cflq + (size_t)pick(blk, m) * Q + qtr; });   // merged by k_cfl_merge
  }
  if (st) atomicOr(P.status, st);
}

}  // namespace fhy
