// hy_variant.cu -- instantiates the step kernels for one arithmetic variant.
// Compiled once per variant (see flash5_b200/build.py):
//   FHY_VARIANT=1  FP64, no FMA contraction (--fmad=false): the parity path
//   FHY_VARIANT=2  FP64 with FMA contraction
//   FHY_VARIANT=3  FP32 reconstruction / Riemann solve, FP64 update; compiled
//                  once per threads-per-CTA candidate of the direction
//                  kernels (FHY_MXSEL = 0, 1, 2), the transverse-flux pass
//                  and the dispatcher only in unit 0
#include <string.h>
#include "hy_launch.h"
#include "../../include/flash_hy.h"
#if FHY_VARIANT == 3
#include "hy_mixed.cuh"
#else
#include "hy_dir64.cuh"
#endif

#if FHY_VARIANT == 3
#ifndef FHY_MXSEL
#define FHY_MXSEL 0
#endif
#define FHY_PASTE2(a, b) a##b
#define FHY_PASTE(a, b) FHY_PASTE2(a, b)
typedef float Real;
#define FHY_ENTRY FHY_PASTE(step_mixed_nt, FHY_MXSEL)
#elif FHY_VARIANT == 2
typedef double Real;
#define FHY_ENTRY step_fp64_fma
#else
typedef double Real;
#define FHY_ENTRY step_fp64_exact
#endif

namespace fhy {

// the direction kernels take runs of blocks (full uniform 3D grids with run
// maps, the plain step)
static bool use_runs(const StepArgs &a) {
  return a.tma_run && a.nlev == 0 && a.P.blk_list == nullptr && a.P.fmode == 0 &&
         a.nlaunch == a.nblocks;
}

// ORD: sweep order of the mixed path (0 = x, y, z; 1 = z, y, x); the FP64
// variants always run x, y, z
template <int NDIM, int NX, int NY, int NZ, int DIR, bool FIRST, bool LAST, int RS, int ORD = 0>
static bool launch_dir_one(const StepArgs &a) {
#if FHY_VARIANT == 3
  using G = MxGeom<NDIM, NX, NY, NZ, DIR, RS>;
  constexpr int NT = MxThreads<NDIM, NX, NY, NZ>::pick(FHY_MXSEL);
  auto kern = k_dir_mx<NDIM, NX, NY, NZ, DIR, FIRST, LAST, RS, NT, 1, 1, ORD>;
  const int threads = NT;
  const size_t smem = G::smem_bytes();
  if (a.set_attr && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return false;
  TmaLine tl;
  memset(&tl, 0, sizeof tl);
  // full uniform grid: runs of kMxRun blocks along the sweep.  An eighth's
  // phases have at most 288 cells, so the HLLC runs have one form, that of
  // 288 threads (unit 0, step_mixed); the exact solver's quarters keep the
  // candidates
  if constexpr (NDIM == 3 && (RS == 1 || FHY_MXSEL == 0)) {
    if (use_runs(a)) {
      constexpr int Q = run_parts(true, RS == 1);
      static_assert(Q != 8 || NT == 288, "one pass of every phase of an eighth");
      using GR = MxGeom<NDIM, NX, NY, NZ, DIR, RS, kMxRun, Q>;
      auto kr = k_dir_mx<NDIM, NX, NY, NZ, DIR, FIRST, LAST, RS, NT, kMxRun, Q, ORD>;
      const size_t smr = GR::smem_bytes();
      if (a.set_attr && cudaFuncSetAttribute(kr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smr) != cudaSuccess)
        return false;
      tl = a.tma_run[DIR - 1];
      kr<<<a.nlaunch / kMxRun * Q, NT, smr, a.stream>>>(a.P, (const Real *)a.sig, a.acc, a.aux, a.ncells, a.part, a.cflq, tl);
      if (LAST)
        k_cfl_merge<NX, NY, Q><<<(a.nblocks + 255) / 256, 256, 0, a.stream>>>(a.cflq, nullptr, a.nblocks, a.P.cfl,
                                                                                   a.part);
      return cudaGetLastError() == cudaSuccess;
    }
  }
  if (NDIM == 3 && a.tma && a.nlev == 0) tl = a.tma[DIR - 1];
  kern<<<a.nlaunch, threads, smem, a.stream>>>(a.P, (const Real *)a.sig, a.acc, a.aux, a.ncells, a.part, a.cflq, tl);
#else
  static_assert(ORD == 0, "the FP64 variants sweep x, y, z");
  TmaLine tl;
  memset(&tl, 0, sizeof tl);
  if constexpr (NDIM == 3) {
    if (use_runs(a)) {
      constexpr int Q = run_parts(false, RS == 1);
      using G = Dir64<NDIM, NX, NY, NZ, DIR, Q, kMxRun>;
      auto kern = k_dir<NDIM, NX, NY, NZ, DIR, FIRST, LAST, FHY_VARIANT, RS, Q, kMxRun>;
      const size_t smem = G::smem_bytes();
      if (a.set_attr && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return false;
      // one pass of every phase at 288 threads (288 slope cells, 272 line cells)
      constexpr int most = Dir64Bounds<NDIM, NX, kMxRun>::threads;
      const int threads = a.dir_threads < most ? a.dir_threads : most;
      kern<<<a.nlaunch / kMxRun * Q, threads, smem, a.stream>>>(a.P, (const Real *)a.sig, a.acc, a.aux,
                                                                       a.ncells, a.part, a.cflq, a.tma_run[DIR - 1]);
      return cudaGetLastError() == cudaSuccess;
    }
  }
  constexpr int Q = dir64_parts<NDIM>();
  using G = Dir64<NDIM, NX, NY, NZ, DIR, Q, 1>;
  auto kern = k_dir<NDIM, NX, NY, NZ, DIR, FIRST, LAST, FHY_VARIANT, RS, Q, 1>;
  const size_t smem = G::smem_bytes();
  if (a.set_attr && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return false;
  const int threads = a.dir_threads;
  kern<<<a.nlaunch * Q, threads, smem, a.stream>>>(a.P, (const Real *)a.sig, a.acc, a.aux, a.ncells, a.part, a.cflq, tl);
#endif
  return cudaGetLastError() == cudaSuccess;
}

// one direction: a single launch, or on an AMR hierarchy one launch per
// level, finest first
template <int NDIM, int NX, int NY, int NZ, int DIR, bool FIRST, bool LAST, int RS, int ORD = 0>
static bool launch_dir(const StepArgs &a) {
  if (a.nlev == 0) {
    if (!launch_dir_one<NDIM, NX, NY, NZ, DIR, FIRST, LAST, RS, ORD>(a)) return false;
  } else {
    StepArgs b = a;
    for (int l = a.nlev; l >= 1; --l) {
      if (a.lev_count[l] == 0) continue;
      b.P.blk_list = a.lev_list[l];
      b.nlaunch = a.lev_count[l];
      if (!launch_dir_one<NDIM, NX, NY, NZ, DIR, FIRST, LAST, RS, ORD>(b)) return false;
      b.set_attr = false;
    }
  }
#if FHY_VARIANT != 3
  // the CTAs that share a block left a CFL candidate each
  constexpr int Q = dir64_parts<NDIM>();
  if (LAST && Q > 1 && a.P.fmode != 2) {
    const int *list = a.nlev ? a.leaves : a.P.blk_list;
    const int n = a.nlev ? a.nleaves : a.nlaunch;
    if (use_runs(a)) k_cfl_merge<NX, NY, run_parts(false, RS == 1)><<<(n + 255) / 256, 256, 0, a.stream>>>(a.cflq, list, n, a.P.cfl, a.part);
    else k_cfl_merge<NX, NY, Q><<<(n + 255) / 256, 256, 0, a.stream>>>(a.cflq, list, n, a.P.cfl, a.part);
    return cudaGetLastError() == cudaSuccess;
  }
#endif
  return true;
}

// the transverse-flux pass (all leaves on an AMR hierarchy)
#if FHY_VARIANT != 3 || FHY_MXSEL == 0
template <int NDIM, int NX, int NY, int NZ>
static bool launch_sig(const StepArgs &a) {
  auto kern = k_sig<NDIM, NX, NY, NZ, Real, FHY_VARIANT>;
  const size_t smem = SigStage<NDIM, NX, NY, NZ>::smem_bytes();
  if (a.set_attr && smem > 48 * 1024 &&
      (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
       cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
           cudaSuccess))
    return false;
  if (a.nlev == 0) {
    kern<<<a.nlaunch, a.threads, smem, a.stream>>>(a.P, (Real *)a.sig);
  } else {
    DevParams P = a.P;
    P.blk_list = a.leaves;
    kern<<<a.nleaves, a.threads, smem, a.stream>>>(P, (Real *)a.sig);
  }
  return cudaGetLastError() == cudaSuccess;
}
#if FHY_VARIANT == 3
bool sig_mixed(const StepArgs &a, int ndim, int nx, int ny, int nz) {
  if (ndim == 2 && nx == 8 && ny == 8) return launch_sig<2, 8, 8, 1>(a);
  if (ndim == 2 && nx == 16 && ny == 16) return launch_sig<2, 16, 16, 1>(a);
  if (ndim == 3 && nx == 8 && ny == 8 && nz == 8) return launch_sig<3, 8, 8, 8>(a);
  return false;
}
#endif
#else
template <int NDIM, int NX, int NY, int NZ>
static bool launch_sig(const StepArgs &a) { return sig_mixed(a, NDIM, NX, NY, NZ); }
#endif

// RS: 0 = HLLC, 1 = exact Riemann solver
template <int NDIM, int NX, int NY, int NZ, int RS>
static int run_rs(const StepArgs &a) {
  if (!a.no_sig && !launch_sig<NDIM, NX, NY, NZ>(a)) return -2;
  int nl = 1;
  const int nsig = a.no_sig ? 0 : 1;
  if (a.nlev > 0) {
    nl = 0;
    for (int l = 1; l <= a.nlev; ++l) nl += a.lev_count[l] > 0;
  }
  // z, y, x on the mixed path when asked (the plain step and AMR; the split
  // step's flux modes keep x, y, z).  The middle direction of 3D has the
  // same AUX slot in both orders, so it shares the x, y, z kernel.
  bool ok;
  if constexpr (FHY_VARIANT == 3) {
    if (a.sweep == 1 && a.P.fmode == 0) {
      if constexpr (NDIM == 2)
        ok = launch_dir<NDIM, NX, NY, NZ, 2, true, false, RS, 1>(a) &&
             launch_dir<NDIM, NX, NY, NZ, 1, false, true, RS, 1>(a);
      else
        ok = launch_dir<NDIM, NX, NY, NZ, 3, true, false, RS, 1>(a) &&
             launch_dir<NDIM, NX, NY, NZ, 2, false, false, RS>(a) &&
             launch_dir<NDIM, NX, NY, NZ, 1, false, true, RS, 1>(a);
      return ok ? nsig + NDIM * nl + (NDIM == 3 && use_runs(a) ? 1 : 0) : -2;
    }
  }
  if constexpr (NDIM == 2) {
    ok = launch_dir<NDIM, NX, NY, NZ, 1, true, false, RS>(a) && launch_dir<NDIM, NX, NY, NZ, 2, false, true, RS>(a);
    return ok ? nsig + 2 * nl : -2;
  } else {
    ok = launch_dir<NDIM, NX, NY, NZ, 1, true, false, RS>(a) &&
         launch_dir<NDIM, NX, NY, NZ, 2, false, false, RS>(a) &&
         launch_dir<NDIM, NX, NY, NZ, 3, false, true, RS>(a);
    // + the CFL merge of the runs / of the parts of the FP64 kernel's blocks
    const bool merge = FHY_VARIANT == 3 ? use_runs(a) : a.P.fmode != 2;
    return ok ? nsig + 3 * nl + (merge ? 1 : 0) : -2;
  }
}

template <int NDIM, int NX, int NY, int NZ>
static int run(const StepArgs &a) {
  return a.P.riemann == FLASH_HY_RS_EXACT ? run_rs<NDIM, NX, NY, NZ, 1>(a) : run_rs<NDIM, NX, NY, NZ, 0>(a);
}

int FHY_ENTRY(const StepArgs &a, int ndim, int nx, int ny, int nz) {
  if (ndim == 2 && nx == 8 && ny == 8) return run<2, 8, 8, 1>(a);
  if (ndim == 2 && nx == 16 && ny == 16) return run<2, 16, 16, 1>(a);
  if (ndim == 3 && nx == 8 && ny == 8 && nz == 8) return run<3, 8, 8, 8>(a);
  return -1;
}

#if FHY_VARIANT == 3 && FHY_MXSEL == 0
int step_mixed(const StepArgs &a, int ndim, int nx, int ny, int nz) {
  switch (use_runs(a) && a.P.riemann != FLASH_HY_RS_EXACT ? 0 : a.mx_sel) {
    case 0: return step_mixed_nt0(a, ndim, nx, ny, nz);
    case 2: return step_mixed_nt2(a, ndim, nx, ny, nz);
    default: return step_mixed_nt1(a, ndim, nx, ny, nz);
  }
}
int mx_threads_of(int sel, int ndim, int nx) {
  if (ndim == 3) return MxThreads<3, 8, 8, 8>::pick(sel);
  return nx == 8 ? MxThreads<2, 8, 8, 1>::pick(sel) : MxThreads<2, 16, 16, 1>::pick(sel);
}
#endif

#if FHY_VARIANT == 1
template <int NDIM, int NX, int NY, int NZ>
static int run_cfl(const StepArgs &a) {
  k_cfl<NDIM, NX, NY, NZ><<<a.nlaunch, a.threads, 0, a.stream>>>(a.P, a.part);
  return cudaGetLastError() == cudaSuccess ? 1 : -2;
}
int cfl_state(const StepArgs &a, int ndim, int nx, int ny, int nz) {
  if (ndim == 2 && nx == 8 && ny == 8) return run_cfl<2, 8, 8, 1>(a);
  if (ndim == 2 && nx == 16 && ny == 16) return run_cfl<2, 16, 16, 1>(a);
  if (ndim == 3 && nx == 8 && ny == 8 && nz == 8) return run_cfl<3, 8, 8, 8>(a);
  return -1;
}
size_t sig_bytes_per_block(int ndim, int nx, int ny, int nz, int real_bytes) {
  size_t box = (size_t)(nx + 2) * (ndim > 1 ? ny + 2 : 1) * (ndim > 2 ? nz + 2 : 1);
  return box * 6 * ndim * real_bytes;
}
#endif

}  // namespace fhy
