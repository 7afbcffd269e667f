// hy_tma.cuh -- TMA tile copies into shared memory for the direction kernels.
#pragma once
#include <cuda.h>
#include "../../include/flash_hy.h"

namespace fhy {

// ---------------------------------------------------------------------------
// TMA staging of the direction kernels' line stencils (uniform 3D grids).
// Each state variable is described by tensor maps over its natural layout
// (x fastest, then y, then z of every block: dims 8 x 8 x 8*nblocks); one
// 3D tile copy brings a block's interior (box 8 x 8 x 8) and one a
// neighbour's 4-cell slab along the sweep direction (box 4 x 8 x 8,
// 8 x 4 x 8 or 8 x 8 x 4), straight into the staged layout below.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// one bounded poll of phase `parity`; true once it has completed
__device__ __forceinline__ bool mbar_try(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// 3D tile copy global -> shared through a tensor map (no multicast)
// fetch a tensor map into the descriptor cache ahead of its first copy
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<unsigned long long>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int c0, int c1, int c2,
                                            unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];\n" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// SM cycles (about a second) a CTA waits for its tile copies before it gives
// up (FLASH_HY_ERR_TIMEOUT)
constexpr long long kTmaWaitCycles = 1LL << 31;

// Bounded wait of the whole CTA for its tile copies (phase 0 of bar).  False
// where it gave up: FLASH_HY_ERR_TIMEOUT is flagged, the copies in flight
// have been waited for (bounded) once more, and the CTA leaves.
__device__ __forceinline__ bool tma_wait(unsigned long long *bar, unsigned *status) {
  bool done = false;
  const long long t0 = clock64();
  while (!done && clock64() - t0 < kTmaWaitCycles) done = mbar_try(bar, 0);
  if (!__syncthreads_or(!done)) return true;
  if (threadIdx.x == 0) atomicOr(status, (unsigned)FLASH_HY_ERR_TIMEOUT);
  const long long t1 = clock64();
  while (clock64() - t1 < kTmaWaitCycles && !mbar_try(bar, 0)) {
  }
  return false;
}

}  // namespace fhy
