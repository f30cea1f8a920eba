// rh_device.cuh — constants of the cell time step and PTX helpers (mbarriers and
// asynchronous copies into shared memory) of the pencil kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "rh_bulk.h"

namespace rh {

// ---------------------------------------------------------------------------
// Constants of cmpdt (godunov_utils.f90:228-333) with bb=0,
// induction=.false.  With zero magnetic field the reference's fast speed
// sqrt(c2+sqrt(c2**2)) equals sqrt(a2) exactly in IEEE arithmetic
// (sqrt(fl(x*x)) == x).
// ---------------------------------------------------------------------------
struct CflConst {
  double gamma, gm1, smallr, smallp;  // smallp = smallc**2/gamma
  double cdx_smallc;                  // courant*dx/smallc
  double two_cdx;                     // 2*courant*dx
  double two_c;                       // 2*courant
  double gsum_dx;                     // (|gx|+|gy|+|gz|)*dx
  double k0;                          // 2*courant*dx/(1+sqrt(1+2*courant*1e-4)): dt*ctot without gravity
  int ndim;
};

// ---------------------------------------------------------------------------
// PTX helpers: mbarrier + bulk async copy (global -> shared, no multicast)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// Returns true once the phase with the given parity has completed.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst_smem)),
      "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// asynchronous copy of 16 aligned bytes by one thread
__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src_gmem) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)), "l"(src_gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most N of this thread's groups are still in flight.
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

}  // namespace rh
