// tc_ptx.cuh -- tcgen05, mbarrier and bulk-copy primitives (inline PTX) shared
// by the tensor-core kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace rbc {
namespace dev {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// tcgen05 shared-memory matrix descriptor, no swizzle: start address, leading
// (K-direction) and stride (M/N-direction) byte offsets between core matrices.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  return d;
}

__device__ __forceinline__ void mbar_init(uint64_t* m, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count));
}
__device__ __forceinline__ bool mbar_try(uint64_t* m, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

constexpr long long kWaitLimit = 1LL << 22;  // try_wait polls before a completion wait is declared lost
__device__ __forceinline__ void mbar_arrive(uint64_t* m) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(m)) : "memory");
}
// one arrival that also announces `bytes` of asynchronous transfer to come
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* m, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                   smem_u32(m)),
               "r"(bytes)
               : "memory");
}
// bulk copy global -> shared (16-byte aligned, size a multiple of 16), its
// completion counted on the mbarrier's transaction count
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* m) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(m))
               : "memory");
}

// bounded wait of one warp for phase `parity` of an mbarrier: lane 0 polls
// (giving up early once the tile is aborted), the outcome goes to all lanes
__device__ __forceinline__ bool warp_mbar_wait(uint64_t* m, uint32_t parity, long long limit,
                                               volatile int* abort_flag) {
  int ok = 0;
  if ((threadIdx.x & 31) == 0) {
    for (long long i = 0; i < limit; i++) {
      if (mbar_try(m, parity)) {
        ok = 1;
        break;
      }
      if ((i & 1023) == 1023 && *abort_flag) break;
    }
    if (!ok) *abort_flag = 1;
  }
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

}  // namespace dev
}  // namespace rbc
