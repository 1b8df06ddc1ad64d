// Device helpers shared by the kernel files: the batch's work-item lookup, and bulk
// asynchronous copies with mbarrier completion.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "de_internal.h"

namespace de {
namespace {

__device__ __forceinline__ int find_pair(const int* prefix, int n, int item) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= item) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Bulk asynchronous copies (cp.async.bulk, the TMA engine's 1-D form) with
// mbarrier completion.  Every wait is bounded: if a phase never completes the
// kernel records it in the batch status word and runs on to its end.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return uint32_t(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
constexpr int kWaitLimit = 1 << 22;                  // try_wait rounds before giving up
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, int* err,
                                          int limit = kWaitLimit) {
  for (int i = 0; i < limit; ++i)
    if (mbar_test(bar, parity)) return;
  if (err) atomicExch(err, 1);
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

}  // namespace
}  // namespace de
