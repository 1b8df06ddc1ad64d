// Device helpers shared by the kernel files: the batch's work-item lookup, the graded
// score and the filter step, and bulk asynchronous copies with mbarrier completion.
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

// One recursive-filter step (core/tools/de_dense.cpp:419): int32 carry, +2^14
// rounding, arithmetic shift.
__device__ __forceinline__ int32_t rf_step(int32_t c, int32_t f, int32_t a) {
  return c + ((a * (f - c) + (1 << 14)) >> 15);
}

__device__ __forceinline__ uint32_t pack2(int32_t lo, int32_t hi) {
  return (uint32_t(uint16_t(lo))) | (uint32_t(hi) << 16);
}

// Packed census words (windows of <= 48 bits): lo32 = bits 0..31; hi32 = bits
// 32..47 | guard bit 19 (left words only) | pixel byte at bits 20..27.  Then
// (left.hi - right.hi) >> 20 is exactly L - R: the guard keeps the census bits from
// borrowing into the pixel field.  (left ^ right) masked to the census bits gives the
// Hamming input as before.
constexpr uint32_t kCensusHiMask = 0xFFFFu;
constexpr uint32_t kGuard = 1u << 19;
constexpr int kPixShift = 20;

constexpr int kVolBias = 32768;

// The volume holds scores with a bias of 32768 (the filter commutes with it), so that a
// 16-bit value is one byte permute away from a float in the column kernel.
// Score table: (h, m) -> Q14 score + bias, h = Hamming distance, m = |L - R| clamped to
// TS-1 (exact: the AD score saturates at ad_trunc < TS).  Stored m-major with 64
// h-entries per row, so the many lookups that share the saturated m read adjacent
// entries, not one bank.
template <int TS, int CP>
struct ScoreTable {
  __host__ __device__ static constexpr size_t bytes() { return size_t(TS) * 64 * 2; }
};

template <bool PACKED, int TS, int CP>
__device__ __forceinline__ int32_t graded(uint64_t lw, uint64_t rw, const void* tab,
                                          const uint8_t* sLp, const uint8_t* sRp, int xl,
                                          int xr) {
  int h, ad;
  if (PACKED) {
    const uint32_t lh = uint32_t(lw >> 32), rh = uint32_t(rw >> 32);
    h = __popc(uint32_t(lw) ^ uint32_t(rw)) + __popc((lh ^ rh) & kCensusHiMask);
    ad = int(__usad(lh >> kPixShift, rh >> kPixShift, 0u));
  } else {
    h = __popcll(lw ^ rw);
    ad = abs(int(sLp[xl]) - int(sRp[xr]));
  }
  if (TS == 16) ad = min(ad, 15);
  return static_cast<const uint16_t*>(tab)[ad * 64 + h];
}

// The table, by the whole CTA (any multiple of 32 threads).  A thread keeps its Hamming
// distance, so the parameter tables are read once per thread at diverging addresses and
// then at one address for all (both per entry: 6-9 k clocks at the start of every row CTA).
template <int TS>
__device__ __forceinline__ void fill_scores(const DevCfg& cfg, void* tab) {
  uint16_t* t16 = static_cast<uint16_t*>(tab);
  const int per = max(1, int(blockDim.x) >> 6);       // threads that share a distance
  for (int h = threadIdx.x & 63; h < 64; h += blockDim.x) {
    const int32_t c = int32_t(cfg.tbl[h]) * (1024 - cfg.wq);
    for (int m = threadIdx.x >> 6; m < TS; m += per)
      t16[m * 64 + h] = uint16_t(kVolBias + ((c + int32_t(cfg.adt[m]) * cfg.wq) >> 10));
  }
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
