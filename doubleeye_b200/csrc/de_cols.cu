// k_cols_tm: vertical forward, vertical backward + top-2 + neighbours, with the forward
// results held in tensor memory; the column kernel of work too small to fill the GPU.
//
// Vertical passes: core/tools/de_dense.cpp:490-507.  Top-2 semantics: :1276-1292
// (ascending k, strictly greater, ties keep the smaller k), sub-pixel neighbour capture
// :1276-1285.
//
// With one pair the streaming kernel (k_cols) has one or two warps a scheduler, each
// doing a column's loads, filter, top-2 and lane merges in turn, and a second trip of the
// volume through memory (the backward pass needs the forward results in reverse).  Here
// the stages have warps of their own and the forward results stay on chip: nothing on
// this path is a contraction, so the 256 KB of tensor memory per SM are free.  A thread
// that owns two disparities of a column needs one 32-bit word a row, and a tensor-memory
// lane has 512 words, so 128 threads keep 256 filter chains of 512 rows.  Rows above the
// last 512 go back to the volume in place.
//
// A CTA (one per SM, persistent) takes tiles of 128 words a row: 4, 2 or 1 adjacent
// columns at Dpad 64, 128, 192/256, 512 contiguous bytes of every image row.  Its warps:
//   12-14 producers: 32-row stages of 16-byte asynchronous copies into a 5-stage ring,
//         running ahead into the next tile while this one's backward pass computes (one
//         512-byte bulk copy a row took 69 clocks each to issue; a second and third
//         producer warp gained 6 us of 89 at 848x480 D=128);
//   15    the next tile's filter coefficients, as floats;
//   0-3   the filter chains: a thread steps its two disparities down the column, 32 rows
//         a block, each block's results one tcgen05.st; then up again from tcgen05.ld.
//         The next block's words are read while a block is filtered;
//   4-11  the top-2: eight lanes a row, 32 disparities each, so no shuffle chain is in
//         the filter's way.
// Block hand-offs are mbarriers; every wait is bounded (a wait that runs out sets the
// batch status word, later ones give up at once, each lane waits for its own copies and the
// tensor memory is freed).
//
// The step runs on the FP32 pipe, exactly.  With u = v + 32768 (the volume's bias) and
// values held as 2^23 + u, c + ((a (f - c) + 2^14) >> 15) = floor(u_c + 1/2 + a' (u_f -
// u_c)), a' = a / 2^15: the difference is exact, the fused multiply-add onto 2^22 + u_c +
// 1/2 rounds down to a multiple of 1/2, and adding 2^22 rounding down leaves the floor.
// Four full-rate instructions; the integer step and its sign extensions are mostly
// half-rate ALU, which the top-2's minima and maxima need (integer chains: 91 us at
// 848x480 D=128, these 83).  Keys leave the chain as u << 16 | 255 - k (one integer
// multiply-add, which also zeroes a disparity with no candidate).
//
// What bounds it: the chains' latency, about 42 clocks a row down and 45 up with one
// chain warp a scheduler.  Measured (column stage, one pair, streaming -> this as first
// written; the producers' start since took another 1-3 us off each):
// 320x240 D=64 52 -> 24 us, 450x375 D=60 79 -> 30, 848x480 D=64 101 -> 56, 848x480 D=128
// 124 -> 83, 640x480 D=256 179 -> 124, 1280x720 D=64 186 -> 137.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "de_dev.cuh"
#include "de_internal.h"

namespace de {
namespace {

constexpr int kBlk = 32;                 // rows per block
constexpr int kRow = 128;                // words per tile row
constexpr int kStages = 5;               // ring: 80 KB, 160 rows ahead
constexpr int kOut = 3;                  // blocks between the chains and the top-2
constexpr int kTm = 512;                 // tensor-memory columns: all of them
constexpr int kThreads = 512;
constexpr uint32_t kZero2 = 0x80008000u; // two zero scores

// A poll that returns at once.  Against the suspending form (try_wait) the column stage
// took 23 instead of 27 us at 320x240 D=64, each launch timed by itself; no difference at
// 848x480.
__device__ __forceinline__ bool mbar_poll(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits with a memory: after one has run out the rest return quickly.
struct Waiter {
  int* err;
  bool dead = false;
  __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity) {
    if (!mbar_poll(bar, parity)) dead = slow(bar, parity, err, dead);
  }
  // By a whole warp, whose lanes leave together: the tensor-memory instructions want them at
  // the same one.  `seen`: what this lane's poll ahead of the wait returned.
  __device__ __forceinline__ void wait_warp(uint64_t* bar, uint32_t parity, bool seen = false) {
    if (__all_sync(0xffffffffu, seen) || __all_sync(0xffffffffu, mbar_poll(bar, parity))) return;
    dead = __any_sync(0xffffffffu, slow(bar, parity, err, dead));
  }
  static __device__ __noinline__ bool slow(uint64_t* bar, uint32_t parity, int* err, bool dead) {
    const int limit = dead ? 16 : kWaitLimit;
    for (int i = 0; i < limit; ++i)
      if (mbar_poll(bar, parity)) return dead;
    if (err) atomicExch(err, 1);
    return true;
  }
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// One arrival a warp, after all its lanes' accesses; predicated, so that no lane leaves the
// others.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  asm volatile(
      "{\n .reg .pred p;\n setp.eq.s32 p, %1, 0;\n"
      " @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(smem_addr(bar)), "r"(lane)
      : "memory");
}

// Tensor memory as thread-private storage: lane i of a warp reads back the words it wrote.
__device__ __forceinline__ void tm_alloc(uint32_t* slot, uint32_t cols) {     // one warp
  __syncwarp();                          // (its first lane has set up the barriers)
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_addr(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_free(uint32_t base, uint32_t cols) {       // the same warp
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tm_st(uint32_t addr, const uint32_t (&r)[kBlk]) {
  static_assert(kBlk == 32, "one store a block");
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {"
      "%1, %2, %3, %4, %5, %6, %7, %8, "
      "%9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, "
      "%25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
      "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tm_ld(uint32_t addr, uint32_t (&r)[kBlk]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {"
      "%0, %1, %2, %3, %4, %5, %6, %7, "
      "%8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, "
      "%24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tm_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// The registers pass through, so no use of them moves ahead of the wait.
__device__ __forceinline__ void tm_wait_ld(uint32_t (&r)[kBlk]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ float fbits(uint32_t v) { return __uint_as_float(v); }

// RK: the filtered costs also go back to the volume, for the reverse match; the top-2
// warps write them (from the chains, whose latency bounds the kernel, it cost 23 us more at
// 848x480 D=64).
template <int G, bool RK>
__global__ void __launch_bounds__(kThreads, 1) k_cols_tm(DevCfg cfg, Batch b, int cstride) {
  constexpr int DP = 64 * G;                          // Dpad
  constexpr int KW = DP / 2;                          // words per column
  constexpr int NCOL = kRow / KW;                     // columns per tile
  constexpr int LPC = G == 3 ? 8 : 2 * G;             // top-2 lanes per column and row
  extern __shared__ __align__(128) uint32_t sm[];
  uint32_t* const ring = sm;                          // [kStages][kBlk][kRow]
  uint32_t* const outb = ring + kStages * kBlk * kRow;    // [kOut][kBlk][2 kRow] keys
  float* const coef = reinterpret_cast<float*>(outb + kOut * kBlk * 2 * kRow);  // [2][NCOL][cstride]
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], ofull[kOut], oempty[kOut],
      cfull[2], cempty[2], cfirst;
  __shared__ uint32_t tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total = b.cols_prefix[b.n];
  const int hw = cfg.hw, hh = cfg.hh, dmin = cfg.dmin;
  // coefficients of a tile's columns; past the image 1, the step that leaves the state
  // as it is (t-th of n threads)
  auto load_coef = [&](int tile, int buf, int t, int nt) {
    const int pi = find_pair(b.cols_prefix, b.n, tile);
    const DevPair& P = b.p[pi];
    const int W = P.W, H = P.H, xb = hw + dmin + (tile - b.cols_prefix[pi]) * NCOL;
    const int n = ((H - hh + kBlk - 1) / kBlk * kBlk + 1) * NCOL;
    float* const dst = coef + buf * NCOL * cstride;
    for (int i0 = t; i0 < n; i0 += 8 * nt) {
      uint32_t a[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + nt * u, y = hh + i / NCOL, x = min(xb + i % NCOL, W - 1);
        a[u] = (i < n && y < H) ? uint32_t(P.ay[size_t(y) * W + x]) : (1u << 15);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + nt * u;
        if (i < n) dst[(i % NCOL) * cstride + i / NCOL] = float(a[u]) * (1.f / 32768.f);
      }
    }
  };
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], 32); mbar_init(&empty[i], 4); }
    for (int i = 0; i < kOut; ++i) { mbar_init(&ofull[i], 4); mbar_init(&oempty[i], 8); }
    for (int i = 0; i < 2; ++i) { mbar_init(&cfull[i], 1); mbar_init(&cempty[i], 4); }
    mbar_init(&cfirst, 256);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tm_alloc(&tmem, kTm);
  __syncthreads();
  Waiter wt{b.err};

  if (warp < 4) {
    // ---- the filter chains --------------------------------------------------------
    const int col = (G == 3) ? 0 : tid / KW;          // G == 3: words 96.. carry nothing
    const int k0 = 2 * (tid - col * KW);
    const uint32_t tb = tmem + (uint32_t(warp) << 21);     // this warp's 32 lanes
    const float kHalf = -4194304.f + 0.5f, kUp = 4194304.f;  // 2^23 -> 2^22 + 1/2, and back
    uint32_t st = 0, sph = 0, ob = 0, oph = 0;
    int it = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++it) {
      const int pi = find_pair(b.cols_prefix, b.n, tile);
      const DevPair& P = b.p[pi];
      const int W = P.W, H = P.H;
      const int x = hw + dmin + (tile - b.cols_prefix[pi]) * NCOL + col;
      const int kmax = x < W - hw ? min(P.D - 1, x - hw - dmin) : -1;
      const uint32_t m0 = k0 <= kmax ? 65536u : 0u, i0 = k0 <= kmax ? uint32_t(255 - k0) : 0u;
      const uint32_t m1 = k0 < kmax ? 65536u : 0u, i1 = k0 < kmax ? uint32_t(254 - k0) : 0u;
      const int yin = H - hh;                         // rows >= yin have zero input
      const int nb = (H - hh + kBlk - 1) / kBlk, nbl = (yin - hh + kBlk - 1) / kBlk;
      const int nspill = max(0, nb - kTm / kBlk);     // blocks that do not fit on chip
      const size_t rs = size_t(W) * KW;               // image row in words
      uint32_t* const gcol = reinterpret_cast<uint32_t*>(P.vol) + size_t(x) * KW + k0 / 2;
      const float* const cf = coef + ((it & 1) * NCOL + col) * cstride;
      if (it == 0) wt.wait_warp(&cfirst, 0);
      else wt.wait_warp(&cfull[it & 1], ((it - (it & 1 ? 1 : 2)) >> 1) & 1);
      float f0 = 8388608.f + 32768.f, f1 = f0;
      auto step = [&](uint32_t c, float a) {
        const float c0 = fbits(__byte_perm(c, 0x4B000000u, 0x7610));
        const float c1 = fbits(__byte_perm(c, 0x4B000000u, 0x7632));
        f0 = __fadd_rd(__fmaf_rd(a, f0 - c0, c0 + kHalf), kUp);
        f1 = __fadd_rd(__fmaf_rd(a, f1 - c1, c1 + kHalf), kUp);
      };
      bool ready = false;                             // the next stage has landed (polled ahead)
      auto take = [&](uint32_t (&c)[kBlk]) {          // the next block's words
        wt.wait_warp(&full[st], sph, ready);
        const uint32_t* s = ring + st * (kBlk * kRow) + tid;
#pragma unroll
        for (int r = 0; r < kBlk; ++r) c[r] = s[r * kRow];
      };
      auto down = [&](int blk, uint32_t (&c)[kBlk], uint32_t (&nx)[kBlk]) {
        const uint32_t mine = st;                     // block blk + 1's stage
        if (blk + 1 < nbl) {
          take(nx);
          if (++st == kStages) { st = 0; sph ^= 1; }
          ready = mbar_poll(&full[st], sph);
        }
        const int rows = yin - (hh + blk * kBlk);     // rows of the block with input
        if (rows < kBlk) {
#pragma unroll
          for (int r = 0; r < kBlk; ++r) c[r] = r < rows ? c[r] : kZero2;
        }
#pragma unroll
        for (int q = 0; q < kBlk / 4; ++q) {
          const float4 a = reinterpret_cast<const float4*>(cf + blk * kBlk)[q];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            step(c[4 * q + u], u == 0 ? a.x : u == 1 ? a.y : u == 2 ? a.z : a.w);
            c[4 * q + u] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x5410);
          }
        }
        if (blk >= nspill) {
          tm_st(tb + uint32_t(blk - nspill) * kBlk, c);
        } else if (k0 <= kmax) {
          uint32_t* g = gcol + size_t(hh + blk * kBlk) * rs;
#pragma unroll
          for (int r = 0; r < kBlk; ++r) __stcg(g + r * rs, c[r]);
        }
        if (blk < nspill) __syncwarp();               // (lanes with and without a store)
        if (blk + 1 < nbl) {
          warp_arrive(&empty[mine], lane);
        }
      };
      uint32_t ca[kBlk], cb[kBlk];
      if (nbl > 0) {
        take(ca);
        warp_arrive(&empty[st], lane);
        if (++st == kStages) { st = 0; sph ^= 1; }
        ready = mbar_poll(&full[st], sph);
      }
      for (int blk = 0; blk < nb; blk += 2) {
        down(blk, ca, cb);
        if (blk + 1 < nb) down(blk + 1, cb, ca);
      }
      tm_wait_st();
      // backward from H-1 (its value is the forward one; rows past it carry it through)
      auto fetch = [&](int blk, uint32_t (&c)[kBlk]) {
        if (blk >= nspill) {
          tm_ld(tb + uint32_t(blk - nspill) * kBlk, c);
        } else {
          const uint32_t* g = gcol + size_t(hh + blk * kBlk) * rs;
#pragma unroll
          for (int r = 0; r < kBlk; ++r) c[r] = (k0 <= kmax) ? __ldcg(g + r * rs) : kZero2;
          __syncwarp();
        }
      };
      bool room = false;
      auto up = [&](int blk, uint32_t (&c)[kBlk], uint32_t (&nx)[kBlk]) {
        float next = cf[blk * kBlk + kBlk];           // coefficient at y + 1
        if (blk >= nspill) tm_wait_ld(c);
        if (blk > 0) fetch(blk - 1, nx);
        wt.wait_warp(&oempty[ob], oph ^ 1, room);
        uint32_t* o = outb + ob * (kBlk * 2 * kRow) + 2 * tid;
        const uint32_t mine = ob;
        if (++ob == kOut) { ob = 0; oph ^= 1; }
        room = mbar_poll(&oempty[ob], oph ^ 1);
#pragma unroll
        for (int q = kBlk / 4 - 1; q >= 0; --q) {
          const float4 a = reinterpret_cast<const float4*>(cf + blk * kBlk)[q];
#pragma unroll
          for (int u = 3; u >= 0; --u) {
            step(c[4 * q + u], u == 3 ? next : u == 2 ? a.w : u == 1 ? a.z : a.y);
            *reinterpret_cast<uint2*>(o + (4 * q + u) * 2 * kRow) =
                make_uint2(__float_as_uint(f0) * m0 + i0, __float_as_uint(f1) * m1 + i1);
          }
          next = a.x;
        }
        warp_arrive(&ofull[mine], lane);
      };
      fetch(nb - 1, ca);
      for (int blk = nb - 1; blk >= 0; blk -= 2) {
        up(blk, ca, cb);
        if (blk > 0) up(blk - 1, cb, ca);
      }
      warp_arrive(&cempty[it & 1], lane);
    }
  } else if (warp < 12) {
    // ---- the top-2 ------------------------------------------------------------------
    const int t = tid - 128;
    if (int(blockIdx.x) < total) {                    // the first tile's coefficients
      load_coef(blockIdx.x, 0, t, 256);
      mbar_arrive(&cfirst);
    }
    const int r = t >> 3, s = t & 7;                  // tile row, 32-disparity segment
    const int col = (G == 3) ? 0 : s / (2 * G);
    uint32_t n = 0;                                   // block count over the tiles
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const int pi = find_pair(b.cols_prefix, b.n, tile);
      const DevPair& P = b.p[pi];
      const int W = P.W, yin = P.H - hh;
      const int x = hw + dmin + (tile - b.cols_prefix[pi]) * NCOL + col;
      const int nb = (P.H - hh + kBlk - 1) / kBlk;
      for (int blk = nb - 1; blk >= 0; --blk, ++n) {
        const int y = hh + blk * kBlk + r;
        const uint32_t ob = n % kOut;
        wt.wait(&ofull[ob], (n / kOut) & 1);
        const uint32_t* row = outb + (ob * kBlk + r) * (2 * kRow);
        const uint4* seg = reinterpret_cast<const uint4*>(row + s * 32);
        // RK: this lane's 32 costs of the row go back (where they came from: the chains are
        // past them)
        uint2* const vrow = RK && x < W - hw && y < yin && 32 * s < NCOL * DP
                                ? reinterpret_cast<uint2*>(P.vol + (size_t(y) * W + x) * DP) + 8 * (s % (DP / 32))
                                : nullptr;
        uint32_t p0 = 0, p1 = 0;
        // two more keys: the greatest of three, and their median against the second.
        // The keys are distinct, but for zeros (no candidate); a key names its own
        // disparity, so the eight lanes may read their segments' 16-byte groups in
        // different orders, each in another bank group.
        auto add2 = [&](uint32_t ka, uint32_t kb) {
          const uint32_t sum = p0 + ka + kb;
          const uint32_t hi = __vimax3_u32(p0, ka, kb), lo = __vimin3_u32(p0, ka, kb);
          p0 = hi;
          p1 = max(p1, sum - hi - lo);
        };
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 v = seg[i ^ s];
          add2(v.x, v.y);
          add2(v.z, v.w);
          if (RK && vrow)
            __stcg(vrow + (i ^ s), make_uint2(__byte_perm(v.x, v.y, 0x7632),
                                              __byte_perm(v.z, v.w, 0x7632)));
        }
#pragma unroll
        for (int o = 1; o < LPC; o <<= 1) {
          const uint32_t o0 = __shfl_xor_sync(0xffffffffu, p0, o);
          const uint32_t o1 = __shfl_xor_sync(0xffffffffu, p1, o);
          const uint32_t m = min(p0, o0);
          p0 = max(p0, o0);
          p1 = __vimax3_u32(p1, o1, m);
        }
        // the winner's neighbours
        const int kw = 255 - int(p0 & 255u);
        auto cost = [&](int k) {
          const uint32_t key = row[col * DP + k];
          return key ? int32_t(key >> 16) - 32768 : -32768;
        };
        const int32_t nm = p0 && kw >= 1 ? cost(kw - 1) : -32768;
        const int32_t np = p0 && kw + 1 < DP ? cost(kw + 1) : -32768;
        warp_arrive(&oempty[ob], lane);
        if (s % LPC == 0 && x < W - hw && y < yin) {
          const size_t i = size_t(y) * W + x;
          P.key0[i] = __byte_perm(p0, 0u, 0x4320);    // v + 32768 << 8 | 255 - k
          P.key1[i] = __byte_perm(p1, 0u, 0x4320);
          P.nb[i] = __byte_perm(uint32_t(nm), uint32_t(np), 0x5410);
        }
      }
    }
  } else if (warp < 15) {
    // ---- producers: three warps take the stages in turn -----------------------------
    uint32_t n = 0;                                   // blocks so far, over the tiles
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const int pi = find_pair(b.cols_prefix, b.n, tile);
      const DevPair& P = b.p[pi];
      const int W = P.W, yin = P.H - hh;
      const int xb = hw + dmin + (tile - b.cols_prefix[pi]) * NCOL;
      const uint32_t bytes = uint32_t(min(NCOL, W - hw - xb)) * DP * 2;
      const int nbl = (yin - hh + kBlk - 1) / kBlk;
      for (int blk = 0; blk < nbl; ++blk, ++n) {
        if (int(n % 3) != warp - 12) continue;
        const uint32_t st = n % kStages, sph = (n / kStages) & 1;
        const int y0 = hh + blk * kBlk, rows = min(kBlk, yin - y0);
        wt.wait(&empty[st], sph ^ 1);
        const uint8_t* src = reinterpret_cast<const uint8_t*>(P.vol + (size_t(y0) * W + xb) * DP) +
                             16 * lane;
        uint32_t* dst = ring + st * (kBlk * kRow) + 4 * lane;
        if (16 * uint32_t(lane) < bytes) {
#pragma unroll
          for (int r = 0; r < kBlk; ++r)
            if (r < rows) cp_async16(dst + r * kRow, src + size_t(r) * W * (2 * DP));
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(
                         smem_addr(&full[st])) : "memory");
      }
    }
    // every copy has landed before the CTA ends, also where a wait ran out above: each lane
    // waits for its own, then for the arrivals of the last fill of each stage (an earlier one
    // had landed before the chains freed its stage) with a limit of its own
    asm volatile("cp.async.wait_all;" ::: "memory");
    wt.dead = false;
    for (uint32_t f = n > kStages ? n - kStages : 0; f < n; ++f)
      if (int(f % 3) == warp - 12) wt.wait(&full[f % kStages], (f / kStages) & 1);
  } else {
    // ---- coefficients of the tiles after the first ------------------------------------
    int it = 1;
    for (int tile = blockIdx.x + gridDim.x; tile < total; tile += gridDim.x, ++it) {
      const int buf = it & 1;
      if (it >= 2) wt.wait(&cempty[buf], ((it - 2) >> 1) & 1);   // tile it - 2 is done
      load_coef(tile, buf, lane, 32);
      warp_arrive(&cfull[buf], lane);
    }
  }
  __syncthreads();
  if (warp == 0) tm_free(tmem, kTm);
}

int coef_stride(int H, int hh) { return (H - hh + kBlk - 1) / kBlk * kBlk + 4; }
size_t tm_smem(int G, int cstride) {
  const int ncol = G == 1 ? 4 : (G == 2 ? 2 : 1);
  return size_t(kStages + 2 * kOut) * kBlk * kRow * 4 + size_t(2) * ncol * cstride * 4;
}

template <int G, bool RK>
cudaError_t launch_g(const DevCfg& cfg, const Batch& b, int maxH, cudaStream_t s) {
  const int cstride = coef_stride(maxH, cfg.hh);
  const size_t sm = tm_smem(G, cstride);
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const cudaError_t e = allow_smem(k_cols_tm<G, RK>, sm);
  if (e != cudaSuccess) return e;
  k_cols_tm<G, RK><<<std::min(b.cols_prefix[b.n], nsm), kThreads, sm, s>>>(cfg, b, cstride);
  return cudaGetLastError();
}

}  // namespace

bool cols_tm_fits(int H, int Dpad, int hh) {
  return tm_smem(Dpad / 64, coef_stride(H, hh)) <= size_t(224) << 10;
}

// `b0`: pairs of one disparity group that all fit (cols_tm_fits).
cudaError_t launch_cols_tm(const DevCfg& cfg, const Batch& b0, cudaStream_t s) {
  thread_local Batch b;                               // tiles instead of columns
  b = b0;
  const int G = b.maxDpad / 64, ncol = G == 1 ? 4 : (G == 2 ? 2 : 1);
  int maxH = 0;
  b.cols_prefix[0] = 0;
  for (int i = 0; i < b.n; ++i) {
    const int cols = std::max(0, b.p[i].W - 2 * cfg.hw - cfg.dmin);
    b.cols_prefix[i + 1] = b.cols_prefix[i] + (cols + ncol - 1) / ncol;
    maxH = std::max(maxH, b.p[i].H);
  }
  if (b.cols_prefix[b.n] == 0) return cudaSuccess;
  auto go = [&](auto rk) -> cudaError_t {
    constexpr bool RK = decltype(rk)::value;
    switch (G) {
      case 1: return launch_g<1, RK>(cfg, b, maxH, s);
      case 2: return launch_g<2, RK>(cfg, b, maxH, s);
      case 3: return launch_g<3, RK>(cfg, b, maxH, s);
      default: return launch_g<4, RK>(cfg, b, maxH, s);
    }
  };
  // (a batch has reverse keys for all its pairs or for none)
  return b.p[0].rkey ? go(std::true_type()) : go(std::false_type());
}

}  // namespace de
