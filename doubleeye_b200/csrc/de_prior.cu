// The disparity prior as a per-plane mask: core/tools/de_dense.cpp:797-853 (mask),
// :438-483 (filter over a rectangle), :1166-1297 (score, filter and insert under the
// mask), driven by --prior (:1756-1813).
//
// A prior (a previous frame's disparity, a coarse pass) says where each disparity
// plane is worth computing: plane d is needed at the pixels whose band
// [round(prior) - band, round(prior) + band] contains d.  Per image row and plane this
// is an interval of x; per plane a bounding box.  The reference then scores and
// filters each needed plane only over its bounding box padded by 8 pixels (the
// recursive filter's chains start at the rectangle's edges, so values differ from the
// full-plane filter there) and inserts the plane into a pixel's top-2 only inside the
// row intervals.  Sub-pixel refinement is off under a prior (the tool turns it off).
//
// Layout here: the plane-minor volume [y][x][Dpad] of the dense path.  Rows: a CTA per
// image row with its census words in shared memory, a thread per pair of planes.
// Columns: a group of lanes per column, two, four or eight planes a lane, whose top-2 are
// merged over the group.  Each plane's rectangle enters as its own filter coefficient: 0
// at the rectangle's first pixel takes the input as it is, 2^15 outside carries the state
// through, both exactly, so all planes of a thread step together without branches.
//
// What bounds them: the serial chains at few warps an SM (one pair).  848x480 D=128, band
// 2 (us, rows / columns): 888 / 1072 with a thread per plane, its loads in the chain, a
// constant-memory score table and a compare-and-swap per insert; 200 / 247 now.
#include <algorithm>
#include <type_traits>

#include <cuda_runtime.h>

#include "de_dev.cuh"
#include "de_internal.h"

namespace de {
namespace {

constexpr int kMaskPad = 8;          // core/tools/de_dense.cpp:857 (MPAD)
constexpr int kHold = 1 << 15;       // the coefficient that leaves a state as it is

struct Rect { int ylo, yhi, xlo, xhi, pylo, pyhi; };

__device__ __forceinline__ bool plane_rect(const int* box, int D, int k, int W, int H, int hw,
                                           int hh, int d, Rect* r) {
  const int pylo = box[k], pyhi = box[D + k], pxlo = box[2 * D + k], pxhi = box[3 * D + k];
  if (pyhi < pylo) return false;                       // no pixel wants this plane
  r->ylo = max(hh, pylo - kMaskPad);
  r->yhi = min(H - hh, pyhi + 1 + kMaskPad);
  r->xlo = max(hw + d, pxlo - kMaskPad);
  r->xhi = min(W - hw, pxhi + 1 + kMaskPad);
  r->pylo = pylo;
  r->pyhi = pyhi;
  return r->yhi - r->ylo >= 1 && r->xhi - r->xlo >= 2;
}

__global__ void k_prior_init(int* box, int D, int W, int H) {
  for (int k = threadIdx.x; k < D; k += blockDim.x) {
    box[k] = H;
    box[D + k] = -1;
    box[2 * D + k] = W;
    box[3 * D + k] = -1;
  }
}

// One CTA per image row: the row's intervals in shared memory, then the planes'
// bounding boxes.  Pixels with a non-finite prior want no plane.  mx: per row and plane
// the interval, first | last << 16 (empty: W | -1), Dpad planes a row.
__global__ void k_prior_mask(const float* __restrict__ prior, int W, int H, int D, int Dpad,
                             int dmin, int dmax, int band, uint32_t* mx, int* box) {
  extern __shared__ int sm[];
  int* r0 = sm;
  int* r1 = sm + D;
  const int y = blockIdx.x;
  for (int k = threadIdx.x; k < D; k += blockDim.x) {
    r0[k] = W;
    r1[k] = -1;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < W; x += blockDim.x) {
    const float p = prior[size_t(y) * W + x];
    if (!isfinite(p)) continue;
    const int dc = int(lroundf(fminf(fmaxf(p, -1e6f), 1e6f)));
    const int klo = max(dmin, dc - band) - dmin;
    const int khi = min(dmax, dc + band) - dmin;
    for (int k = klo; k <= khi; ++k) {
      atomicMin(&r0[k], x);
      atomicMax(&r1[k], x);
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < Dpad; k += blockDim.x) {
    const int a = k < D ? r0[k] : W, b = k < D ? r1[k] : -1;
    mx[size_t(y) * Dpad + k] = pack2(a, b);
    if (b < a) continue;
    atomicMin(&box[k], y);
    atomicMax(&box[D + k], y);
    atomicMin(&box[2 * D + k], a);
    atomicMax(&box[3 * D + k], b);
  }
}

// A plane's extent along one direction as a filter coefficient rule.
struct Span {
  int lo = 1 << 28, n = 0;               // first position, positions after it
  __device__ __forceinline__ int last() const { return lo + n; }
  // forward step at p, with coefficient a inside
  __device__ __forceinline__ int down(int p, int a) const {
    return unsigned(p - lo - 1) < unsigned(n) ? a : (p == lo ? 0 : kHold);
  }
  // backward step at p (its coefficient is position p + 1's); the last position holds the
  // forward value
  __device__ __forceinline__ int up(int p, int a) const {
    return unsigned(p - lo) < unsigned(n) ? a : kHold;
  }
};

__device__ __forceinline__ int warp_min(int v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// Horizontal passes over each needed plane's rectangle: CTA = row, thread = two planes.
// The forward results go to the volume and come back eight words ahead.
template <int TS>
__global__ void __launch_bounds__(128) k_prior_rows(DevCfg cfg, DevPair P,
                                                    const int* __restrict__ box, int apart) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int D = P.D, W = P.W, H = P.H, XS = P.Dpad / 2;
  const int y = blockIdx.x, tid = threadIdx.x;
  Span s0, s1;
  for (int j = 0; j < 2; ++j) {
    const int k = 2 * tid + j;
    Rect r;
    if (k >= D || !plane_rect(box, D, k, W, H, cfg.hw, cfg.hh, cfg.dmin + k, &r) || y < r.ylo ||
        y >= r.yhi)
      continue;
    Span& sp = j ? s1 : s0;
    sp.lo = r.xlo;
    sp.n = r.xhi - r.xlo - 1;
  }
  const int lo = min(s0.lo, s1.lo), hi = max(s0.n ? s0.last() : -1, s1.n ? s1.last() : -1);
  if (!__syncthreads_or(hi >= 0)) return;
  uint64_t* sL = reinterpret_cast<uint64_t*>(smem);
  uint64_t* sR = sL + W;
  uint8_t* tab = reinterpret_cast<uint8_t*>(sR + W);
  uint16_t* sax = reinterpret_cast<uint16_t*>(tab + ScoreTable<TS, 1>::bytes());
  for (int x = tid; x < W; x += blockDim.x) {
    sL[x] = P.cwL[size_t(y) * P.cpitch + P.lpad + x];
    sR[x] = P.cwR[size_t(y) * P.cpitch + x];
    sax[x] = P.ax[size_t(y) * P.apitch + P.lpad + x];
  }
  fill_scores<TS>(cfg, tab);
  __syncthreads();
  const int xs = warp_min(lo), xe = warp_max(hi);       // the warp's planes
  if (xe < 0) return;
  // inside every needed plane's rectangle the coefficient is the image's (what the other
  // planes hold is not looked at)
  const int xi = warp_max(max(s0.n ? s0.lo : -1, s1.n ? s1.lo : -1));
  const int xj = warp_min(min(s0.n ? s0.last() : 1 << 28, s1.n ? s1.last() : 1 << 28));
  const int d0 = cfg.dmin + 2 * tid;
  uint32_t* out = reinterpret_cast<uint32_t*>(P.vol) + size_t(y) * W * XS + tid;
  // The lanes step over x together, so that a step's words are adjacent, or each from its own
  // first position, where the planes' rectangles are short and far apart (a prior that
  // slants across the image): `apart` times fewer steps at least.
  const int own = warp_max(hi >= 0 ? hi - lo : 0);
  auto passes = [&](auto by_lane) {
    constexpr bool APART = decltype(by_lane)::value;
    const int x0 = APART ? (hi >= 0 ? lo : xs) : xs, n = APART ? own : xe - xs;
    auto at = [&](int x) { return APART ? min(x, W - 1) : x; };   // (past a lane's last)
    int32_t f0 = kVolBias, f1 = kVolBias;
    // (a lane before its own rectangle reads a clamped right word that nothing looks at)
    uint64_t rprev = sR[max(x0 - 1 - d0, 0)];
#pragma unroll 4
    for (int t = 0; t <= n; ++t) {
      const int x = x0 + t, xc = at(x);
      const uint64_t lw = sL[xc], rw = sR[max(xc - d0, 0)];
      const int a = sax[xc];
      const int32_t c0 = graded<true, TS, 1>(lw, rw, tab, nullptr, nullptr, 0, 0);
      const int32_t c1 = graded<true, TS, 1>(lw, rprev, tab, nullptr, nullptr, 0, 0);
      rprev = rw;
      int a0 = a, a1 = a;
      if (APART || x <= xi || x > xj) { a0 = s0.down(x, a); a1 = s1.down(x, a); }
      f0 = rf_step(c0, f0, a0);
      f1 = rf_step(c1, f1, a1);
      if (x >= lo && x <= hi) out[size_t(x) * XS] = pack2(f0, f1);
    }
    // backward, eight words ahead
    constexpr int PF = 8;
    uint32_t cur[PF], nxt[PF];
    auto fetch = [&](int t, uint32_t (&w)[PF]) {
#pragma unroll
      for (int i = 0; i < PF; ++i) w[i] = __ldcg(out + size_t(at(x0 + max(t - i, 0))) * XS);
    };
    fetch(n - 1, cur);
    for (int t = n - 1; t >= 0; t -= PF) {
      fetch(t - PF, nxt);
#pragma unroll
      for (int i = 0; i < PF; ++i) {
        if (t < i) break;
        const int p = x0 + t - i, a = sax[at(p + 1)];
        int a0 = a, a1 = a;
        if (APART || p < xi || p >= xj) { a0 = s0.up(p, a); a1 = s1.up(p, a); }
        f0 = rf_step(int32_t(cur[i] & 0xFFFFu), f0, a0);
        f1 = rf_step(int32_t(cur[i] >> 16), f1, a1);
        if (p >= lo && p <= hi) out[size_t(p) * XS] = pack2(f0, f1);
      }
#pragma unroll
      for (int i = 0; i < PF; ++i) cur[i] = nxt[i];
    }
  };
  if (apart * own < xe - xs) passes(std::true_type());
  else passes(std::false_type());
}

// One column's vertical passes and masked top-2 by TPC lanes, each with planes k0 to k0 + KT.
template <int KT, int TPC>
__device__ __forceinline__ void prior_column(const DevCfg& cfg, const DevPair& P,
                                             const int* __restrict__ box,
                                             const uint32_t* __restrict__ mx, int x, int sub,
                                             int k0) {
  constexpr int KW = KT / 2, PF = KT <= 4 ? 8 : 4;     // words a lane and row, rows ahead
  constexpr int MW = KT < 4 ? KT : 4;                  // interval words a load
  const int D = P.D, W = P.W, H = P.H, Dpad = P.Dpad;
  Span sp[KT];
  uint32_t on = 0;                       // planes needed in this column
  int lo = 1 << 28, hi = -1, in_lo = -1, in_hi = 1 << 28;
#pragma unroll
  for (int i = 0; i < KT; ++i) {
    Rect r;
    if (k0 + i >= D || !plane_rect(box, D, k0 + i, W, H, cfg.hw, cfg.hh, cfg.dmin + k0 + i, &r) ||
        x < r.xlo || x >= r.xhi)
      continue;
    sp[i].lo = r.ylo;
    sp[i].n = r.yhi - r.ylo - 1;
    lo = min(lo, r.ylo);
    hi = max(hi, r.yhi - 1);
    on |= 1u << i;
    in_lo = max(in_lo, r.ylo);
    in_hi = min(in_hi, r.yhi - 1);
  }
  const int ys = warp_min(lo), ye = warp_max(hi);       // the warp's planes
  if (ye < 0) return;
  const int yi = warp_max(in_lo), yj = warp_min(in_hi);   // inside all of them between
  const int xc = min(x, W - 1), kc = min(k0, Dpad - KT);   // any address for idle lanes
  const size_t st = size_t(W) * Dpad / 2;
  uint32_t* col = reinterpret_cast<uint32_t*>(P.vol) + (size_t(xc) * Dpad + kc) / 2;
  const uint16_t* ay = P.ay + xc;
  int32_t f[KT];
#pragma unroll
  for (int i = 0; i < KT; ++i) f[i] = kVolBias;
  auto load = [&](int y, uint32_t (&w)[KW]) {
    const uint32_t* g = col + size_t(y) * st;
    if constexpr (KW == 1) {
      w[0] = __ldcg(g);
    } else if constexpr (KW == 2) {
      const uint2 v = __ldcg(reinterpret_cast<const uint2*>(g));
      w[0] = v.x; w[1] = v.y;
    } else {
      const uint4 v = __ldcg(reinterpret_cast<const uint4*>(g));
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
  };
  uint32_t ring[PF][KW];
  int ring_a[PF];
#pragma unroll
  for (int j = 0; j < PF; ++j) {
    load(min(ys + j, ye), ring[j]);
    ring_a[j] = ay[size_t(min(ys + j, ye)) * W];
  }
  for (int y0 = ys; y0 <= ye; y0 += PF) {
#pragma unroll
    for (int j = 0; j < PF; ++j) {
      const int y = y0 + j;
      uint32_t c[KW];
#pragma unroll
      for (int i = 0; i < KW; ++i) c[i] = ring[j][i];
      const int a = ring_a[j];
      load(min(y + PF, ye), ring[j]);
      ring_a[j] = ay[size_t(min(y + PF, ye)) * W];
      if (y > ye) continue;
      int co[KT];
#pragma unroll
      for (int i = 0; i < KT; ++i) co[i] = a;
      if (y <= yi || y > yj) {
#pragma unroll
        for (int i = 0; i < KT; ++i) co[i] = sp[i].down(y, a);
      }
#pragma unroll
      for (int i = 0; i < KT; ++i)
        f[i] = rf_step(int32_t(i & 1 ? c[i / 2] >> 16 : c[i / 2] & 0xFFFFu), f[i], co[i]);
      if (y >= lo && y <= hi) {
        uint32_t* g = col + size_t(y) * st;
        if constexpr (KW == 1)
          *g = pack2(f[0], f[1]);
        else if constexpr (KW == 2)
          *reinterpret_cast<uint2*>(g) = make_uint2(pack2(f[0], f[1]), pack2(f[2], f[3]));
        else
          *reinterpret_cast<uint4*>(g) = make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]),
                                                    pack2(f[4], f[5]), pack2(f[6], f[7]));
      }
    }
  }
  // backward and the insert; a row's intervals come with its words
  uint32_t ring_m[PF][KT];
  auto load_m = [&](int y, uint32_t (&m)[KT]) {
    const uint32_t* g = mx + size_t(y) * Dpad + kc;
#pragma unroll
    for (int i = 0; i < KT; i += MW) {
      if constexpr (MW == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(g + i);
        m[i] = v.x; m[i + 1] = v.y;
      } else {
        const uint4 v = *reinterpret_cast<const uint4*>(g + i);
        m[i] = v.x; m[i + 1] = v.y; m[i + 2] = v.z; m[i + 3] = v.w;
      }
    }
  };
#pragma unroll
  for (int j = 0; j < PF; ++j) {
    const int y = max(ye - j, ys);
    load(y, ring[j]);
    load_m(y, ring_m[j]);
    ring_a[j] = ay[size_t(min(y + 1, H - 1)) * W];
  }
  for (int y0 = ye; y0 >= ys; y0 -= PF) {
#pragma unroll
    for (int j = 0; j < PF; ++j) {
      const int y = y0 - j;
      uint32_t c[KW];
      uint32_t m[KT];
#pragma unroll
      for (int i = 0; i < KW; ++i) c[i] = ring[j][i];
#pragma unroll
      for (int i = 0; i < KT; ++i) m[i] = ring_m[j][i];
      const int a = ring_a[j], yn = max(y - PF, ys);
      load(yn, ring[j]);
      load_m(yn, ring_m[j]);
      ring_a[j] = ay[size_t(min(yn + 1, H - 1)) * W];
      if (y < ys) continue;
      int co[KT];
#pragma unroll
      for (int i = 0; i < KT; ++i) co[i] = a;
      if (y < yi || y >= yj) {
#pragma unroll
        for (int i = 0; i < KT; ++i) co[i] = sp[i].up(y, a);
      }
      uint32_t p0 = 0, p1 = 0;
#pragma unroll
      for (int i = 0; i < KT; ++i) {
        f[i] = rf_step(int32_t(i & 1 ? c[i / 2] >> 16 : c[i / 2] & 0xFFFFu), f[i], co[i]);
        const uint32_t w = m[i];
        // (a needed plane's rows with an interval lie in its rectangle)
        const bool in = on >> i & 1 && x >= int(int16_t(w & 0xFFFFu)) &&
                        x <= (int32_t(w) >> 16);
        const uint32_t key = in ? (uint32_t(f[i]) << 8) | uint32_t(255 - k0 - i) : 0u;
        const uint32_t l = min(p0, key);
        p0 = max(p0, key);
        p1 = max(p1, l);
        if (P.rkey && in) atomicMax(P.rkey + size_t(y) * W + x - cfg.dmin - k0 - i, key);
      }
      if (!__any_sync(0xffffffffu, p0 != 0)) continue;
#pragma unroll
      for (int o = 1; o < TPC; o <<= 1) {
        const uint32_t o0 = __shfl_xor_sync(0xffffffffu, p0, o), o1 = __shfl_xor_sync(0xffffffffu, p1, o);
        const uint32_t l = min(p0, o0);
        p0 = max(p0, o0);
        p1 = max(max(p1, o1), l);
      }
      if (sub == 0 && p0) {
        P.key0[size_t(y) * W + x] = p0;
        P.key1[size_t(y) * W + x] = p1;
      }
    }
  }
}

// Vertical passes and the masked top-2: TPC lanes a column, KT planes a lane: four planes
// up to Dpad 128 (a warp per column: the most warps for one pair), else eight.  A warp whose
// column's needed planes lie within 64 of each other (a slanted or smooth prior) takes two a
// lane there (3000x200 D=256, slanted prior, band 0: the call 508 us without, 356 with).
template <int KT, int TPC>
__global__ void __launch_bounds__(128) k_prior_cols(DevCfg cfg, DevPair P,
                                                    const int* __restrict__ box,
                                                    const uint32_t* __restrict__ mx) {
  const int sub = threadIdx.x % TPC, k0 = sub * KT;
  const int x = cfg.hw + cfg.dmin + blockIdx.x * (128 / TPC) + threadIdx.x / TPC;
  if constexpr (TPC == 32) {
    int first = 1 << 28, last = -1;
#pragma unroll
    for (int i = 0; i < KT; ++i) {
      const int k = k0 + i;
      Rect r;
      if (k >= P.D || !plane_rect(box, P.D, k, P.W, P.H, cfg.hw, cfg.hh, cfg.dmin + k, &r) ||
          x < r.xlo || x >= r.xhi)
        continue;
      first = min(first, k);
      last = k;
    }
    first = warp_min(first) & ~1;
    last = warp_max(last);
    if (last < 0) return;
    if (last - first < 2 * TPC) {
      prior_column<2, TPC>(cfg, P, box, mx, x, sub, first + 2 * sub);
      return;
    }
  }
  prior_column<KT, TPC>(cfg, P, box, mx, x, sub, k0);
}

}  // namespace

size_t prior_ws_bytes(int W, int H, int D) {
  auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
  return up(size_t(H) * ((D + 63) & ~63) * 4) + up(size_t(D) * 16);
}

cudaError_t launch_prior(const DevCfg& cfg, const Batch& b, const float* prior, int band,
                         void* ws, cudaStream_t s) {
  const DevPair& P = b.p[0];
  const int W = P.W, H = P.H, D = P.D, Dpad = P.Dpad;
  auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
  uint32_t* mx = static_cast<uint32_t*>(ws);
  int* box = reinterpret_cast<int*>(static_cast<uint8_t*>(ws) + up(size_t(H) * Dpad * 4));
  // no candidate where no plane is inserted; sub-pixel neighbours are never looked at
  cudaError_t e = cudaMemsetAsync(P.key0, 0, size_t(W) * H * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(P.key1, 0, size_t(W) * H * 4, s);
  if (e != cudaSuccess) return e;
  k_prior_init<<<1, 256, 0, s>>>(box, D, W, H);
  k_prior_mask<<<H, 256, size_t(2) * D * sizeof(int), s>>>(prior, W, H, D, Dpad, cfg.dmin,
                                                           cfg.dmin + D - 1, band, mx, box);
  // Lanes that step apart write 32 sectors a step instead of four: no loss while the rows'
  // chains are what bounds, so with few warps an SM, else only for so many fewer steps.
  // Measured (one pair, slanted prior, us; together / apart): 60 warps at 3.5 times fewer
  // steps 969 / 497; 400 at 4.1 times 338 / 264; 800 at 4.2 times 711 / 792, at 20 times
  // 606 / 508; 2160 at 13 times 1707 / 1768, at 21 times 1682 / 1555; 4000 at 14 times
  // 1222 / 1339.
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int apart = std::max(2, 2 * H * (Dpad / 64) / nsm);
  auto rows = [&](auto kern, size_t table) -> cudaError_t {
    const size_t sm = size_t(W) * 18 + table;
    const cudaError_t e2 = allow_smem(kern, sm);
    if (e2 != cudaSuccess) return e2;
    kern<<<H, Dpad / 2, sm, s>>>(cfg, P, box, apart);
    return cudaGetLastError();
  };
  e = cfg.trunc < 16 ? rows(k_prior_rows<16>, ScoreTable<16, 1>::bytes())
                     : rows(k_prior_rows<256>, ScoreTable<256, 1>::bytes());
  const int ncols = W - 2 * cfg.hw - cfg.dmin;
  if (e != cudaSuccess || ncols <= 0) return e;
  auto grid = [&](int tpc) { return (ncols + 128 / tpc - 1) / (128 / tpc); };
  if (Dpad == 64) k_prior_cols<4, 16><<<grid(16), 128, 0, s>>>(cfg, P, box, mx);
  else if (Dpad == 128) k_prior_cols<4, 32><<<grid(32), 128, 0, s>>>(cfg, P, box, mx);
  else k_prior_cols<8, 32><<<grid(32), 128, 0, s>>>(cfg, P, box, mx);
  return cudaGetLastError();
}

}  // namespace de
