// Sparse products on the device.
//
// CRS (crs_matrix_spmv_impl, crs_matrix.hpp:1505-1516): persistent kernels
// walk the matrix in row order as warp work items of at most 512 nonzeros,
// packed once per matrix on the device from the row offsets.  An item is
// either a tile of consecutive short rows (up to 248 rows; for k_crs a bounded
// number of products per lane) or a piece of a long row (k_finalize adds the
// pieces in order).  FP32 arithmetic (k_crs): a warp streams the item's values
// and column ids with coalesced evict-first loads, gathers x through the
// read-only path, stages the products in its own shared-memory slice and sums
// each row with 1..32 lanes.  FP64 arithmetic (k_crs64): the rows are cut
// among the lanes by entries, so that every FP64 instruction serves 32 lanes.
// All reductions have a fixed order, so results are deterministic run to run.
//
// The optional logistic epilogue is compute_wtx + logistic_gradient::
// compute_dloss + `* sample_weight` + bias sum (gradient_descent.hpp:196-211,
// gradient.hpp:15-53): dloss*sw per row and per-CTA compensated partial sums of
// the loss and of dloss*sw.  FP32 arithmetic: fused into k_crs (FP32 Kahan sums,
// which keep GB300's narrow FP64 unit out of the per-row work), the partials
// reduced in FP64 by k_finalize.  FP64 arithmetic: a kernel of its own over the
// finished product (k_logreg_rows).
#include <algorithm>
#include <mutex>
#include <vector>

#include "device_common.cuh"

namespace fvg {

// ------------------------------------------------------------ kernel args
struct CrsK {
  const i32* off;
  const i32* idx;
  const void* val;
  const void* x;
  const Item* items;
  i64 nitems;
  void* y;
  void* partials;
  // logistic epilogue
  const double* label;
  const double* sw;
  const float* label_f;
  const float* sw_f;
  const double* intercept;
  int icpt;
  void* r;
  double* cta_part;
  int loss;    // GLM loss kind
  double eps;  // its epsilon
  const float* ybase;  // FP32 path: per-row partial sums from another pass, added before the epilogue
};

template <class AT, class YT, int EPI, class S>
__device__ __forceinline__ void epilogue(const CrsK& p, i32 row, AT acc, AT b, S& ls, S& bs) {
  if (EPI == EPI_STORE) {
    ((YT*)p.y)[row] = (YT)acc;
  } else {
    AT wtx = acc + b;
    if constexpr (sizeof(AT) == 4)
      if (p.ybase) wtx += p.ybase[row];
    AT loss, d;
    if constexpr (sizeof(AT) == 8) {
      glm_row<AT>(p.loss, (AT)p.eps, wtx, p.label[row], loss, d);
      if (p.sw) d = d * p.sw[row];
    } else {
      glm_row<AT>(p.loss, (AT)p.eps, wtx, p.label_f[row], loss, d);
      if (p.sw_f) d = d * p.sw_f[row];
    }
    ((YT*)p.r)[row] = (YT)d;
    ls.add(loss);
    if (p.icpt) bs.add(d);  // without an intercept the bias sum is reported as 0
  }
}

// ------------------------------------------------------------ warp tiles

// Persistent CRS kernel of the FP32-arithmetic paths.  Warp g of the grid
// handles items g, g+W, g+2W, ... (W = warps in the grid).  Phase 1: the warp
// streams the item's nonzeros with coalesced loads (lane L: nonzeros L, L+32,
// ...; a group of rounds issued before any use), gathers x and writes the
// products to its own shared-memory slice.  Phase 2: rows of a tile are
// summed from shared memory by 1..32 lanes each (32 / rows, rounded to a
// power of two), the lanes of a row combined by shuffles; a piece is summed
// by the whole warp.  No CTA-wide barrier inside the loop.
template <class VT, class XT, class AT, class YT, int EPI>
__global__ void __launch_bounds__(kThreads, FVG_CRS_MIN_BLOCKS) k_crs(const CrsK p) {
  static_assert(sizeof(AT) == 4, "FP64 sums: k_crs64");
  constexpr int SPAN = kWarpTile;        // products slice per warp
  constexpr int NR = SPAN / 32;          // element rounds per lane
  constexpr int RG = FVG_CRS_ROUNDS;     // rounds in flight together
  __shared__ AT sprod[kThreads / 32][SPAN];
  __shared__ int soffs[kThreads / 32][kTileRows + 1];
  using Sum = typename SumOf<AT>::type;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  AT* prod = sprod[w];
  int* soff = soffs[w];
  const i64 W = (i64)gridDim.x * (kThreads / 32);
  const i64 n = p.nitems;
  const XT* __restrict__ x = (const XT*)p.x;
  const VT* __restrict__ val = (const VT*)p.val;
  Sum ls, bs;
  const AT bias = (EPI == EPI_LOGREG && p.icpt) ? (AT)*p.intercept : (AT)0;
  i64 t = (i64)blockIdx.x * (kThreads / 32) + w;
  Item nx = (t < n) ? p.items[t] : Item{0, 0, 0, 0};
  for (; t < n; t += W) {
    const Item it = nx;
    if (t + W < n) nx = p.items[t + W];  // prefetch the next descriptor
    const int a0 = it.e0;
    const int span = it.e1 - a0;
    // row boundaries of a tile into the warp's offsets slice
    if (it.r1 >= 0)
      for (int k = lane; k <= it.r1 - it.r0; k += 32) soff[k] = __ldg(p.off + it.r0 + k);
    // phase 1: lane L takes nonzeros L, L+32, ... so one gather instruction
    // covers 32 consecutive nonzeros (neighbouring columns / rows share
    // sectors); RG rounds of loads are issued before their gathers.
#pragma unroll
    for (int g = 0; g < NR; g += RG) {
      int c[RG];
      AT v[RG];
#pragma unroll
      for (int q = 0; q < RG; q++) {
        const int k = (g + q) * 32 + lane;
        if (g + q < NR && k < span) {
          c[q] = __ldcs(p.idx + a0 + k);
          v[q] = ld_val<VT, AT>(val + a0 + k);
        }
      }
#pragma unroll
      for (int q = 0; q < RG; q++) {
        const int k = (g + q) * 32 + lane;
        if (g + q < NR && k < span) prod[k] = v[q] * (AT)__ldg(x + c[q]);
      }
    }
    __syncwarp();
    // phase 2
    if (it.r1 >= 0) {
      // Gl lanes per row: 32 / R rounded to a power of two; tiles of 32 or
      // more (short) rows take rounds of 32 rows, one lane each
      const int R = it.r1 - it.r0;
      const int Gl = lanes_per_row(R);  // the packer keeps a lane's share <= kLaneWork
      const int per_round = 32 / Gl;
      for (int rb = 0; rb < R; rb += per_round) {
        const int j = rb + lane / Gl, sub = lane % Gl;
        AT acc = 0;
        if (j < R) {
          const int s = soff[j] - a0, e = soff[j + 1] - a0;
          int k = s + sub;
          AT a1 = 0, a2 = 0, a3 = 0;
          for (; k + 3 * Gl < e; k += 4 * Gl) {
            acc += prod[k];
            a1 += prod[k + Gl];
            a2 += prod[k + 2 * Gl];
            a3 += prod[k + 3 * Gl];
          }
          for (; k < e; k += Gl) acc += prod[k];
          acc = (acc + a1) + (a2 + a3);
        }
        for (int o = Gl >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (j < R && sub == 0) epilogue<AT, YT, EPI>(p, it.r0 + j, acc, bias, ls, bs);
      }
    } else {
      AT acc = 0;
      for (int k = it.e0 - a0 + lane; k < span; k += 32) acc += prod[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) ((AT*)p.partials)[-1 - it.r1] = acc;
    }
    __syncwarp();
  }
  if (EPI == EPI_LOGREG) block_csum2(ls.total(), bs.total(), &p.cta_part[2 * blockIdx.x], &p.cta_part[2 * blockIdx.x + 1]);
}

// ---------------------------------------------------------- FP64 products
// The FP64 product.  A warp-wide FP64 instruction holds its scheduler's FP64
// unit for 64 clocks whether 2 or 32 of its lanes are used (an SM of four
// schedulers runs about two FP64 operations a clock), while some 60 other
// instructions issue beside it: the row sums must keep every lane's FP64 slot
// busy and may spend integer work freely.
// Phase 1 (as k_crs): lane L streams nonzeros L, L+32, ... with coalesced
// loads (one gather instruction covers 32 consecutive nonzeros) and puts the
// gathered x and the value into the warp's shared slices.  Phase 2: lane L
// owns ch = ceil(nonzeros / 32) consecutive nonzeros (16 of a full item) and
// adds them with one fused multiply-add each, starting anew at the rows'
// first entries, which sit as bits in a 512-bit map; the sum up to each row
// start is parked in the slot of that start.  The segments open at the
// chunks' ends are joined in lane order by a segmented scan that stops once
// every lane has met a row start (rows of 60 entries: 3 of its 5 steps), and
// added to the sum parked at the next chunk's first mark.  Phase 3, a lane
// per row: the row's sum is the one parked at its end.  An item costs 16 +
// about 4 FP64 instructions for 512 nonzeros; lanes_per_row() lanes a row
// cost 30 to 60 on rows of uneven length and re-read the values lane by lane
// from L1.  A long row's piece is added in registers by the whole warp.  The
// next item's ids are loaded before this item's sums.
// The gathers miss L1 one by one (an SM takes about one such sector a clock:
// 2M x 2M with uniform columns cannot go below 0.27 ms), and each needs an L1
// line while it is under way, so shared memory is kept to 3 CTAs of 4 warps:
// 24 warps (222 KB of slices) took 1.21 ms where 12 (111 KB) take 0.44.
// Measured (before: k_crs's rows by lanes, and its loss rows): 2M x 2M
// power-law 558 -> 442 us; 1M x 100,000, 6.0e7 nonzeros, A w with hinge loss
// 372 -> 221 + 42, A^T r 238 -> 221; 100,000 x 20,000, 4.0e6 nonzeros, A w
// with logistic loss 81 -> 18 + 20, A^T r 22.6 -> 18.3.  At 6.0e7 nonzeros L1's
// data pipe is 74% and the FP64 pipe 59% busy.
static_assert(kWarpTile == 512, "k_crs64: 16 entries a lane, a 16-word row map");
constexpr int kC64 = 16;                               // entries per lane
constexpr int kC64Pad = kWarpTile + kWarpTile / kC64;  // doubles per slice
constexpr int kC64SoffB = ((kTileRows + 1) * 2 + 15) / 16 * 16;
constexpr int kC64Map = kWarpTile / 32 + 4;  // words of the row map (and padding)
constexpr int kC64WarpB = 2 * kC64Pad * 8 + 4 * kC64Map + kC64SoffB;  // x, values, row map, row offsets
static_assert(kC64WarpB % 16 == 0, "slices stay 16-byte aligned");
#ifndef FVG_CRS64_WARPS
#define FVG_CRS64_WARPS 4
#endif
#ifndef FVG_CRS64_BLOCKS
#define FVG_CRS64_BLOCKS 3
#endif
#ifndef FVG_CRS64_RG
#define FVG_CRS64_RG 16
#endif
constexpr int kC64Threads = 32 * FVG_CRS64_WARPS;
constexpr int kC64Blocks = FVG_CRS64_BLOCKS;  // resident CTAs per SM
constexpr int kC64Smem = kC64WarpB * FVG_CRS64_WARPS;

struct Crs64K {
  const i32* off;
  const i32* idx;
  const double* val;
  const double* x;
  const Item* items;
  i64 nitems;
  double* y;
  double* partials;
};

__global__ void __launch_bounds__(kC64Threads, kC64Blocks) k_crs64(const Crs64K p) {
  constexpr int NR = kWarpTile / 32, RG = FVG_CRS64_RG;
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem64[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* xs = reinterpret_cast<double*>(smem64 + w * kC64WarpB);
  double* vs = xs + kC64Pad;
  unsigned* map = reinterpret_cast<unsigned*>(vs + kC64Pad);
  unsigned short* soff = reinterpret_cast<unsigned short*>(map + kC64Map);
  const i64 W = (i64)gridDim.x * (FVG_CRS64_WARPS), n = p.nitems;
  const double* __restrict__ x = p.x;
  const double* __restrict__ val = p.val;
  // consecutive items go to different CTAs: small matrices spread over the SMs
  i64 t = (i64)w * gridDim.x + blockIdx.x;
  if (t >= n) return;
  Item it = p.items[t], nx = (t + W < n) ? p.items[t + W] : Item{0, 0, 0, 0};
  int c[NR];  // this item's column ids
  auto fetch = [&](const Item& q) {
    const int span = q.e1 - q.e0;
#pragma unroll
    for (int r = 0; r < NR; r++) {
      const int k = r * 32 + lane;
      c[r] = (k < span) ? __ldcs(p.idx + q.e0 + k) : 0;
    }
  };
  fetch(it);
  for (; t < n; t += W) {
    const int a0 = it.e0, span = it.e1 - a0;
    const Item cur = it;
    it = nx;
    if (t + 2 * W < n) nx = p.items[t + 2 * W];
    if (cur.r1 < 0) {  // piece of a long row
      double s = 0.0;  // (one warp a scheduler keeps its FP64 unit busy: no second chain)
#pragma unroll
      for (int g = 0; g < NR; g += RG) {
        double xv[RG], vv[RG];
#pragma unroll
        for (int q = 0; q < RG; q++) {
          const int k = (g + q) * 32 + lane;
          xv[q] = (k < span) ? __ldg(x + c[g + q]) : 0.0;
          vv[q] = (k < span) ? __ldcs(val + a0 + k) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < RG; q++) s = fma(vv[q], xv[q], s);
      }
      if (t + W < n) fetch(it);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
      if (lane == 0) p.partials[-1 - cur.r1] = s;
      continue;
    }
    const int R = cur.r1 - cur.r0;
    // ch entries a lane; chunks start at odd multiples of 8 bytes, so that 32
    // lanes reading their chunks' k-th entries meet no bank conflict
    const int ch = max((span + 31) >> 5, 1), cap = 32 * ch;
    const unsigned rcp = (ch & 1) ? 0u : (65536u + ch - 1) / ch;  // k / ch = k * rcp >> 16 for k < 1024
    auto pos = [&](int k) { return k + (int)((unsigned)k * rcp >> 16); };
#pragma unroll
    for (int g = 0; g < NR; g += RG) {
      double xv[RG], vv[RG];
#pragma unroll
      for (int q = 0; q < RG; q++) {
        const int k = (g + q) * 32 + lane;
        xv[q] = (k < span) ? __ldg(x + c[g + q]) : 0.0;
        vv[q] = (k < span) ? __ldcs(val + a0 + k) : 0.0;
      }
      if (g == 0) {
        if (lane < kC64Map) map[lane] = 0u;
        for (int k = lane; k <= R; k += 32) soff[k] = (unsigned short)(__ldg(p.off + cur.r0 + k) - a0);
        __syncwarp();
        for (int j = lane; j < R; j += 32) {
          const int s = soff[j];
          if (soff[j + 1] > s) atomicOr(map + (s >> 5), 1u << (s & 31));
        }
      }
#pragma unroll
      for (int q = 0; q < RG; q++) {
        const int k = (g + q) * 32 + lane;
        if (k < cap) {
          xs[pos(k)] = xv[q];
          vs[pos(k)] = vv[q];
        }
      }
    }
    if (t + W < n) fetch(it);
    __syncwarp();
    const int first = lane * ch;  // the lane's first entry; a 17th word pads the map
    const unsigned marks = __funnelshift_r(map[first >> 5], map[(first >> 5) + 1], first & 31) & ((1u << ch) - 1u);
    double* xc = xs + pos(first);
    double S = 0.0;
    {
      const double* vc = vs + pos(first);
#pragma unroll
      for (int k = 0; k < kC64; k++) {
        if (k >= ch) break;
        const bool mk = (marks >> k) & 1u;
        const double xk = xc[k], vk = vc[k];
        if (mk) xc[k] = S;
        S = mk ? 0.0 : S;
        S = fma(vk, xk, S);
      }
    }
    bool f = marks != 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      if (!__any_sync(kFull, !f)) break;
      const double u = __shfl_up_sync(kFull, S, o);
      const bool fu = __shfl_up_sync(kFull, (int)f, o) != 0;
      if (lane >= o) {
        S = f ? S : u + S;
        f = f || fu;
      }
    }
    // the row open at this lane's start ends at its first mark
    const double carry = __shfl_up_sync(kFull, S, 1), last = __shfl_sync(kFull, S, 31);
    if (lane > 0 && marks) xc[__ffs(marks) - 1] += carry;
    __syncwarp();
    for (int j = lane; j < R; j += 32) {
      const int s = soff[j], e = soff[j + 1];
      // the last row ends with the item: the scan's last value
      p.y[cur.r0 + j] = e == s ? 0.0 : (e == span ? last : xs[pos(e)]);
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------- finalize
struct FinK {
  const i32* long_rows;
  const i32* long_piece0;
  i64 nlong;
  int per_warp;  // rows a warp takes at a time: 4 or 1
  const void* partials;
  void* y;
  // logistic
  const float* label_f;
  const float* sw_f;
  const double* intercept;
  int icpt;
  void* r;
  const double* cta_part;
  i64 ncta;
  double* long_part;
  double* out;        // [loss, bias]
  double* grad_bias;  // optional
  unsigned* ticket;
  int loss;
  double eps;
  const float* ybase;
};

// The last CTA's reduction of every loss / bias partial, in a fixed order,
// by the whole CTA: out[0] = loss, out[1] = bias (0 without an intercept).
__device__ __forceinline__ void reduce_loss(const double* cta_part, i64 ncta, const double* long_part, i64 nlong,
                                            int icpt, double* out, double* grad_bias, unsigned* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  CSum ls, bs;
  for (i64 i = threadIdx.x; i < ncta; i += kThreads) {
    ls.add(__ldcg(&cta_part[2 * i]));
    bs.add(__ldcg(&cta_part[2 * i + 1]));
  }
  for (i64 i = threadIdx.x; i < nlong; i += kThreads) {
    ls.add(__ldcg(&long_part[2 * i]));
    bs.add(__ldcg(&long_part[2 * i + 1]));
  }
  double tl = 0, tb = 0;
  block_csum2(ls.total(), bs.total(), &tl, &tb);
  if (threadIdx.x == 0) {
    out[0] = tl;
    out[1] = icpt ? tb : 0.0;
    if (grad_bias) *grad_bias = icpt ? tb : 0.0;
    *ticket = 0u;
  }
}

// Long rows: sum the pieces' partials in a fixed order and apply the
// epilogue; then (logistic, FP32 sums) the last CTA reduces every partial
// loss / bias in a fixed order.  A warp takes f.per_warp rows: 4 of 8 lanes
// each (lane s adds pieces s, s+8, ..., then a tree), or 1.  The kernel is
// bound by the latency of one row's chain of loads and adds, so where there
// are more rows than warps four share it (2M x 2M power-law rows, mostly
// under 40 pieces: 32 -> 6 us); a row of more than kFinShort pieces then takes
// the whole warp in turn.
constexpr i64 kFinShort = 32;
template <class AT, class YT, int EPI>
__global__ void __launch_bounds__(kThreads) k_finalize(const FinK f) {
  static_assert(EPI == EPI_STORE || sizeof(AT) == 4, "the FP64 loss rows run in k_logreg_rows");
  const AT b = (EPI == EPI_LOGREG && f.icpt) ? (AT)*f.intercept : (AT)0;
  const int lane = threadIdx.x & 31;
  const int G = 32 / f.per_warp, sub = lane & (G - 1);
  const AT* part = (const AT*)f.partials;
  // a warp's rows lie `rows` apart: the longest rows of a matrix with sorted
  // columns are neighbours, and land in different warps
  const i64 rows = (f.nlong + f.per_warp - 1) / f.per_warp;
  for (i64 b0 = (i64)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); b0 < rows;
       b0 += (i64)gridDim.x * (kThreads / 32)) {
    const i64 i = b0 + (lane / G) * rows;
    const bool valid = i < f.nlong;
    const i32 c0 = valid ? f.long_piece0[i] : 0, c1 = valid ? f.long_piece0[i + 1] : 0;
    const i32 row = valid ? f.long_rows[i] : 0;
    const bool big = G < 32 && c1 - c0 > kFinShort;
    AT acc = 0;
    if (!big) {
#pragma unroll 4
      for (i32 j = c0 + sub; j < c1; j += G) acc += part[j];
    }
    for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    for (unsigned todo = __ballot_sync(0xffffffffu, big && sub == 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const i32 d0 = __shfl_sync(0xffffffffu, c0, src), d1 = __shfl_sync(0xffffffffu, c1, src);
      AT s = 0;
#pragma unroll 4
      for (i32 j = d0 + lane; j < d1; j += 32) s += part[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == src) acc = s;
    }
    if (valid && sub == 0) {
      if constexpr (EPI == EPI_STORE) {
        ((YT*)f.y)[row] = (YT)acc;
      } else {
        AT loss, d, wtx = acc + b;
        if (f.ybase) wtx += f.ybase[row];
        glm_row<AT>(f.loss, (AT)f.eps, wtx, f.label_f[row], loss, d);
        if (f.sw_f) d = d * f.sw_f[row];
        ((YT*)f.r)[row] = (YT)d;
        f.long_part[2 * i] = (double)loss;
        f.long_part[2 * i + 1] = (double)d;
      }
    }
  }
  if (EPI == EPI_LOGREG)
    reduce_loss(f.cta_part, f.ncta, f.long_part, f.nlong, f.icpt, f.out, f.grad_bias, f.ticket);
}

// ------------------------------------------------- per-row logistic pass
// The loss rows over a finished product z = A w (in place when wtx == r):
// layouts whose product is computed first (ELL / JDS / hybrid) and the FP64
// CRS pass.  A thread per row, so that all 32 lanes share each FP64
// instruction of the loss: inside the product kernel only the lanes that
// held a row total (12 of 32 at 40 entries a row) would.  The last CTA
// reduces the CTAs' loss / bias partials in a fixed order.
//
// FP64: bound by the FP64 unit (64 clocks of its scheduler a warp instruction) and, on small
// matrices, by the launch and the reduction.  With the loss of logistic64.cuh
// and a thread's first row stored as its sum (the compensated add costs 4
// FP64 instructions, and up to 311,000 rows a thread has one): 100,000
// logistic rows 20.4 us, 26.3 with the library's exp, log and division.
template <class V> struct FirstRow {
  V v = 0;
  __device__ __forceinline__ void add(V x) { v = x; }
};
template <class AT>
__global__ void __launch_bounds__(kThreads) k_logreg_rows(const AT* wtx, i64 m, const CrsK p, double* out,
                                                          double* grad_bias, unsigned* ticket) {
  typename SumOf<AT>::type ls, bs;
  const AT b = p.icpt ? (AT)*p.intercept : (AT)0;
  i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < m) {
    FirstRow<AT> l1, b1;
    epilogue<AT, AT, EPI_LOGREG>(p, (i32)r, wtx[r], b, l1, b1);
    ls.s = l1.v;
    bs.s = b1.v;
  }
  for (r += (i64)gridDim.x * blockDim.x; r < m; r += (i64)gridDim.x * blockDim.x)
    epilogue<AT, AT, EPI_LOGREG>(p, (i32)r, wtx[r], b, ls, bs);
  block_csum2(ls.total(), bs.total(), &p.cta_part[2 * blockIdx.x], &p.cta_part[2 * blockIdx.x + 1]);
  reduce_loss(p.cta_part, gridDim.x, nullptr, 0, p.icpt, out, grad_bias, ticket);
}

// ------------------------------------------------------------- host side
static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

struct PassScratch {
  unsigned* ticket;
  double* out;
  double* cta_part;
  double* long_part;
  void* partials;
};

static size_t carve(char* base, const Sched& s, int grid, size_t at_size, PassScratch* ps) {
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += align256(b); return base ? base + r : nullptr; };
  char* t = take(sizeof(unsigned) * 2);
  char* out = take(sizeof(double) * 2);
  char* cp = take(sizeof(double) * 2 * (size_t)grid);
  char* lp = take(sizeof(double) * 2 * (size_t)std::max<i64>(s.nlong, 1));
  char* pa = take(at_size * (size_t)std::max<i64>(s.npieces, 1));
  if (ps) {
    ps->ticket = (unsigned*)t;
    ps->out = (double*)out;
    ps->cta_part = (double*)cp;
    ps->long_part = (double*)lp;
    ps->partials = pa;
  }
  return o;
}

i64 crs_pass_scratch_bytes(fvg_ctx* c, DevCRS& a, int storage) {
  const Sched& s = pass_sched(c, a, storage);
  return (i64)carve(nullptr, s, c->grid_spmv, 8, nullptr);
}

// Long rows a warp of k_finalize takes at a time: one while every row can
// have a warp of its own, four above that (4,864 rows on 152 SMs).
static int fin_rows(fvg_ctx* c, const Sched& s) { return s.nlong > 4ll * c->num_sms * (kThreads / 32) ? 4 : 1; }
static int fin_grid(fvg_ctx* c, const Sched& s) {
  const i64 per_cta = (i64)fin_rows(c, s) * (kThreads / 32);
  return (int)std::max<i64>(1, std::min<i64>((s.nlong + per_cta - 1) / per_cta, 4 * c->num_sms));
}

template <class VT, class XT, class AT, class YT, int EPI>
static int crs_grid(fvg_ctx* c) {
  return occupancy_blocks((const void*)k_crs<VT, XT, AT, YT, EPI>, kThreads) * c->num_sms;
}

template <class VT, class XT, class AT, class YT, int EPI>
static void launch_crs(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, const void* x, void* y,
                       const LogregEpi* lr, const PassScratch& ps, bool timed = true) {
  CrsK p;
  p.off = a.off.as<i32>();
  p.idx = a.idx.as<i32>();
  p.val = a.val[storage].p;
  p.x = x;
  p.items = s.items.as<Item>();
  p.nitems = s.nitems;
  p.y = y;
  p.partials = ps.partials;
  p.label = lr ? lr->label : nullptr;
  p.sw = lr ? lr->sw : nullptr;
  p.label_f = lr ? lr->label_f : nullptr;
  p.sw_f = lr ? lr->sw_f : nullptr;
  p.intercept = lr ? lr->intercept : nullptr;
  p.icpt = lr ? lr->icpt : 0;
  p.r = lr ? lr->r : nullptr;
  p.ybase = lr ? lr->ybase : nullptr;
  p.cta_part = ps.cta_part;
  p.loss = lr ? lr->loss : 0;
  p.eps = lr ? lr->eps : 0.0;
  int grid = (int)std::max<i64>(1, std::min<i64>(crs_grid<VT, XT, AT, YT, EPI>(c), s.nitems));
  grid = std::min(grid, c->grid_spmv);
  if (s.nitems > 0) {
    k_crs<VT, XT, AT, YT, EPI><<<grid, kThreads, 0, c->stream>>>(p);
    check_launch("k_crs");
    count_launch(c);
  }
  if (s.nlong > 0 || EPI == EPI_LOGREG) {
    FinK f;
    f.long_rows = s.long_rows.as<i32>();
    f.long_piece0 = s.long_piece0.as<i32>();
    f.nlong = s.nlong;
    f.partials = ps.partials;
    f.y = y;
    f.label_f = p.label_f;
    f.sw_f = p.sw_f;
    f.intercept = p.intercept;
    f.icpt = p.icpt;
    f.r = p.r;
    f.ybase = p.ybase;
    f.cta_part = ps.cta_part;
    f.ncta = s.nitems > 0 ? grid : 0;
    f.long_part = ps.long_part;
    f.out = (lr && lr->out) ? lr->out : ps.out;
    f.grad_bias = lr ? lr->grad_bias : nullptr;
    f.ticket = ps.ticket;
    f.loss = p.loss;
    f.eps = p.eps;
    f.per_warp = fin_rows(c, s);
    const int fg = fin_grid(c, s);
    ProfScope pf(c, timed ? P_FINALIZE : P_NKEYS);
    k_finalize<AT, YT, EPI><<<fg, kThreads, 0, c->stream>>>(f);
    check_launch("k_finalize");
    count_launch(c);
  }
}

// Raises the FP64 kernel's shared memory limit and sets its share of the
// SM's memory, once per device.
static void crs64_setup(fvg_ctx* c) {
  static std::mutex mu;  // contexts of different host threads launch concurrently
  static std::vector<int> done;
  std::lock_guard<std::mutex> lock(mu);
  if (std::find(done.begin(), done.end(), c->device) != done.end()) return;
  int per_sm = 0, reserved = 0;
  FVG_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c->device));
  FVG_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, c->device));
  FVG_CUDA(cudaFuncSetAttribute(k_crs64, cudaFuncAttributeMaxDynamicSharedMemorySize, kC64Smem));
  const i64 need = 100ll * kC64Blocks * (kC64Smem + reserved);
  FVG_CUDA(cudaFuncSetAttribute(k_crs64, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)std::min<i64>(100, (need + per_sm - 1) / per_sm)));
  done.push_back(c->device);
}

// y = A x, FP64 values and vectors.
static void launch_crs64(fvg_ctx* c, DevCRS& a, const Sched& s, const void* x, void* y, void* partials,
                         bool timed = true) {
  if (s.nitems > 0) {
    Crs64K p;
    p.off = a.off.as<i32>();
    p.idx = a.idx.as<i32>();
    p.val = a.val[FVG_F64].as<double>();
    p.x = (const double*)x;
    p.items = s.items.as<Item>();
    p.nitems = s.nitems;
    p.y = (double*)y;
    p.partials = (double*)partials;
    crs64_setup(c);
    const int grid = (int)std::min<i64>((i64)kC64Blocks * c->num_sms, s.nitems);
    k_crs64<<<grid, kC64Threads, kC64Smem, c->stream>>>(p);
    check_launch("k_crs64");
    count_launch(c);
  }
  if (s.nlong > 0) {
    FinK f = {};
    f.long_rows = s.long_rows.as<i32>();
    f.long_piece0 = s.long_piece0.as<i32>();
    f.nlong = s.nlong;
    f.partials = partials;
    f.y = y;
    f.per_warp = fin_rows(c, s);
    const int fg = fin_grid(c, s);
    ProfScope pf(c, timed ? P_FINALIZE : P_NKEYS);
    k_finalize<double, double, EPI_STORE><<<fg, kThreads, 0, c->stream>>>(f);
    check_launch("k_finalize");
    count_launch(c);
  }
}

// The per-row loss pass over z (see k_logreg_rows); ticket zero on entry.
static int logreg_rows_grid(fvg_ctx* c, i64 m) {
  return (int)std::max<i64>(1, std::min<i64>(c->grid_spmv, (m + kThreads - 1) / kThreads));
}
static void launch_logreg_rows(fvg_ctx* c, const void* z, int z_dt, i64 m, const LogregEpi& lr, unsigned* ticket,
                               double* cta_part, double* out) {
  CrsK p = {};
  p.label = lr.label;
  p.sw = lr.sw;
  p.label_f = lr.label_f;
  p.sw_f = lr.sw_f;
  p.intercept = lr.intercept;
  p.icpt = lr.icpt;
  p.r = lr.r;
  p.cta_part = cta_part;
  p.loss = lr.loss;
  p.eps = lr.eps;
  const int grid = logreg_rows_grid(c, m);
  if (z_dt == FVG_F64)
    k_logreg_rows<double><<<grid, kThreads, 0, c->stream>>>((const double*)z, m, p, out, lr.grad_bias, ticket);
  else
    k_logreg_rows<float><<<grid, kThreads, 0, c->stream>>>((const float*)z, m, p, out, lr.grad_bias, ticket);
  check_launch("k_logreg_rows");
  count_launch(c);
}

void crs_pass(fvg_ctx* c, DevCRS& a, int storage, int x_dt, const void* x, int y_dt, void* y, int epi,
              const LogregEpi* lr, void* scratch, int prof_key) {
  const Sched& s = pass_sched(c, a, storage);
  if (!a.val[storage].p) fail(FVG_ERR_INTERNAL, "missing value plane for the requested storage");
  const size_t at_size = (storage == FVG_F64) ? 8 : 4;
  DBuf tmp;
  PassScratch ps = {};
  if (scratch) {
    carve((char*)scratch, s, c->grid_spmv, at_size, &ps);
  } else if (epi == EPI_STORE) {  // a lone product: long rows' partials are all it needs
    if (s.npieces > 0) tmp.alloc(at_size * (size_t)s.npieces, c->stream);
    ps.partials = tmp.p;
  } else {
    tmp.alloc(carve(nullptr, s, c->grid_spmv, at_size, nullptr), c->stream);
    FVG_CUDA(cudaMemsetAsync(tmp.p, 0, 256, c->stream));  // ticket
    carve((char*)tmp.p, s, c->grid_spmv, at_size, &ps);
  }
  if (epi == EPI_LOGREG && storage != FVG_F64 && !(lr && lr->label_f))
    fail(FVG_ERR_INTERNAL, "FP32 logistic pass needs FP32 labels");
  ProfScope pr(c, prof_key);
  const int out_dt = (epi == EPI_LOGREG) ? (lr ? lr->r_dt : y_dt) : y_dt;
  if (storage == FVG_F64) {
    if (x_dt != FVG_F64 || out_dt != FVG_F64) fail(FVG_ERR_INVALID_ARG, "FP64 values need FP64 vectors");
    if (epi == EPI_STORE) {
      launch_crs64(c, a, s, x, y, ps.partials);
    } else {  // z into r, then the loss rows in place
      launch_crs64(c, a, s, x, lr->r, ps.partials);
      launch_logreg_rows(c, lr->r, FVG_F64, a.m, *lr, ps.ticket, ps.cta_part, lr->out ? lr->out : ps.out);
    }
  } else if (storage == FVG_F32) {
    if (x_dt != FVG_F32) fail(FVG_ERR_INVALID_ARG, "FP32 values need FP32 input vectors");
    if (epi == EPI_STORE && out_dt == FVG_F64)
      launch_crs<float, float, float, double, EPI_STORE>(c, a, s, storage, x, y, lr, ps);
    else if (epi == EPI_STORE)
      launch_crs<float, float, float, float, EPI_STORE>(c, a, s, storage, x, y, lr, ps);
    else
      launch_crs<float, float, float, float, EPI_LOGREG>(c, a, s, storage, x, y, lr, ps);
  } else {
    if (x_dt != FVG_F32) fail(FVG_ERR_INVALID_ARG, "BF16 values need FP32 input vectors");
    if (epi == EPI_STORE && out_dt == FVG_F64)
      launch_crs<bf16, float, float, double, EPI_STORE>(c, a, s, storage, x, y, lr, ps);
    else if (epi == EPI_STORE)
      launch_crs<bf16, float, float, float, EPI_STORE>(c, a, s, storage, x, y, lr, ps);
    else
      launch_crs<bf16, float, float, float, EPI_LOGREG>(c, a, s, storage, x, y, lr, ps);
  }
}

// y = A x over a CRS layout whose work schedule already exists, with the
// caller's scratch (piece partial sums only) and no allocation of any kind.
// Returns the scratch bytes the pass needs when scratch is null.
size_t crs_spmv_no_alloc(fvg_ctx* c, DevCRS& a, int storage, const void* x, void* y, void* scratch,
                         size_t scratch_bytes) {
  // its own work items; where another storage's first use made the matrix's
  // only ones, those (both kernels take either list)
  const int own = storage == FVG_F64 ? 2 : 0;
  const Sched* s = a.sched[a.sched[own] ? own : 2 - own].get();
  if (!s) fail(FVG_ERR_INVALID_ARG, "matrix not prepared: call fvg_matrix_prepare(ctx, mat, FVG_CRS, ...) first");
  if (!a.val[storage].p) fail(FVG_ERR_INVALID_ARG, "value plane missing: call fvg_matrix_add_storage first");
  const size_t at_size = (storage == FVG_F64) ? 8 : 4;
  const size_t need = at_size * (size_t)std::max<i64>(s->npieces, 1);
  if (!scratch) return need;
  if (need > scratch_bytes) fail(FVG_ERR_INVALID_ARG, "matrix needs more scratch than the allocation-free entry point has");
  PassScratch ps = {};
  ps.partials = scratch;
  if (storage == FVG_F64)
    launch_crs64(c, a, *s, x, y, ps.partials, false);
  else if (storage == FVG_F32)
    launch_crs<float, float, float, float, EPI_STORE>(c, a, *s, storage, x, y, nullptr, ps, false);
  else
    launch_crs<bf16, float, float, float, EPI_STORE>(c, a, *s, storage, x, y, nullptr, ps, false);
  return need;
}

// ------------------------------------------------------------------- JDS
// Work items (JdsItem): a warp per block of 32 consecutive permuted rows
// (lane = row) and at most kJdsSeg of the block's diagonals.  Diagonal d of
// row p sits at off[d] + p, so the warp reads each diagonal's 32 entries
// with one coalesced access; row p has diagonal d iff the diagonal's length
// off[d+1] - off[d] exceeds p.  Four diagonals are summed into four
// accumulators, added as (a0 + a1) + (a2 + a3) at the item's end.  A block
// with more diagonals than one item holds leaves per-row partials, which
// k_jds_split adds in diagonal order.  part (hybrid) adds the CRS tail of
// the first npart permuted rows after the JDS sum, as
// jds_crs_hybrid_spmv_impl does (jds_crs_hybrid.hpp:198-211).
template <class VT, class XT, class AT>
__device__ __forceinline__ AT jds_term(const VT* __restrict__ val, const i32* __restrict__ idx,
                                       const XT* __restrict__ x, i64 q) {
  return (AT)val[q] * (AT)__ldg(x + __ldg(idx + q));
}

template <class VT, class XT, class AT, class YT>
__global__ void __launch_bounds__(256) k_jds(const JdsItem* __restrict__ items, i64 nitems,
                                             const i32* __restrict__ perm, const i64* __restrict__ off,
                                             const i32* __restrict__ idx, const VT* __restrict__ val, i64 m,
                                             const XT* __restrict__ x, YT* __restrict__ y,
                                             const AT* __restrict__ part, i64 npart, AT* __restrict__ partials) {
  const int lane = threadIdx.x & 31;
  const i64 nw = ((i64)gridDim.x * blockDim.x) >> 5;
  for (i64 it = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < nitems; it += nw) {
    const JdsItem t = items[it];
    const i64 p = (i64)t.b * 32 + lane;
    AT a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    i64 d = t.d0;
    i64 o = __ldg(off + d);
    for (; d + 3 < t.d1; d += 4) {
      const i64 o1 = __ldg(off + d + 1), o2 = __ldg(off + d + 2), o3 = __ldg(off + d + 3), o4 = __ldg(off + d + 4);
      if (p < o1 - o) a0 += jds_term<VT, XT, AT>(val, idx, x, o + p);
      if (p < o2 - o1) a1 += jds_term<VT, XT, AT>(val, idx, x, o1 + p);
      if (p < o3 - o2) a2 += jds_term<VT, XT, AT>(val, idx, x, o2 + p);
      if (p < o4 - o3) a3 += jds_term<VT, XT, AT>(val, idx, x, o3 + p);
      o = o4;
    }
    for (; d < t.d1; d++) {
      const i64 o1 = __ldg(off + d + 1);
      if (p < o1 - o) a0 += jds_term<VT, XT, AT>(val, idx, x, o + p);
      o = o1;
    }
    AT acc = (a0 + a1) + (a2 + a3);
    if (t.slot >= 0) {
      partials[(i64)t.slot * 32 + lane] = acc;
    } else if (p < m) {
      if (p < npart) acc = acc + part[p];
      y[perm[p]] = (YT)acc;
    }
  }
}

// blocks cut into several items: their partials in diagonal order
template <class AT, class YT>
__global__ void __launch_bounds__(256) k_jds_split(const JdsSplit* __restrict__ sp, i64 nsplits,
                                                   const i32* __restrict__ perm, i64 m, YT* __restrict__ y,
                                                   const AT* __restrict__ part, i64 npart,
                                                   const AT* __restrict__ partials) {
  const int lane = threadIdx.x & 31;
  const i64 nw = ((i64)gridDim.x * blockDim.x) >> 5;
  for (i64 i = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nsplits; i += nw) {
    const JdsSplit s = sp[i];
    const i64 p = (i64)s.b * 32 + lane;
    AT acc = 0;
    for (int q = 0; q < s.nslot; q++) acc += partials[(i64)(s.slot0 + q) * 32 + lane];
    if (p < m) {
      if (p < npart) acc = acc + part[p];
      y[perm[p]] = (YT)acc;
    }
  }
}

template <class T> __global__ void k_zero(T* y, i64 n) {
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) y[i] = (T)0;
}

static unsigned grid_rows(i64 n) {
  i64 g = (n + 255) / 256;
  if (g > 152 * 16) g = 152 * 16;
  return (unsigned)(g < 1 ? 1 : g);
}

template <class VT, class XT, class AT, class YT>
static void launch_jds(fvg_ctx* c, DevJDS& j, int storage, const void* x, void* y, const void* part, i64 npart) {
  if (j.m == 0) return;
  if (j.empty_perm) {
    k_zero<YT><<<grid_rows(j.m), 256, 0, c->stream>>>((YT*)y, j.m);
  } else {
    DBuf partials;
    if (j.nslots > 0) partials.alloc(sizeof(AT) * 32 * (size_t)j.nslots, c->stream);
    k_jds<VT, XT, AT, YT><<<grid_rows(j.nitems * 32), 256, 0, c->stream>>>(
        j.items.as<JdsItem>(), j.nitems, j.perm.as<i32>(), j.off.as<i64>(), j.idx.as<i32>(), j.val[storage].as<VT>(),
        j.m, (const XT*)x, (YT*)y, (const AT*)part, npart, partials.as<AT>());
    if (j.nsplits > 0) {
      check_launch("k_jds");
      count_launch(c);
      k_jds_split<AT, YT><<<grid_rows(j.nsplits * 32), 256, 0, c->stream>>>(
          j.splits.as<JdsSplit>(), j.nsplits, j.perm.as<i32>(), j.m, (YT*)y, (const AT*)part, npart,
          partials.as<AT>());
    }
  }
  check_launch("k_jds");
  count_launch(c);
}

static void jds_dispatch(fvg_ctx* c, DevJDS& j, int storage, int x_dt, const void* x, int y_dt, void* y,
                         const void* part, i64 npart) {
  if (storage == FVG_F64) {
    if (x_dt != FVG_F64 || y_dt != FVG_F64) fail(FVG_ERR_INVALID_ARG, "FP64 values need FP64 vectors");
    launch_jds<double, double, double, double>(c, j, storage, x, y, part, npart);
  } else if (storage == FVG_F32) {
    if (y_dt == FVG_F64) launch_jds<float, float, float, double>(c, j, storage, x, y, part, npart);
    else launch_jds<float, float, float, float>(c, j, storage, x, y, part, npart);
  } else {
    if (y_dt == FVG_F64) launch_jds<bf16, float, float, double>(c, j, storage, x, y, part, npart);
    else launch_jds<bf16, float, float, float>(c, j, storage, x, y, part, npart);
  }
}

void jds_spmv(fvg_ctx* c, DevJDS& j, int storage, int x_dt, const void* x, int y_dt, void* y, bool) {
  ProfScope pr(c, P_SPMV_JDS);
  ensure_plane_generic(c, j.val, j.nnz, storage, FVG_F64);
  jds_dispatch(c, j, storage, x_dt, x, y_dt, y, nullptr, 0);
}

void hyb_spmv(fvg_ctx* c, DevHYB& h, int storage, int x_dt, const void* x, int y_dt, void* y) {
  ProfScope pr(c, P_SPMV_HYB);
  if (h.all_crs) {  // whole matrix in the CRS part, natural row order
    crs_pass(c, h.crs, storage, x_dt, x, y_dt, y, EPI_STORE, nullptr, nullptr, P_NKEYS);
    return;
  }
  DBuf part;
  const int at = (storage == FVG_F64) ? FVG_F64 : FVG_F32;
  if (h.crs_rows > 0) {
    part.alloc((size_t)dtype_size(at) * h.crs_rows, c->stream);
    crs_pass(c, h.crs, storage, x_dt, x, at, part.p, EPI_STORE, nullptr, nullptr, P_NKEYS);
  }
  jds_dispatch(c, h.jds, storage, x_dt, x, y_dt, y, part.p, h.crs_rows);
}

// ------------------------------------------------------------------- ELL
template <class VT, class XT, class AT, class YT>
__global__ void __launch_bounds__(256) k_ell(const i32* __restrict__ idx, const VT* __restrict__ val, i64 m,
                                             i64 width, const XT* __restrict__ x, YT* __restrict__ y) {
  for (i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += (i64)gridDim.x * blockDim.x) {
    AT a0 = 0, a1 = 0;
    i64 k = 0;
    for (; k + 1 < width; k += 2) {
      i64 q0 = k * m + r, q1 = q0 + m;
      a0 += (AT)val[q0] * (AT)__ldg(x + idx[q0]);
      a1 += (AT)val[q1] * (AT)__ldg(x + idx[q1]);
    }
    if (k < width) a0 += (AT)val[k * m + r] * (AT)__ldg(x + idx[k * m + r]);
    y[r] = (YT)(a0 + a1);
  }
}

void ell_spmv(fvg_ctx* c, DevELL& e, int storage, int x_dt, const void* x, int y_dt, void* y) {
  ProfScope pr(c, P_SPMV_ELL);
  if (e.m == 0) return;
  ensure_plane_generic(c, e.val, e.m * e.width, storage, FVG_F64);
  unsigned g = grid_rows(e.m);
  if (storage == FVG_F64) {
    if (x_dt != FVG_F64 || y_dt != FVG_F64) fail(FVG_ERR_INVALID_ARG, "FP64 values need FP64 vectors");
    k_ell<double, double, double, double><<<g, 256, 0, c->stream>>>(e.idx.as<i32>(), e.val[storage].as<double>(),
                                                                    e.m, e.width, (const double*)x, (double*)y);
  } else if (storage == FVG_F32) {
    if (y_dt == FVG_F64)
      k_ell<float, float, float, double><<<g, 256, 0, c->stream>>>(e.idx.as<i32>(), e.val[storage].as<float>(), e.m,
                                                                   e.width, (const float*)x, (double*)y);
    else
      k_ell<float, float, float, float><<<g, 256, 0, c->stream>>>(e.idx.as<i32>(), e.val[storage].as<float>(), e.m,
                                                                  e.width, (const float*)x, (float*)y);
  } else {
    if (y_dt == FVG_F64)
      k_ell<bf16, float, float, double><<<g, 256, 0, c->stream>>>(e.idx.as<i32>(), e.val[storage].as<bf16>(), e.m,
                                                                  e.width, (const float*)x, (double*)y);
    else
      k_ell<bf16, float, float, float><<<g, 256, 0, c->stream>>>(e.idx.as<i32>(), e.val[storage].as<bf16>(), e.m,
                                                                 e.width, (const float*)x, (float*)y);
  }
  check_launch("k_ell");
  count_launch(c);
}

// Resident CTAs per SM of the heaviest CRS instantiation (sizes the
// persistent grid).
// Upper bound of resident 256-thread CTAs per SM; sizes the per-CTA partial
// buffers (the launch itself uses the occupancy of each instantiation).
int crs_blocks_per_sm() { return 2048 / kThreads; }

// logistic_regression_model<T>::predict_probability (ml/glm/linear_model.hpp:
// 376-392): v += intercept (when non-zero); exp argument above 709 → 0.
__global__ void k_sigmoid(double* v, i64 m, double b) {
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (i64)gridDim.x * blockDim.x) {
    double x = v[i];
    if (b != 0) x += b;
    double e = -1.0 * x;
    v[i] = (e > 709) ? 0.0 : 1.0 / (1.0 + exp(e));
  }
}

void sigmoid_probability(fvg_ctx* c, double* v, i64 m, double b) {
  if (m <= 0) return;
  k_sigmoid<<<grid_rows(m), 256, 0, c->stream>>>(v, m, b);
  check_launch("k_sigmoid");
  count_launch(c);
}

void logreg_rows(fvg_ctx* c, const void* wtx, int wtx_dt, i64 m, const LogregEpi& lr) {
  DBuf tmp;
  tmp.alloc(512 + sizeof(double) * 2 * (size_t)logreg_rows_grid(c, m), c->stream);
  FVG_CUDA(cudaMemsetAsync(tmp.p, 0, 256, c->stream));
  launch_logreg_rows(c, wtx, wtx_dt, m, lr, (unsigned*)tmp.p, (double*)((char*)tmp.p + 512),
                     lr.out ? lr.out : (double*)((char*)tmp.p + 256));
}

}  // namespace fvg
