// Shared-memory gathers for the FP32-arithmetic passes, and the device
// packing of every work-item schedule.
//
// Backward product g = A^T r (row panels).  The reference multiplies its
// transposed copy (crs_matrix.hpp:356-412 builds it, gradient_descent.hpp:211
// multiplies it with dloss), and so does the plain path here: every nonzero
// of A^T gathers r[source row].  With millions of rows r sits in L2 and each
// gather of a sparsely used column fetches a 32-byte sector for 4 useful
// bytes, so that pass is bound by L2-to-SM traffic, far below HBM speed.
// The row-panel layout regroups the columns that occur in most stretches of
// rows.  A's rows are cut into panels of `rows` consecutive rows.  A CTA
// copies one panel's slice of r into shared memory and streams the panel's
// entries of the hot columns, gathering from shared memory; each (panel, hot
// column) pair gives one partial sum ("panel row" q = panel * nhot + h).  g[hot column] is the compensated sum of its
// partials in a fixed order.  Columns with fewer entries keep their rows in
// a transposed CRS of their own (the hot rows emptied), multiplied by the
// plain CRS kernel first.
//
// Forward product A w (forward head).  The entries of A's most frequent
// columns form a CRS of their own with 2-byte column slots; every CTA stages
// w at those columns once and sums its share of the rows' head entries with
// the same kernel; the rest of each row goes through the plain CRS kernel,
// whose logistic epilogue adds the head partial (crs_matrix.hpp:1505-1516 is
// the product, gradient_descent.hpp:227-240 and gradient.hpp:15-53 the
// epilogue).
//
// Every sum has a fixed order, so results are the same on every run.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "bulk_copy.cuh"
#include "device_common.cuh"
#include "df64.cuh"
#include "split_bits.h"

namespace fvg {

namespace {

unsigned grid_n(i64 n, int threads = 256) {
  i64 g = (n + threads - 1) / threads;
  if (g > 152 * 32) g = 152 * 32;
  return (unsigned)(g < 1 ? 1 : g);
}
// Warps of the streamed product, bulk copies in flight per warp, chunks a copy
// (build-time knobs; the defaults are the measured best).
#ifndef FVG_STREAM_WARPS
#define FVG_STREAM_WARPS 20
#endif
#ifndef FVG_STREAM_STAGES
#define FVG_STREAM_STAGES 2
#endif
#ifndef FVG_STREAM_CHUNKS
#define FVG_STREAM_CHUNKS 2
#endif
#define PGRID_STRIDE(i, n) for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (i64)gridDim.x * blockDim.x)
#define PWARP_STRIDE(q, n)                                                              \
  for (i64 q = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < (n);             \
       q += ((i64)gridDim.x * blockDim.x) >> 5)

constexpr i64 kPanelMinRows = 4096;      // auto: shortest panels
// auto: rows of a matrix that gets panels, 22 of the shortest.  A^T x, 50
// entries a row, BF16 values: the plain product takes 31 us at 89,000 rows, the
// panels 60; 46 and 65 at 200,000; 71 and 70 at 400,000; 153 and 104 at
// 1,000,000.  Between the line and 400,000 rows the panels are there for their
// error: 6e-8 to 9e-8 of the 64-bit product, 9e-8 to 1.3e-7 without.
constexpr i64 kPanelMinMatrix = 22 * kPanelMinRows;
// auto: rows per SM of a matrix that gets a head.  A w and the loss rows, 50
// entries a row, with / without: BF16 values 40 / 34 us at 100,000 rows, 54 / 53
// at 300,000, 60 / 67 at 450,000, 73 / 92 at 700,000; split values 39 / 38, 67 /
// 76, 80 / 105 and 106 / 153.
constexpr i64 kHeadMinPerSm = 2048;
constexpr double kPanelMinAuto = 2.0;    // hot: >= this many entries per panel on average

// ------------------------------------------------------------------ build
__global__ void k_hot_flags(const i32* __restrict__ toff, i64 n, i64 thresh, i64* __restrict__ flag) {
  PGRID_STRIDE(c, n) flag[c] = ((i64)toff[c + 1] - toff[c] >= thresh) ? 1 : 0;
}

__global__ void k_hot_list(const i64* __restrict__ flag, const i64* __restrict__ pos, i64 n, i32* __restrict__ hot) {
  PGRID_STRIDE(c, n) if (flag[c]) hot[pos[c]] = (i32)c;
}

// B[h*(np+1) + p]: position in A^T of the first entry of hot column h whose
// source row is >= p*rows (the column's source rows ascend).
__global__ void k_panel_bounds(const i32* __restrict__ toff, const i32* __restrict__ tidx, const i32* __restrict__ hot,
                               i64 nhot, i64 np, i64 rows, i32* __restrict__ B) {
  PGRID_STRIDE(i, nhot * (np + 1)) {
    const i64 h = i / (np + 1), p = i - h * (np + 1);
    const i32 c = hot[h];
    i64 lo = toff[c], hi = toff[c + 1];
    const i64 target = p * rows;
    while (lo < hi) {
      const i64 mid = (lo + hi) >> 1;
      if ((i64)tidx[mid] < target) lo = mid + 1;
      else hi = mid;
    }
    B[i] = (i32)lo;
  }
}

__global__ void k_panel_lens(const i32* __restrict__ B, i64 nhot, i64 np, i64* __restrict__ len) {
  PGRID_STRIDE(q, np * nhot) {
    const i64 p = q / nhot, h = q - p * nhot;
    len[q] = (i64)B[h * (np + 1) + p + 1] - B[h * (np + 1) + p];
  }
}

__global__ void k_i64_to_i32(const i64* __restrict__ s, i32* __restrict__ d, i64 n) {
  PGRID_STRIDE(i, n) d[i] = (i32)s[i];
}

// The source's other value planes (FP32, BF16, split residual) that a fill
// copies beside the master plane, so that a layout built from a matrix that
// already holds them needs no conversion afterwards; null where absent.
struct SidePlanes {
  const float* s32 = nullptr;
  float* d32 = nullptr;
  const bf16* s16 = nullptr;
  bf16* d16 = nullptr;
  const bf16* slo = nullptr;
  bf16* dlo = nullptr;
  __device__ __forceinline__ void copy(i64 from, i64 to) const {
    if (s32) d32[to] = s32[from];
    if (s16) d16[to] = s16[from];
    if (slo) dlo[to] = slo[from];
  }
};

__global__ void k_cold_lens(const i32* __restrict__ toff, const i64* __restrict__ flag, i64 n, i64* __restrict__ len) {
  PGRID_STRIDE(c, n) len[c] = flag[c] ? 0 : (i64)toff[c + 1] - toff[c];
}

template <class T>
__global__ void k_cold_fill(const i32* __restrict__ toff, const i64* __restrict__ flag, const i64* __restrict__ coff,
                            i64 n, const i32* __restrict__ tidx, const T* __restrict__ tval, i32* __restrict__ cidx,
                            T* __restrict__ cval, const SidePlanes sp) {
  const int lane = threadIdx.x & 31;
  PWARP_STRIDE(c, n) {
    if (flag[c]) continue;
    const i64 s = toff[c], e = toff[c + 1], d = coff[c];
    for (i64 k = lane; k < e - s; k += 32) {
      cidx[d + k] = tidx[s + k];
      cval[d + k] = tval[s + k];
      sp.copy(s + k, d + k);
    }
  }
}

// Work items of a CRS, one CTA per chunk of `step` rows (at most kPackRows),
// with the CRS schedule's packing rules
// (tiles of short rows within `tile` entries, kTileRows rows and lane_work
// products per lane; longer rows in pieces cut at 8-element boundaries).  The
// greedy packing is sequential from tile to tile, but where a tile ends
// depends only on where it starts: thread t finds the end of a tile starting
// at the chunk's row t (every limit, once passed, stays passed), one thread
// follows the ends from row 0 and marks the starts met, and the marked rows
// are counted and written side by side.  Pass 0 counts each chunk's items,
// long rows and pieces; pass 1 writes them at the scanned offsets `base`
// (chunk-major: a chunk's items, long rows and pieces are contiguous and
// numbered globally).
// Bound by the walk over the starts (up to 256 dependent reads of shared
// memory): 12.7 us a pass over the transposed 25,600 x 20,000 minibatches of a
// Zipf matrix; 44 us with the warp searching each tile's end in turn.
constexpr int kPackThreads = (int)kPackRows;
__global__ void __launch_bounds__(kPackThreads) k_pack(const i32* __restrict__ off, i64 nrows, i64 step, i64 np, int tile,
                                                    int write, i32* __restrict__ cnt,
                                                    const i32* __restrict__ base, Item* __restrict__ items,
                                                    i32* __restrict__ lrows, i32* __restrict__ lpiece0,
                                                    i32* __restrict__ lfirst, int lane_work) {
  constexpr int kWarps = kPackThreads / 32;
  __shared__ i32 so[kPackThreads + 1];
  __shared__ short nxt[kPackThreads];
  __shared__ unsigned char start[kPackThreads];
  __shared__ i32 wsum[3][kWarps];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (i64 p = blockIdx.x; p < np; p += gridDim.x) {
    const i64 r0 = min(p * step, nrows);
    const int R = (int)(min(r0 + step, nrows) - r0);  // rows of the chunk
    __syncthreads();
    if (t < R) so[t + 1] = __ldg(off + r0 + t + 1);
    if (t == 0) so[0] = __ldg(off + r0);
    start[t] = 0;
    __syncthreads();
    const i32 ob = t < R ? so[t] : 0, oe = t < R ? so[t + 1] : 0;
    const bool lng = oe - ob > tile;
    int e = t + 1;  // one past the last row of the item that starts at row t
    if (t < R && !lng) {
      i32 prev = oe;
      int mx = oe - ob;
      for (; e < R && e - t < kTileRows; e++) {
        const i32 o = so[e + 1];
        const int len = o - prev;
        mx = max(mx, len);
        if (len > tile || o - ob > tile || mx > lane_work * lanes_per_row(e - t + 1)) break;
        prev = o;
      }
    }
    nxt[t] = (short)e;
    __syncthreads();
    if (t == 0)
      for (int q = 0; q < R; q = nxt[q]) start[q] = 1;
    __syncthreads();
    const bool mine = start[t] != 0;
    const bool ml = mine && lng;
    const i64 b8 = (i64)ob & ~7ll;
    const i32 npr = ml ? (i32)(((i64)oe - b8 + tile - 1) / tile) : 0;  // pieces: b8 + k*tile < oe
    // items, long rows and pieces up to this row
    i32 v[3] = {ml ? npr : (mine ? 1 : 0), ml ? 1 : 0, npr}, x[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      x[q] = v[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const i32 u = __shfl_up_sync(0xffffffffu, x[q], o);
        if (lane >= o) x[q] += u;
      }
      if (lane == 31) wsum[q][w] = x[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; q++)
      for (int u = 0; u < w; u++) x[q] += wsum[q][u];
    if (!write) {
      if (t == kPackThreads - 1) {
        cnt[p] = x[0];
        cnt[np + p] = x[1];
        cnt[2 * np + p] = x[2];
      }
      continue;
    }
    const i32 it = base[p] + x[0] - v[0];
    if (ml) {
      const i32 l = base[(np + 1) + p] + x[1] - 1;
      lrows[l] = (i32)(r0 + t);
      lpiece0[l] = base[2 * (np + 1) + p] + x[2] - npr;
      lfirst[l] = it;  // its pieces' items follow (k_long_pieces)
    } else if (mine) {
      items[it] = Item{(int32_t)(r0 + t), (int32_t)(r0 + e), ob, so[e]};
    }
  }
}

// The items of the long rows' pieces (piece k of a row starting at st:
// [st, b8 + tile) for k = 0, then [b8 + k*tile, b8 + (k+1)*tile) cut at the
// row's end, b8 = st rounded down to 8), a warp per long row.
__global__ void k_long_pieces(const i32* __restrict__ off, const i32* __restrict__ lrows,
                              const i32* __restrict__ lpiece0, const i32* __restrict__ lfirst, i64 nlong, int tile,
                              Item* __restrict__ items) {
  const int lane = threadIdx.x & 31;
  PWARP_STRIDE(L, nlong) {
    const i32 r = lrows[L];
    const i64 st = off[r], en = off[r + 1], b8 = st & ~7ll;
    const i64 npr = (en - b8 + tile - 1) / tile;
    const i64 it0 = lfirst[L], pc0 = lpiece0[L];
    for (i64 k = lane; k < npr; k += 32) {
      const i64 e0 = (k == 0) ? st : b8 + k * tile, e1 = min(en, b8 + (k + 1) * tile);
      items[it0 + k] = Item{(int32_t)r, (int32_t)(-1 - (pc0 + k)), (int32_t)e0, (int32_t)e1};
    }
  }
}

// ---------------------------------------------------------- forward head
// The forward product y = A w gathers w[col] for every nonzero; the
// frequent columns' part of it takes the same route as the panels: A's
// entries in the H most frequent columns ("head") form their own CRS with
// uint16 column slots, and every CTA stages w at those columns in shared
// memory once.  The rows are cut into one stretch per CTA ("virtual
// panels" of the panel kernel); the rest of each row ("tail") stays a CRS
// with int32 column ids whose pass adds the head partial before the
// logistic epilogue.

// sort keys of the head selection: decreasing count (31-bit), the column
__global__ void k_head_keys(const i32* __restrict__ toff, i64 n, uint32_t* __restrict__ keys,
                            uint32_t* __restrict__ cols) {
  PGRID_STRIDE(j, n) {
    keys[j] = 0x7fffffffu - (uint32_t)(toff[j + 1] - toff[j]);
    cols[j] = (uint32_t)j;
  }
}

__global__ void k_head_slots(const uint32_t* __restrict__ cols, i64 H, i32* __restrict__ slot) {
  PGRID_STRIDE(i, H) slot[cols[i]] = (i32)i;
}

// per row: entries in head columns (slot >= 0) and in the tail
__global__ void k_head_counts(const i32* __restrict__ off, const i32* __restrict__ idx, i64 m,
                              const i32* __restrict__ slot, i64* __restrict__ hcnt, i64* __restrict__ tcnt) {
  const int lane = threadIdx.x & 31;
  PWARP_STRIDE(r, m) {
    const i64 s0 = off[r], e0 = off[r + 1];
    int h = 0;
    for (i64 e = s0 + lane; e < e0; e += 32) h += slot[idx[e]] >= 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
    if (lane == 0) {
      hcnt[r] = h;
      tcnt[r] = (e0 - s0) - h;
    }
  }
}

// head offsets padded to Q rows (rows past m are empty)
__global__ void k_head_off(const i64* __restrict__ hoff, i64 m, i64 Q, i32* __restrict__ poff) {
  PGRID_STRIDE(q, Q + 1) poff[q] = (i32)hoff[q < m ? q : m];
}

// a warp per row: its tail entries (column, value), in the row's order
template <class T>
__global__ void k_tail_fill(const i32* __restrict__ off, const i32* __restrict__ idx, const T* __restrict__ val,
                            i64 m, const i32* __restrict__ slot, const i64* __restrict__ toff,
                            i32* __restrict__ tidx, T* __restrict__ tval, const SidePlanes sp) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  PWARP_STRIDE(r, m) {
    const i64 s0 = off[r], e0 = off[r + 1];
    i64 tp = toff[r];
    constexpr int kRounds = 2;  // loads under way together
    for (i64 b = s0; b < e0; b += 32 * kRounds) {
      i32 col[kRounds];
      bool tail[kRounds];
#pragma unroll
      for (int u = 0; u < kRounds; u++) col[u] = b + 32 * u + lane < e0 ? idx[b + 32 * u + lane] : -1;
#pragma unroll
      for (int u = 0; u < kRounds; u++) tail[u] = col[u] >= 0 && slot[col[u]] < 0;
#pragma unroll
      for (int u = 0; u < kRounds; u++) {
        const unsigned tb = __ballot_sync(0xffffffffu, tail[u]);
        if (tail[u]) {
          const i64 e = b + 32 * u + lane, q = tp + __popc(tb & lt);
          tidx[q] = col[u];
          tval[q] = val[e];
          sp.copy(e, q);
        }
        tp += __popc(tb);
      }
    }
  }
}

// ---------------------------------------------------------------- product
// Streamed layout.  A panel row's entries are cut into segments of at most
// kSegChunks chunks of 4 entries; a panel's segments are sorted by length
// (stable, longest first) and dealt in slices of 32, a lane each.  Chunk c of
// a slice is one record: for every lane the 4 values (and BF16 residuals) and
// the 4 slots of its segment's entries 4c .. 4c+3, each kind contiguous over
// the lanes.  Segments that end earlier are padded with value 0 and the slot
// `rows`, whose staged vector entry is 0.  A warp's share of a panel is a run
// of slices, so it reads one contiguous stretch of memory; a lane adds its own
// segment from front to back and nothing is exchanged between lanes.
// (Measured against staging 480 entries a warp in row order, cutting them
// among the lanes by position and joining the rows with marks, selects and a
// segmented scan: that took 69 warp instructions per 32 entries of split
// values, this 30.  10M x 1M split values, 4.7e8 head and 4.9e8 panel entries:
// 1.12 + 1.29 ms before with 11,000-entry slices, 0.81 each now with 17,484
// head columns and panels of 16,448 rows, 5.4 TB/s of records, rows and sums;
// 2M x 200,000 BF16 values: 135 -> 124 us.  More copies in flight, larger
// copies, and records asked into L2 ahead of the copies change nothing or cost
// time, as does leaving out the gathers or the sums: the split stream is bound
// by HBM.  The BF16 one, half the bytes a chunk, is bound by the chain of a
// warp's copies: 8 / 16 / 24 warps took 188 / 124 / 113 us, 20 take 124, but
// the split rings of 24 warps leave too small a slice, and one layout serves
// every storage.)
constexpr int kStreamWarps = FVG_STREAM_WARPS;    // one CTA per SM
constexpr int kStreamStages = FVG_STREAM_STAGES;  // copies in flight per warp
constexpr int kStreamChunks = FVG_STREAM_CHUNKS;  // chunks of one copy
constexpr int kSegChunks = 16;                    // longest segment: 64 entries
constexpr int kAhead = 4;                         // slices whose row numbers are loaded early (a power of two)
constexpr i32 kNoRow = (i32)0x80000000;           // lane without a segment

// Record of a chunk by value storage: bytes of the values, residuals, slots.
template <int ST> struct StreamRec {
  using X = std::conditional_t<ST == FVG_SPLIT, float2, float>;  // vector entry
  static constexpr int kValB = (ST == FVG_BF16 ? 2 : 4) * 128;
  static constexpr int kLoB = ST == FVG_SPLIT ? 256 : 0;
  static constexpr int kB = kValB + kLoB + 256;
  static constexpr int kBarB = (8 * kStreamWarps * kStreamStages + 127) / 128 * 128;
  static constexpr int kRingB = kStreamStages * kStreamChunks * kB;  // per warp
  static constexpr int kStatic = kBarB + kStreamWarps * (kRingB + kAhead * 128);
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Compensated FP32 sum (Knuth's TwoSum).
struct PairSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float t = s + v, bb = t - s;
    c += (s - (t - bb)) + (v - bb);
    s = t;
  }
  __device__ __forceinline__ double total() const { return (double)s + (double)c; }
};

struct StreamK {
  const unsigned char* rec;
  const i32* coff;    // first chunk of each slice
  const i32* vout;    // [slices][32]: panel row, ~piece, or kNoRow
  const i32* wstart;  // [units][kStreamWarps + 1]: first slice of each warp
  const i32* ulong0;  // [units + 1]: first long row of each unit
  const i32* long_rows;
  const i32* long_piece0;
  const void* x;
  const i32* xmap;  // forward head: the slice is x[xmap[0..rows)], staged once
  i64 m, rows;
  i64 nunits;
  void* ypan;
  void* partials;
  unsigned* err;
  unsigned wait_limit;  // poll budget of the copy waits
  int aligned;          // x is 16-byte aligned
};

__device__ __forceinline__ df shfl_xor_df(df a, int o) {
  return {__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)};
}

// One lane's 4 entries of a chunk, and a segment's running sum.  FP32: one
// chain of fused multiply-adds per entry of a chunk and chunk of a copy, so
// chains stay at 8; split: exact products p + t, df sums (TwoSum).
// (FP32 error of A^T x, 2M x 200,000 BF16 values, five draws, from the 64-bit
// product: 1.03e-7 with rounded products in chains of 16 and plain sums over a
// long row's segments; 7.8e-8 with this and compensated sums over them, in the
// same time: 231 and 232 us.)
template <int ST> struct ChunkProd {
  float v[4], x[4];
  __device__ __forceinline__ void load(const unsigned char* rec, int lane, const float* xs) {
    using R = StreamRec<ST>;
    const uint2 q = reinterpret_cast<const uint2*>(rec + R::kValB)[lane];
    if constexpr (ST == FVG_F32) {
      const float4 h = reinterpret_cast<const float4*>(rec)[lane];
      v[0] = h.x; v[1] = h.y; v[2] = h.z; v[3] = h.w;
    } else {
      const uint2 h = reinterpret_cast<const uint2*>(rec)[lane];
      v[0] = __uint_as_float(h.x << 16); v[1] = __uint_as_float(h.x & 0xffff0000u);
      v[2] = __uint_as_float(h.y << 16); v[3] = __uint_as_float(h.y & 0xffff0000u);
    }
    x[0] = xs[q.x & 0xffffu];
    x[1] = xs[q.x >> 16];
    x[2] = xs[q.y & 0xffffu];
    x[3] = xs[q.y >> 16];
  }
};
template <> struct ChunkProd<FVG_SPLIT> {
  float p[4], t[4];
  __device__ __forceinline__ void load(const unsigned char* rec, int lane, const float2* xs) {
    using R = StreamRec<FVG_SPLIT>;
    const uint2 q = reinterpret_cast<const uint2*>(rec + R::kValB + R::kLoB)[lane];
    const float4 h = reinterpret_cast<const float4*>(rec)[lane];
    const uint2 l = reinterpret_cast<const uint2*>(rec + R::kValB)[lane];
    const float2 x0 = xs[q.x & 0xffffu], x1 = xs[q.x >> 16], x2 = xs[q.y & 0xffffu], x3 = xs[q.y >> 16];
    df_prod(h.x, __uint_as_float(l.x << 16), x0, p[0], t[0]);
    df_prod(h.y, __uint_as_float(l.x & 0xffff0000u), x1, p[1], t[1]);
    df_prod(h.z, __uint_as_float(l.y << 16), x2, p[2], t[2]);
    df_prod(h.w, __uint_as_float(l.y & 0xffff0000u), x3, p[3], t[3]);
  }
};
template <int ST> struct SegSum {
  float s[kStreamChunks][4] = {};
  __device__ __forceinline__ void add(const ChunkProd<ST>& c, int of) {
#pragma unroll
    for (int k = 0; k < 4; k++) s[of][k] = fmaf(c.v[k], c.x[k], s[of][k]);
  }
  __device__ __forceinline__ float get() const {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < kStreamChunks; q++) t += (s[q][0] + s[q][1]) + (s[q][2] + s[q][3]);
    return t;
  }
};
template <> struct SegSum<FVG_SPLIT> {
  DfAcc a;
  __device__ __forceinline__ void add(const ChunkProd<FVG_SPLIT>& c, int) {
#pragma unroll
    for (int k = 0; k < 4; k++) a.add(c.p[k], c.t[k]);
  }
  __device__ __forceinline__ float2 get() const { return df_pack(a.get()); }
};

// One CTA of kStreamWarps warps per SM takes units (a row panel; for the
// forward head a CTA's whole share of the rows): b, b+G, ...  Per unit the
// vector's slice goes to shared memory (row panels: r's rows of the panel;
// head: w at the head columns, once), then every warp streams its run of
// slices through a ring of kStreamStages bulk copies (cp.async.bulk, an
// mbarrier each, bounded waits) that passes by L1: a panel's slice leaves
// little L1, and loads under way would need lines there.  After a barrier the
// segments of long rows are added in order.  Every sum has a fixed order.
template <int ST>
__global__ void __launch_bounds__(kStreamWarps * 32, 1) k_panel_stream(const StreamK p) {
  using R = StreamRec<ST>;
  using X = typename R::X;
  constexpr int NW = kStreamWarps, NS = kStreamStages, SC = kStreamChunks;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem) + w * NS;
  unsigned char* ring = smem + R::kBarB + w * R::kRingB;
  X* xs = reinterpret_cast<X*>(smem + R::kStatic);
  const X* __restrict__ x = (const X*)p.x;
  X* ypan = (X*)p.ypan;
  X* partials = (X*)p.partials;
  if (lane == 0)
    for (int i = 0; i < NS; i++) mbar_init(bars + i, 1);
  fence_mbar_init();
  if (threadIdx.x == 0) xs[p.rows] = X{};  // the padding's vector entry
  __syncthreads();
  const uint64_t pol = policy_evict_first();
  int is = 0, us = 0;  // ring slots of the next copy and of the next wait
  unsigned phase = 0;  // parity of the next wait's slot
  int flying = 0;      // copies under way
  bool dead = false;
  // kAhead slices' row numbers, copied asynchronously: each lane reads only
  // its own words
  i32* oq = reinterpret_cast<i32*>(smem + R::kBarB + NW * R::kRingB) + w * (kAhead * 32) + lane;
  for (int u = blockIdx.x; u < (int)p.nunits; u += gridDim.x) {
    const int s0 = p.wstart[(i64)u * (NW + 1) + w], s1 = p.wstart[(i64)u * (NW + 1) + w + 1];
    int g = p.coff[s0];  // next chunk to add
    const int ge = p.coff[s1];
    int gi = g;          // next chunk to copy
    // a copy always takes SC records (the records are padded past the last)
    auto issue = [&]() {
      if (gi >= ge || dead) return;
      if (lane == 0) {
        mbar_arrive_expect_tx(bars + is, SC * R::kB);
        bulk_g2s(ring + is * (SC * R::kB), p.rec + (i64)gi * R::kB, SC * R::kB, bars + is, pol);
      }
      gi += SC;
      flying++;
      is = is + 1 == NS ? 0 : is + 1;
    };
#pragma unroll
    for (int i = 0; i < NS; i++) issue();
    const i32* vo = p.vout + lane;
    auto fetch_out = [&](int s) {
      if (s < s1) cp_async4(oq + (s & (kAhead - 1)) * 32, vo + (i64)s * 32);
      cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < kAhead; i++) fetch_out(s0 + i);
    __syncthreads();  // the slice of the unit before is no longer read
    if (p.xmap) {
      if (u == (int)blockIdx.x)
#pragma unroll 4
        for (int i = threadIdx.x; i < (int)p.rows; i += NW * 32) xs[i] = __ldg(x + p.xmap[i]);
    } else {
      const i64 base = (i64)u * p.rows;
      const int nr = (int)min(p.rows, p.m - base);
      constexpr int V = 16 / (int)sizeof(X);
      const int nv = p.aligned ? nr / V : 0;  // rows is a multiple of 4
      const float4* src = reinterpret_cast<const float4*>(x + base);
#pragma unroll 4
      for (int i = threadIdx.x; i < nv; i += NW * 32) reinterpret_cast<float4*>(xs)[i] = __ldg(src + i);
      for (int i = nv * V + threadIdx.x; i < nr; i += NW * 32) xs[i] = __ldg(x + base + i);
    }
    __syncthreads();
    // lane L holds the end of slice win + L, then of win + 32 + L
    int s = s0, win = s0;
    i32 ends = s0 + lane < s1 ? p.coff[s0 + lane + 1] : 0;
    i32 ends2 = s0 + 32 + lane < s1 ? p.coff[s0 + 32 + lane + 1] : 0;
    int ce = __shfl_sync(0xffffffffu, ends, 0);  // end of slice s
    SegSum<ST> sum;
    // writes slice s's sums and moves to the next one
    auto next_slice = [&]() {
      cp_async_wait<kAhead - 1>();
      const i32 o = oq[(s & (kAhead - 1)) * 32];
      fetch_out(s + kAhead);
      const auto r = sum.get();
      sum = SegSum<ST>();
      if (o >= 0) ypan[o] = r;
      else if (o != kNoRow) partials[~o] = r;
      s++;
      if (s - win == 32) {
        win = s;
        ends = ends2;
        ends2 = s + 32 + lane < s1 ? p.coff[s + 32 + lane + 1] : 0;
      }
      ce = __shfl_sync(0xffffffffu, ends, s - win);
    };
    while (g < ge) {
      if (!mbar_wait_bounded(bars + us, phase, p.err, p.wait_limit)) {
        dead = true;
        break;
      }
      // all the copy's entries first (their shared loads overlap), so that
      // the ring slot is free for the next copy before the sums
      const unsigned char* cur = ring + us * (SC * R::kB);
      ChunkProd<ST> c[SC];
#pragma unroll
      for (int k = 0; k < SC; k++) c[k].load(cur + k * R::kB, lane, xs);
      flying--;
      us++;
      if (us == NS) {
        us = 0;
        phase ^= 1u;
      }
      __syncwarp();  // every lane has read the copy
      issue();
#pragma unroll
      for (int k = 0; k < SC; k++) {
        if (g >= ge) break;
        while (g == ce) next_slice();
        sum.add(c[k], k);
        g++;
      }
    }
    if (!dead)
      while (s < s1) next_slice();
    cp_async_wait<0>();
    __syncthreads();
    const int l1 = p.ulong0[u + 1];
    for (int L = p.ulong0[u] + w; L < l1; L += NW) {
      const int c0 = p.long_piece0[L], c1 = p.long_piece0[L + 1];
      if constexpr (ST == FVG_SPLIT) {
        df a = {0.f, 0.f};
        for (int j = c0 + lane; j < c1; j += 32) a = df_add(a, df_unpack(__ldcg(partials + j)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a = df_add(a, shfl_xor_df(a, o));
        if (lane == 0) ypan[p.long_rows[L]] = df_pack(a);
      } else {
        PairSum a;
        for (int j = c0 + lane; j < c1; j += 32) a.add(__ldcg(partials + j));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float v = __shfl_xor_sync(0xffffffffu, a.s, o), r = __shfl_xor_sync(0xffffffffu, a.c, o);
          a.add(v);
          a.c += r;
        }
        if (lane == 0) ypan[p.long_rows[L]] = a.s + a.c;
      }
    }
  }
  // a warp that gave up still drains its copies in flight (default budget)
  for (; flying > 0; flying--) {
    mbar_wait_bounded(bars + us, phase, nullptr, kCopyPolls);
    us++;
    if (us == NS) {
      us = 0;
      phase ^= 1u;
    }
  }
}

// ------------------------------------------------- streamed layout's build
// Segments per panel row, and the rows cut into several (long rows).
__global__ void k_seg_counts(const i32* __restrict__ poff, i64 Q, i64* __restrict__ nv, i64* __restrict__ lng,
                             i64* __restrict__ lpc) {
  PGRID_STRIDE(q, Q) {
    const i32 n = max(1, (((poff[q + 1] - poff[q]) + 3) / 4 + kSegChunks - 1) / kSegChunks);
    nv[q] = n;
    lng[q] = n > 1;
    lpc[q] = n > 1 ? n : 0;
  }
}

// chunks [c0, c1) of segment j of n of a row of `len` entries
__device__ __forceinline__ void seg_chunks(i32 len, i32 j, i32 n, i32& c0, i32& c1) {
  const i64 c = (len + 3) / 4;
  c0 = (i32)(c * j / n);
  c1 = (i32)(c * (j + 1) / n);
}

// sort keys: the panel, then the segments by decreasing chunks
__global__ void k_seg_keys(const i32* __restrict__ poff, const i64* __restrict__ voff, i64 Q, i64 nhot,
                           uint32_t* __restrict__ keys, uint32_t* __restrict__ ids, i32* __restrict__ vq) {
  PGRID_STRIDE(q, Q) {
    const i64 v0 = voff[q];
    const i32 n = (i32)(voff[q + 1] - v0), len = poff[q + 1] - poff[q];
    const uint32_t p = (uint32_t)(q / nhot) << 5;
    for (i32 j = 0; j < n; j++) {
      i32 c0, c1;
      seg_chunks(len, j, n, c0, c1);
      keys[v0 + j] = p | (uint32_t)(kSegChunks - (c1 - c0));
      ids[v0 + j] = (uint32_t)(v0 + j);
      vq[v0 + j] = (i32)q;
    }
  }
}

// out[i] = src[min(i * step, limit)]
__global__ void k_take_every(const i64* __restrict__ src, i64 step, i64 limit, i64 n, i64* __restrict__ out) {
  PGRID_STRIDE(i, n) out[i] = src[min(i * step, limit)];
}

// per (slice, lane): where the segment's sum goes; per segment its slice and
// lane; per slice its chunks (lane 0 holds the longest segment)
__global__ void k_slices(const i32* __restrict__ poff, const i64* __restrict__ voff, const i64* __restrict__ lpc,
                         const uint32_t* __restrict__ ids, const i32* __restrict__ vq, const i64* __restrict__ sbase,
                         const i64* __restrict__ pstart, i64 np, i64 ns, i32* __restrict__ vout,
                         i32* __restrict__ spos, i64* __restrict__ width) {
  PGRID_STRIDE(t, ns * 32) {
    const i64 s = t >> 5;
    i64 a = 0, b = np;  // the panel holding slice s: sbase[a] <= s < sbase[a + 1]
    while (b - a > 1) {
      const i64 mid = (a + b) >> 1;
      if (sbase[mid] <= s) a = mid;
      else b = mid;
    }
    const i64 i = pstart[a] + (s - sbase[a]) * 32 + (t & 31);
    i32 out = kNoRow, c0 = 0, c1 = 0;
    if (i < pstart[a + 1]) {
      const i64 v = ids[i];
      const i32 q = vq[v];
      const i32 n = (i32)(voff[q + 1] - voff[q]), j = (i32)(v - voff[q]), len = poff[q + 1] - poff[q];
      seg_chunks(len, j, n, c0, c1);
      out = n > 1 ? ~(i32)(lpc[q] + j) : q;
      spos[v] = (i32)t;
    }
    vout[t] = out;
    if ((t & 31) == 0) width[s] = c1 - c0;
  }
}

__global__ void k_long_list(const i64* __restrict__ lng, const i64* __restrict__ lpos, const i64* __restrict__ lpc,
                            i64 Q, i32* __restrict__ rows, i32* __restrict__ piece0) {
  PGRID_STRIDE(q, Q)
    if (lng[q]) {
      rows[lpos[q]] = (i32)q;
      piece0[lpos[q]] = (i32)lpc[q];
    }
}

// first slice of each warp's share of a unit: equal chunks + slices
__global__ void k_warp_starts(const i32* __restrict__ coff, const i64* __restrict__ sbase, i64 group, i64 np,
                              i64 nunits, i32* __restrict__ wstart) {
  PGRID_STRIDE(t, nunits * (kStreamWarps + 1)) {
    const i64 u = t / (kStreamWarps + 1), w = t - u * (kStreamWarps + 1);
    const i64 a = sbase[u * group], b = sbase[min((u + 1) * group, np)];
    const i64 c0 = coff[a] + a, c1 = coff[b] + b;
    const i64 target = c0 + (c1 - c0) * w / kStreamWarps;
    i64 lo = a, hi = b;  // first slice whose start costs at least the target
    while (lo < hi) {
      const i64 mid = (lo + hi) >> 1;
      if (coff[mid] + mid < target) lo = mid + 1;
      else hi = mid;
    }
    wstart[t] = (i32)lo;
  }
}

// Records are written straight from the CRS values the layout is made of (A^T
// for row panels, A for the head), so no second copy of the entries is kept or
// needed while a layout is built: first every record as padding, then each
// panel row's entries at their segments' places.  Neighbouring entries of a
// row share a chunk, and the chunks of a panel stay in L2 until all its rows
// are in.
template <int ST>
__global__ void k_blank_records(unsigned char* __restrict__ rec, i64 nrec, unsigned pad) {
  using R = StreamRec<ST>;
  constexpr int kW = R::kB / 16;
  const unsigned pp = pad | (pad << 16);
  PGRID_STRIDE(i, nrec * kW)
    reinterpret_cast<uint4*>(rec)[i] = (i % kW) * 16 >= R::kValB + R::kLoB ? make_uint4(pp, pp, pp, pp) : uint4{};
}

// Entry e (0..3) of a lane's chunk: the value as `ST` stores it (the same
// roundings as the value planes') and its slot.
template <int ST, class T>
__device__ __forceinline__ void put_entry(unsigned char* chunk, int lane, int e, T v, unsigned slot) {
  using R = StreamRec<ST>;
  const int o = lane * 4 + e;
  if constexpr (ST == FVG_BF16) {
    bf16 b;
    if constexpr (std::is_same_v<T, double>) b = __double2bfloat16(v);
    else if constexpr (std::is_same_v<T, float>) b = __float2bfloat16_rn(v);
    else b = v;
    reinterpret_cast<bf16*>(chunk)[o] = b;
  } else {
    float h;
    unsigned short lo = 0;
    if constexpr (std::is_same_v<T, double>) {
      uint32_t hb;
      if (ST == FVG_SPLIT && split_bits((uint64_t)__double_as_longlong(v), &hb, &lo)) {
        h = __uint_as_float(hb);
      } else {
        h = (float)v;
        if (ST == FVG_SPLIT) lo = __bfloat16_as_ushort(__double2bfloat16(isinf(h) ? 0.0 : v - (double)h));
      }
    } else {
      h = (float)v;
    }
    reinterpret_cast<float*>(chunk)[o] = h;
    if (ST == FVG_SPLIT) reinterpret_cast<unsigned short*>(chunk + R::kValB)[o] = lo;
  }
  reinterpret_cast<unsigned short*>(chunk + R::kValB + R::kLoB)[o] = (unsigned short)slot;
}

// where the segments' records are
struct RecAt {
  const i32* coff;  // first chunk of each slice
  const i32* voff;  // first segment of each panel row
  const i32* spos;  // slice * 32 + lane of each segment
  unsigned char* rec;
};

// row panels: 8 lanes per panel row, a segment after the other.  Bound by the
// chain of loads to a row's segments (its start, the segment's place, the
// slice's first chunk, the entries), so four rows share a warp: 4.9e8 split
// entries 6.6 ms, 8.5 with a warp a row.
constexpr int kRecLanes = 8;
template <int ST, class T>
__global__ void k_panel_records(const i32* __restrict__ B, const i32* __restrict__ tidx, const T* __restrict__ tval,
                                i64 nhot, i64 np, i64 rows, const RecAt at) {
  const int sub = threadIdx.x % kRecLanes;
  const i64 Q = np * nhot;  // below 2^31
  for (i64 q = ((i64)blockIdx.x * blockDim.x + threadIdx.x) / kRecLanes; q < Q;
       q += ((i64)gridDim.x * blockDim.x) / kRecLanes) {
    const i32 p = (i32)q / (i32)nhot, h = (i32)q - p * (i32)nhot;
    const i64 s = B[h * (np + 1) + p];
    const i32 len = (i32)(B[h * (np + 1) + p + 1] - s);
    const i32 v0 = at.voff[q], n = at.voff[q + 1] - v0;
    for (i32 j = 0; j < n; j++) {
      i32 c0, c1;
      seg_chunks(len, j, n, c0, c1);
      const i32 pos = at.spos[v0 + j];
      unsigned char* first = at.rec + (i64)at.coff[pos >> 5] * StreamRec<ST>::kB;
      const i32 k0 = 4 * c0 + sub, k1 = min(4 * c1, len);
      constexpr int kRounds = 4 * kSegChunks / kRecLanes;  // a segment's loads under way together
      T v[kRounds];
      i32 row[kRounds];
#pragma unroll
      for (int u = 0; u < kRounds; u++)
        if (k0 + kRecLanes * u < k1) {
          v[u] = tval[s + k0 + kRecLanes * u];
          row[u] = tidx[s + k0 + kRecLanes * u];
        }
#pragma unroll
      for (int u = 0; u < kRounds; u++) {
        const i32 k = k0 + kRecLanes * u;
        if (k < k1)
          put_entry<ST, T>(first + (i64)((k >> 2) - c0) * StreamRec<ST>::kB, pos & 31, k & 3, v[u],
                           (unsigned)(row[u] - p * rows));
      }
    }
  }
}

// forward head: a warp per row of A, its entries in head columns
template <int ST, class T>
__global__ void k_head_records(const i32* __restrict__ off, const i32* __restrict__ idx, const T* __restrict__ val,
                               i64 m, const i32* __restrict__ slot, const i32* __restrict__ poff, const RecAt at) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  PWARP_STRIDE(r, m) {
    const i64 s0 = off[r], e0 = off[r + 1];
    const i32 len = poff[r + 1] - poff[r], v0 = at.voff[r], n = at.voff[r + 1] - v0;
    const i64 c = (len + 3) / 4;
    i32 k0 = 0;
    constexpr int kRounds = 2;  // loads under way together
    for (i64 b = s0; b < e0; b += 32 * kRounds) {
      i32 sl[kRounds];
      T v[kRounds];
#pragma unroll
      for (int u = 0; u < kRounds; u++) {
        const i64 e = b + 32 * u + lane;
        sl[u] = e < e0 ? idx[e] : -1;
        if (e < e0) v[u] = val[e];
      }
#pragma unroll
      for (int u = 0; u < kRounds; u++)
        if (sl[u] >= 0) sl[u] = slot[sl[u]];
#pragma unroll
      for (int u = 0; u < kRounds; u++) {
        const unsigned hb = __ballot_sync(0xffffffffu, sl[u] >= 0);
        if (sl[u] >= 0) {
          const i32 k = k0 + __popc(hb & lt), ck = k >> 2;
          i32 j = 0, c0 = 0, c1;
          if (n > 1) {
            j = (i32)(((i64)(ck + 1) * n - 1) / c);  // the last segment that starts at or before chunk ck
            seg_chunks(len, j, n, c0, c1);
          }
          const i32 pos = at.spos[v0 + j];
          put_entry<ST, T>(at.rec + ((i64)at.coff[pos >> 5] + ck - c0) * StreamRec<ST>::kB, pos & 31, k & 3, v[u],
                           (unsigned)sl[u]);
        }
        k0 += __popc(hb);
      }
    }
  }
}

// g[hot[h]] = sum over panels of ypan[panel*nhot + h] in a fixed order:
// 32 columns per CTA of kSumWarps warps; warp w adds panels w, w + kSumWarps,
// ... in two compensated FP32 sums (GB300's FP64 unit is too narrow for one
// FP64 add per partial; TwoSum, because the partials' signs differ and Kahan's
// form loses the remainder where an addend is larger than the sum), then warp
// 0 adds the warps' sums in FP64, in order.
// Bound by that FP64 tail where the panels are few (2M rows: 152, 25,000
// columns): 7.3 us with 8 warps, 19.6 with 32.
constexpr int kSumWarps = 8;
template <class YT>
__global__ void __launch_bounds__(32 * kSumWarps) k_panel_colsum(const float* __restrict__ ypan,
                                                                 const i32* __restrict__ hot, i64 nhot, i64 np,
                                                                 YT* __restrict__ y) {
  __shared__ double part[kSumWarps][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (i64 h0 = (i64)blockIdx.x * 32; h0 < nhot; h0 += (i64)gridDim.x * 32) {
    const i64 h = h0 + lane;
    PairSum a, b;
    if (h < nhot) {
      constexpr int U = 8;  // loads under way together
      i64 pn = w;
      for (; pn + (U - 1) * kSumWarps < np; pn += U * kSumWarps) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = __ldcs(ypan + (pn + u * kSumWarps) * nhot + h);
#pragma unroll
        for (int u = 0; u < U; u += 2) {
          a.add(v[u]);
          b.add(v[u + 1]);
        }
      }
      float v[U];
#pragma unroll
      for (int u = 0; u < U; u++) v[u] = pn + u * kSumWarps < np ? __ldcs(ypan + (pn + u * kSumWarps) * nhot + h) : 0.f;
#pragma unroll
      for (int u = 0; u < U; u += 2) {
        a.add(v[u]);
        b.add(v[u + 1]);
      }
    }
    part[w][lane] = a.total() + b.total();
    __syncthreads();
    if (w == 0 && h < nhot) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < kSumWarps; q++) s += part[q][lane];
      y[hot[h]] = (YT)s;
    }
    __syncthreads();
  }
}

// g[hot[h]] = sum over panels of the df partials ypan[panel*nhot + h]:
// 32 columns per CTA of 1024 threads, warp w adds panels w, w+32, ...; warp
// 0 adds the 32 warp sums in order; FP64 result.
__global__ void __launch_bounds__(1024) k_panel_colsum_split(const float2* __restrict__ ypan,
                                                             const i32* __restrict__ hot, i64 nhot, i64 np,
                                                             double* __restrict__ y) {
  __shared__ float2 part[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (i64 h0 = (i64)blockIdx.x * 32; h0 < nhot; h0 += (i64)gridDim.x * 32) {
    const i64 h = h0 + lane;
    df a = {0.f, 0.f};
    if (h < nhot)
      for (i64 pn = w; pn < np; pn += 32) a = df_add(a, df_unpack(__ldcs(ypan + pn * nhot + h)));
    part[w][lane] = df_pack(a);
    __syncthreads();
    if (w == 0 && h < nhot) {
      df s = {0.f, 0.f};
#pragma unroll 8
      for (int q = 0; q < 32; q++) s = df_add(s, df_unpack(part[q][lane]));
      y[hot[h]] = df_to_double(s);
    }
    __syncthreads();
  }
}

template <int ST> int stream_smem_bytes(i64 rows) {
  using R = StreamRec<ST>;
  return R::kStatic + (int)((rows + 1) * (i64)sizeof(typename R::X));  // + the padding's entry
}

// Tallest panel (or head) one CTA can stage beside the copy rings, for every
// value storage alike (split values need the most: 8 bytes an entry of the
// slice and the largest records), so that one layout serves all.
i64 panel_rows_cap(fvg_ctx* c) {
  int per_sm = 0, reserved = 0, optin = 0;
  FVG_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c->device));
  FVG_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, c->device));
  FVG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const i64 per_cta = std::min<i64>((i64)per_sm - (i64)reserved, (i64)optin);
  const i64 cap = std::min<i64>((per_cta - StreamRec<FVG_SPLIT>::kStatic) / 8 - 1, 65535);  // slots are uint16
  return cap & ~3ll;
}

void alloc_padded(fvg_ctx* c, DBuf& b, i64 n, int elem) {
  b.alloc((size_t)(n + kPad) * elem, c->stream);
  FVG_CUDA(cudaMemsetAsync((char*)b.p + (size_t)n * elem, 0, (size_t)kPad * elem, c->stream));
}

// Allocates, for n entries, the planes of `dst` / `dlo` that the source holds
// besides its master plane and returns the copy pointers.
SidePlanes side_planes(fvg_ctx* c, const DBuf* src, const DBuf& slo, int master, DBuf* dst, DBuf& dlo, i64 n) {
  SidePlanes sp;
  if (master != FVG_F32 && src[FVG_F32].p) {
    alloc_padded(c, dst[FVG_F32], n, 4);
    sp.s32 = src[FVG_F32].as<float>();
    sp.d32 = dst[FVG_F32].as<float>();
  }
  if (master != FVG_BF16 && src[FVG_BF16].p) {
    alloc_padded(c, dst[FVG_BF16], n, 2);
    sp.s16 = src[FVG_BF16].as<bf16>();
    sp.d16 = dst[FVG_BF16].as<bf16>();
  }
  if (slo.p) {
    alloc_padded(c, dlo, n, 2);
    sp.slo = slo.as<bf16>();
    sp.dlo = dlo.as<bf16>();
  }
  return sp;
}

template <class T>
void fill_cold(fvg_ctx* c, const DevCRS& at, DevPanels& pn, const i64* flag, const i64* coff) {
  const SidePlanes sp = side_planes(c, at.val, at.lo, pn.master, pn.cold.val, pn.cold.lo, pn.cold.nnz);
  k_cold_fill<T><<<grid_n(32 * pn.n), 256, 0, c->stream>>>(at.off.as<i32>(), flag, coff, pn.n, at.idx.as<i32>(),
                                                           at.val[pn.master].as<T>(), pn.cold.idx.as<i32>(),
                                                           pn.cold.val[pn.master].as<T>(), sp);
  check_launch("cold_fill");
  count_launch(c);
}

}  // namespace

// Work items of a CRS cut into chunks of `chunk` rows (a chunk's items, long
// rows and pieces are contiguous, numbered globally), packed on the device:
// counts, their exclusive scans (a few thousand numbers, on the host), then
// the items.
void device_pack(fvg_ctx* c, const i32* off, i64 nrows, i64 chunk, i64 nchunks, int tile, PackOut& o,
                 int lane_work) {
  const i64 np = std::max<i64>(nchunks, 1);
  DBuf cnt, basev;
  cnt.alloc(sizeof(i32) * 3 * np, c->stream);
  if (chunk > kPackRows) fail(FVG_ERR_INTERNAL, "packing chunk too long");
  const unsigned pg = (unsigned)std::min<i64>(np, 1 << 20);  // a CTA per chunk
  k_pack<<<pg, kPackThreads, 0, c->stream>>>(off, nrows, chunk, np, tile, 0, cnt.as<i32>(), nullptr, nullptr,
                                          nullptr, nullptr, nullptr, lane_work);
  check_launch("pack");
  count_launch(c);
  std::vector<i32> hc((size_t)(3 * np));
  o.base.assign((size_t)(3 * (np + 1)), 0);
  FVG_CUDA(cudaMemcpyAsync(hc.data(), cnt.p, sizeof(i32) * 3 * np, cudaMemcpyDeviceToHost, c->stream));
  FVG_CUDA(cudaStreamSynchronize(c->stream));
  i64 tot[3] = {0, 0, 0};
  for (int kind = 0; kind < 3; kind++) {
    for (i64 p = 0; p < np; p++) {
      o.base[(size_t)(kind * (np + 1) + p)] = (i32)tot[kind];
      tot[kind] += hc[(size_t)(kind * np + p)];
    }
    o.base[(size_t)(kind * (np + 1) + np)] = (i32)tot[kind];
  }
  if (tot[0] >= (1ll << 31) - 1 || tot[2] >= (1ll << 31) - 1) fail(FVG_ERR_INTERNAL, "work schedule too large");
  o.nitems = tot[0];
  o.nlong = tot[1];
  o.npieces = tot[2];
  basev.alloc(sizeof(i32) * 3 * (np + 1), c->stream);
  FVG_CUDA(cudaMemcpyAsync(basev.p, o.base.data(), sizeof(i32) * 3 * (np + 1), cudaMemcpyHostToDevice, c->stream));
  o.items.alloc(sizeof(Item) * std::max<i64>(o.nitems, 1), c->stream);
  o.long_rows.alloc(sizeof(i32) * std::max<i64>(o.nlong, 1), c->stream);
  o.long_piece0.alloc(sizeof(i32) * (o.nlong + 1), c->stream);
  DBuf lfirst;
  lfirst.alloc(sizeof(i32) * std::max<i64>(o.nlong, 1), c->stream);
  k_pack<<<pg, kPackThreads, 0, c->stream>>>(off, nrows, chunk, np, tile, 1, nullptr, basev.as<i32>(),
                                          o.items.as<Item>(), o.long_rows.as<i32>(), o.long_piece0.as<i32>(),
                                          lfirst.as<i32>(), lane_work);
  check_launch("pack");
  count_launch(c);
  if (o.nlong > 0) {
    const unsigned lg = (unsigned)std::min<i64>((o.nlong + 7) / 8, 1 << 20);
    k_long_pieces<<<lg, 256, 0, c->stream>>>(off, o.long_rows.as<i32>(), o.long_piece0.as<i32>(), lfirst.as<i32>(),
                                             o.nlong, tile, o.items.as<Item>());
    check_launch("long_pieces");
    count_launch(c);
  }
  const i32 npc = (i32)o.npieces;
  FVG_CUDA(cudaMemcpyAsync(o.long_piece0.as<i32>() + o.nlong, &npc, sizeof(i32), cudaMemcpyHostToDevice, c->stream));
  FVG_CUDA(cudaStreamSynchronize(c->stream));  // host values go out of scope
}

namespace {

// The streamed layout of the panel rows (poff: their entries' offsets); false
// when it would not fit its index types.
bool stream_layout(fvg_ctx* c, DevPanels& pn) {
  cudaStream_t st = c->stream;
  const i64 np = pn.npanels, nhot = pn.nhot, Q = np * nhot;
  const i32* poff = pn.poff.as<i32>();
  DBuf nv, lng, lpcn, voff, lpos, lpc;
  for (DBuf* b : {&nv, &lng, &lpcn}) b->alloc(sizeof(i64) * Q, st);
  for (DBuf* b : {&voff, &lpos, &lpc}) b->alloc(sizeof(i64) * (Q + 1), st);
  k_seg_counts<<<grid_n(Q), 256, 0, st>>>(poff, Q, nv.as<i64>(), lng.as<i64>(), lpcn.as<i64>());
  check_launch("seg_counts");
  scan_i64(c, nv.as<i64>(), voff.as<i64>(), Q);
  scan_i64(c, lng.as<i64>(), lpos.as<i64>(), Q);
  scan_i64(c, lpcn.as<i64>(), lpc.as<i64>(), Q);
  nv.release();
  lpcn.release();
  // per panel: its first segment; per unit: its first long row
  pn.nunits = (np + pn.group - 1) / pn.group;
  DBuf pstart, ul;
  pstart.alloc(sizeof(i64) * (np + 1), st);
  ul.alloc(sizeof(i64) * (pn.nunits + 1), st);
  k_take_every<<<grid_n(np + 1), 256, 0, st>>>(voff.as<i64>(), nhot, Q, np + 1, pstart.as<i64>());
  k_take_every<<<grid_n(pn.nunits + 1), 256, 0, st>>>(lpos.as<i64>(), nhot * pn.group, Q, pn.nunits + 1,
                                                       ul.as<i64>());
  check_launch("take_every");
  std::vector<i64> hp((size_t)np + 1), sb((size_t)np + 1, 0);
  i64 tot[2];
  FVG_CUDA(cudaMemcpyAsync(hp.data(), pstart.p, sizeof(i64) * (np + 1), cudaMemcpyDeviceToHost, st));
  FVG_CUDA(cudaMemcpyAsync(&tot[0], lpos.as<i64>() + Q, sizeof(i64), cudaMemcpyDeviceToHost, st));
  FVG_CUDA(cudaMemcpyAsync(&tot[1], lpc.as<i64>() + Q, sizeof(i64), cudaMemcpyDeviceToHost, st));
  FVG_CUDA(cudaStreamSynchronize(st));
  const i64 V = hp[(size_t)np];
  for (i64 p = 0; p < np; p++) sb[(size_t)p + 1] = sb[(size_t)p] + (hp[(size_t)p + 1] - hp[(size_t)p] + 31) / 32;
  const i64 ns = sb[(size_t)np];
  if (V >= (1ll << 31) - 1 || ns * 32 >= (1ll << 31) - 1) return false;
  pn.nslices = ns;
  pn.nlong = tot[0];
  pn.npieces = tot[1];
  DBuf keys, ids, vq, sbase, width, coff;
  keys.alloc(sizeof(uint32_t) * std::max<i64>(V, 1), st);
  ids.alloc(sizeof(uint32_t) * std::max<i64>(V, 1), st);
  vq.alloc(sizeof(i32) * std::max<i64>(V, 1), st);
  k_seg_keys<<<grid_n(Q), 256, 0, st>>>(poff, voff.as<i64>(), Q, nhot, keys.as<uint32_t>(), ids.as<uint32_t>(),
                                        vq.as<i32>());
  check_launch("seg_keys");
  int bits = 5;
  while ((1ll << (bits - 5)) < np) bits++;
  radix_sort_pairs(c, keys.as<uint32_t>(), ids.as<uint32_t>(), V, bits);
  sbase.alloc(sizeof(i64) * (np + 1), st);
  FVG_CUDA(cudaMemcpyAsync(sbase.p, sb.data(), sizeof(i64) * (np + 1), cudaMemcpyHostToDevice, st));
  pn.vout.alloc(sizeof(i32) * std::max<i64>(ns * 32, 1), st);
  pn.spos.alloc(sizeof(i32) * std::max<i64>(V, 1), st);
  width.alloc(sizeof(i64) * std::max<i64>(ns, 1), st);
  coff.alloc(sizeof(i64) * (ns + 1), st);
  k_slices<<<grid_n(ns * 32), 256, 0, st>>>(poff, voff.as<i64>(), lpc.as<i64>(), ids.as<uint32_t>(), vq.as<i32>(),
                                            sbase.as<i64>(), pstart.as<i64>(), np, ns, pn.vout.as<i32>(),
                                            pn.spos.as<i32>(), width.as<i64>());
  check_launch("slices");
  scan_i64(c, width.as<i64>(), coff.as<i64>(), ns);
  FVG_CUDA(cudaMemcpyAsync(&pn.nchunks, coff.as<i64>() + ns, sizeof(i64), cudaMemcpyDeviceToHost, st));
  FVG_CUDA(cudaStreamSynchronize(st));
  if (pn.nchunks + ns >= (1ll << 31) - 1) return false;
  pn.voff.alloc(sizeof(i32) * (Q + 1), st);
  k_i64_to_i32<<<grid_n(Q + 1), 256, 0, st>>>(voff.as<i64>(), pn.voff.as<i32>(), Q + 1);
  pn.coff.alloc(sizeof(i32) * (ns + 1), st);
  k_i64_to_i32<<<grid_n(ns + 1), 256, 0, st>>>(coff.as<i64>(), pn.coff.as<i32>(), ns + 1);
  pn.ulong0.alloc(sizeof(i32) * (pn.nunits + 1), st);
  k_i64_to_i32<<<grid_n(pn.nunits + 1), 256, 0, st>>>(ul.as<i64>(), pn.ulong0.as<i32>(), pn.nunits + 1);
  pn.long_rows.alloc(sizeof(i32) * std::max<i64>(pn.nlong, 1), st);
  pn.long_piece0.alloc(sizeof(i32) * (pn.nlong + 1), st);
  k_long_list<<<grid_n(Q), 256, 0, st>>>(lng.as<i64>(), lpos.as<i64>(), lpc.as<i64>(), Q, pn.long_rows.as<i32>(),
                                         pn.long_piece0.as<i32>());
  const i32 npc = (i32)pn.npieces;
  FVG_CUDA(cudaMemcpyAsync(pn.long_piece0.as<i32>() + pn.nlong, &npc, sizeof(i32), cudaMemcpyHostToDevice, st));
  pn.wstart.alloc(sizeof(i32) * pn.nunits * (kStreamWarps + 1), st);
  k_warp_starts<<<grid_n(pn.nunits * (kStreamWarps + 1)), 256, 0, st>>>(pn.coff.as<i32>(), sbase.as<i64>(), pn.group,
                                                                        np, pn.nunits, pn.wstart.as<i32>());
  check_launch("stream_layout");
  count_launch(c, 10);
  FVG_CUDA(cudaStreamSynchronize(st));  // host values go out of scope
  return true;
}

// The records of a value storage, from the matrix's own values.
template <int ST> void fill_records(fvg_ctx* c, fvg_matrix* M, DevPanels& pn) {
  ProfScope ps(c, pn.shared ? P_HEAD_BUILD : P_PANEL_BUILD);
  DBuf rec, slot;
  const i64 nrec = pn.nchunks + kStreamChunks;  // a copy may read past the last
  rec.alloc((size_t)nrec * StreamRec<ST>::kB, c->stream);
  k_blank_records<ST><<<grid_n(nrec * (StreamRec<ST>::kB / 16)), 256, 0, c->stream>>>(rec.as<unsigned char>(), nrec,
                                                                                     (unsigned)pn.rows);
  check_launch("blank_records");
  if (pn.shared) {  // column -> slot
    slot.alloc(sizeof(i32) * pn.n, c->stream);
    fill_i32(c, slot.as<i32>(), -1, pn.n);
    k_head_slots<<<grid_n(pn.rows), 256, 0, c->stream>>>(pn.hot_cols.as<uint32_t>(), pn.rows, slot.as<i32>());
    check_launch("head_slots");
    count_launch(c);
  }
  const RecAt at{pn.coff.as<i32>(), pn.voff.as<i32>(), pn.spos.as<i32>(), rec.as<unsigned char>()};
  auto fill = [&](auto tag) {
    using T = decltype(tag);
    if (pn.shared) {
      const DevCRS& a = M->A;
      k_head_records<ST, T><<<grid_n(32 * a.m), 256, 0, c->stream>>>(a.off.as<i32>(), a.idx.as<i32>(),
                                                                    a.val[pn.master].as<T>(), a.m, slot.as<i32>(),
                                                                    pn.poff.as<i32>(), at);
    } else {
      const DevCRS& t = *M->AT;
      k_panel_records<ST, T><<<grid_n(kRecLanes * pn.npanels * pn.nhot), 256, 0, c->stream>>>(
          pn.src.as<i32>(), t.idx.as<i32>(), t.val[pn.master].as<T>(), pn.nhot, pn.npanels, pn.rows, at);
    }
  };
  if (pn.master == FVG_F64) fill(double{});
  else if (pn.master == FVG_F32) fill(float{});
  else fill(bf16{});
  check_launch("fill_records");
  count_launch(c, 2);
  pn.rec[ST] = std::move(rec);
}

// The buffers of the panel rows' and the pieces' sums, each on its own: the
// layout outlives a call in which only the first could be allocated.
void sum_buffers(fvg_ctx* c, DevPanels& pn, DBuf& ypan, DBuf& partials, size_t elem) {
  if (!ypan.p) ypan.alloc(elem * std::max<i64>(pn.npanels * pn.nhot, 1), c->stream);
  if (!partials.p) partials.alloc(elem * std::max<i64>(pn.npieces, 1), c->stream);
}

// ypan (and the long rows' partials) of the layout for a vector x.
template <int ST> void launch_stream(fvg_ctx* c, DevPanels& pn, const void* x, void* ypan, void* partials) {
  if (!pn.rec[ST].p || !ypan || !partials) fail(FVG_ERR_INTERNAL, "a panel layout without its records or sums");
  auto kfn = k_panel_stream<ST>;
  static std::mutex mu;  // contexts of different host threads launch concurrently
  static std::vector<int> attr_set;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (std::find(attr_set.begin(), attr_set.end(), c->device) == attr_set.end()) {
      int optin = 0;
      FVG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
      FVG_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
      attr_set.push_back(c->device);
    }
  }
  StreamK k;
  k.rec = pn.rec[ST].as<unsigned char>();
  k.coff = pn.coff.as<i32>();
  k.vout = pn.vout.as<i32>();
  k.wstart = pn.wstart.as<i32>();
  k.ulong0 = pn.ulong0.as<i32>();
  k.long_rows = pn.long_rows.as<i32>();
  k.long_piece0 = pn.long_piece0.as<i32>();
  k.x = x;
  k.xmap = pn.shared ? pn.hot_cols.as<i32>() : nullptr;
  k.m = pn.m;
  k.rows = pn.rows;
  k.nunits = pn.nunits;
  k.ypan = ypan;
  k.partials = partials;
  k.err = c->dev_err;
  k.wait_limit = copy_polls(c);
  k.aligned = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) ? 1 : 0;
  const int grid = (int)std::max<i64>(1, std::min<i64>(pn.nunits, c->num_sms));
  kfn<<<grid, kStreamWarps * 32, stream_smem_bytes<ST>(pn.rows), c->stream>>>(k);
  check_launch("k_panel_stream");
  count_launch(c);
}

// Builds the layout from the transposed CRS; null when it would not pay
// (too few panels or too little of the matrix in hot columns) or does not fit
// its index types.
std::unique_ptr<DevPanels> panel_build(fvg_ctx* c, const DevCRS& at, int master, i64 force_rows, double min_pp) {
  ProfScope ps(c, P_PANEL_BUILD);
  const i64 m = at.n, n = at.m, nnz = at.nnz;
  const bool forced = force_rows > 0;
  if (m <= 0 || n <= 0 || nnz <= 0) return nullptr;
  const i64 cap = panel_rows_cap(c);
  i64 rows;
  if (forced) {
    if (force_rows % 4 != 0 || force_rows > cap)
      fail(FVG_ERR_INVALID_ARG, "panel rows must be a multiple of 4 and at most " + std::to_string(cap));
    rows = force_rows;
  } else {
    if (m < kPanelMinMatrix) return nullptr;  // too few panels to pay for the split
    // the fewest whole rounds over the SMs whose panels fit in shared memory
    // (the tallest panels: the most columns count as hot); one round of at
    // least kPanelMinRows rows on smaller matrices
    const i64 grid = c->num_sms, rounds = (m + cap * grid - 1) / (cap * grid);
    rows = std::min<i64>(cap, std::max<i64>(kPanelMinRows, ((m + rounds * grid - 1) / (rounds * grid) + 3) & ~3ll));
  }
  const double mpp = min_pp > 0 ? min_pp : kPanelMinAuto;
  auto pn = std::make_unique<DevPanels>();
  pn->m = m;
  pn->n = n;
  pn->rows = rows;
  pn->npanels = (m + rows - 1) / rows;
  pn->min_per_panel = mpp;
  pn->master = master;
  const i64 np = pn->npanels;
  const i64 thresh = std::max<i64>(1, (i64)std::ceil(mpp * (double)np));
  // hot columns
  DBuf flag, pos;
  flag.alloc(sizeof(i64) * n, c->stream);
  pos.alloc(sizeof(i64) * (n + 1), c->stream);
  k_hot_flags<<<grid_n(n), 256, 0, c->stream>>>(at.off.as<i32>(), n, thresh, flag.as<i64>());
  check_launch("hot_flags");
  count_launch(c);
  scan_i64(c, flag.as<i64>(), pos.as<i64>(), n);
  i64 nhot = 0;
  FVG_CUDA(cudaMemcpyAsync(&nhot, pos.as<i64>() + n, sizeof(i64), cudaMemcpyDeviceToHost, c->stream));
  FVG_CUDA(cudaStreamSynchronize(c->stream));
  if (nhot == 0 || np * nhot >= (1ll << 31) - 1 || np >= (1ll << 26)) return nullptr;
  pn->nhot = nhot;
  pn->hot_cols.alloc(sizeof(i32) * nhot, c->stream);
  k_hot_list<<<grid_n(n), 256, 0, c->stream>>>(flag.as<i64>(), pos.as<i64>(), n, pn->hot_cols.as<i32>());
  check_launch("hot_list");
  count_launch(c);
  // per (panel, hot column) ranges and their offsets
  DBuf len, poff64;
  pn->src.alloc(sizeof(i32) * nhot * (np + 1), c->stream);
  i32* const B = pn->src.as<i32>();
  k_panel_bounds<<<grid_n(nhot * (np + 1)), 256, 0, c->stream>>>(at.off.as<i32>(), at.idx.as<i32>(),
                                                                  pn->hot_cols.as<i32>(), nhot, np, rows, B);
  check_launch("panel_bounds");
  const i64 Q = np * nhot;
  len.alloc(sizeof(i64) * Q, c->stream);
  poff64.alloc(sizeof(i64) * (Q + 1), c->stream);
  k_panel_lens<<<grid_n(Q), 256, 0, c->stream>>>(B, nhot, np, len.as<i64>());
  check_launch("panel_lens");
  count_launch(c, 2);
  scan_i64(c, len.as<i64>(), poff64.as<i64>(), Q);
  i64 E = 0;
  FVG_CUDA(cudaMemcpyAsync(&E, poff64.as<i64>() + Q, sizeof(i64), cudaMemcpyDeviceToHost, c->stream));
  FVG_CUDA(cudaStreamSynchronize(c->stream));
  if (!forced && (double)E < 0.25 * (double)nnz) return nullptr;  // mostly cold: the plain path
  pn->E = E;
  pn->poff.alloc(sizeof(i32) * (Q + 1), c->stream);
  k_i64_to_i32<<<grid_n(Q + 1), 256, 0, c->stream>>>(poff64.as<i64>(), pn->poff.as<i32>(), Q + 1);
  check_launch("poff");
  count_launch(c);
  len.release();
  poff64.release();
  // cold columns: A^T with the hot rows emptied
  DevCRS& cold = pn->cold;
  cold.m = n;
  cold.n = m;
  DBuf clen, coff64;
  clen.alloc(sizeof(i64) * n, c->stream);
  coff64.alloc(sizeof(i64) * (n + 1), c->stream);
  k_cold_lens<<<grid_n(n), 256, 0, c->stream>>>(at.off.as<i32>(), flag.as<i64>(), n, clen.as<i64>());
  check_launch("cold_lens");
  count_launch(c);
  scan_i64(c, clen.as<i64>(), coff64.as<i64>(), n);
  FVG_CUDA(cudaMemcpyAsync(&cold.nnz, coff64.as<i64>() + n, sizeof(i64), cudaMemcpyDeviceToHost, c->stream));
  FVG_CUDA(cudaStreamSynchronize(c->stream));
  cold.off.alloc(sizeof(i32) * (n + 1), c->stream);
  k_i64_to_i32<<<grid_n(n + 1), 256, 0, c->stream>>>(coff64.as<i64>(), cold.off.as<i32>(), n + 1);
  check_launch("cold_off");
  count_launch(c);
  alloc_padded(c, cold.idx, cold.nnz, 4);
  alloc_padded(c, cold.val[master], cold.nnz, dtype_size(master));
  if (master == FVG_F64) fill_cold<double>(c, at, *pn, flag.as<i64>(), coff64.as<i64>());
  else if (master == FVG_F32) fill_cold<float>(c, at, *pn, flag.as<i64>(), coff64.as<i64>());
  else fill_cold<bf16>(c, at, *pn, flag.as<i64>(), coff64.as<i64>());
  cold.max_row = 0;  // not used by the product
  if (!stream_layout(c, *pn)) return nullptr;
  pn->poff.release();  // the records are filled by src
  FVG_CUDA(cudaStreamSynchronize(c->stream));  // host vectors go out of scope
  return pn;
}

// The forward head of A: the H most frequent columns (ties: lower column
// first), H at most what one CTA stages beside the staging buffers.  Null
// when it would not pay (small matrices, or the head holding less than half
// of the entries) unless forced (force_cols > 0).
std::unique_ptr<DevPanels> head_build(fvg_ctx* c, const DevCRS& a, const DevCRS& at, int master, i64 force_cols) {
  ProfScope ps(c, P_HEAD_BUILD);
  const i64 m = a.m, n = a.n, nnz = a.nnz;
  const bool forced = force_cols > 0;
  if (m <= 0 || n <= 0 || nnz <= 0) return nullptr;
  const i64 cap = panel_rows_cap(c);
  if (forced && force_cols > cap)
    fail(FVG_ERR_INVALID_ARG, "head columns must be at most " + std::to_string(cap));
  const i64 grid = c->num_sms;  // one CTA (one stretch of rows) per SM
  if (!forced && m < kHeadMinPerSm * grid) return nullptr;
  const i64 H = std::min<i64>(n, forced ? force_cols : cap);
  // the H largest column counts (from the transposed offsets), on the
  // device: a stable sort of the columns by decreasing count (ties keep
  // column order), the first H take slots 0..H-1
  DBuf keys, cols, dslot;
  keys.alloc(sizeof(uint32_t) * n, c->stream);
  cols.alloc(sizeof(uint32_t) * n, c->stream);
  dslot.alloc(sizeof(i32) * n, c->stream);
  k_head_keys<<<grid_n(n), 256, 0, c->stream>>>(at.off.as<i32>(), n, keys.as<uint32_t>(), cols.as<uint32_t>());
  check_launch("head_keys");
  count_launch(c);
  radix_sort_pairs(c, keys.as<uint32_t>(), cols.as<uint32_t>(), n, 31);
  fill_i32(c, dslot.as<i32>(), -1, n);
  k_head_slots<<<grid_n(H), 256, 0, c->stream>>>(cols.as<uint32_t>(), H, dslot.as<i32>());
  check_launch("head_slots");
  count_launch(c);
  auto hd = std::make_unique<DevPanels>();
  hd->shared = true;
  hd->master = master;
  hd->m = H;  // the staged slice: w at the head columns (slot order)
  hd->n = n;
  hd->rows = H;
  // stretches of at most ~4096 rows, a whole number of them per CTA: their
  // segments are sorted by length stretch by stretch, so that the sums of
  // neighbouring rows are written close together
  const i64 per_cta = std::max<i64>(1, (m + grid * 4096 - 1) / (grid * 4096));
  hd->nhot = (m + grid * per_cta - 1) / (grid * per_cta);  // rows per stretch
  hd->npanels = (m + hd->nhot - 1) / hd->nhot;
  const i64 np = hd->npanels, chunk = hd->nhot, Q = np * chunk;
  hd->hot_cols.alloc(sizeof(i32) * std::max<i64>(H, 1), c->stream);
  FVG_CUDA(cudaMemcpyAsync(hd->hot_cols.p, cols.p, sizeof(i32) * H, cudaMemcpyDeviceToDevice, c->stream));
  DBuf hcnt, tcnt, hoff, tof;
  hcnt.alloc(sizeof(i64) * m, c->stream);
  tcnt.alloc(sizeof(i64) * m, c->stream);
  hoff.alloc(sizeof(i64) * (m + 1), c->stream);
  tof.alloc(sizeof(i64) * (m + 1), c->stream);
  k_head_counts<<<grid_n(32 * m), 256, 0, c->stream>>>(a.off.as<i32>(), a.idx.as<i32>(), m, dslot.as<i32>(),
                                                       hcnt.as<i64>(), tcnt.as<i64>());
  check_launch("head_counts");
  count_launch(c);
  scan_i64(c, hcnt.as<i64>(), hoff.as<i64>(), m);
  scan_i64(c, tcnt.as<i64>(), tof.as<i64>(), m);
  i64 tot[2];
  FVG_CUDA(cudaMemcpyAsync(&tot[0], hoff.as<i64>() + m, sizeof(i64), cudaMemcpyDeviceToHost, c->stream));
  FVG_CUDA(cudaMemcpyAsync(&tot[1], tof.as<i64>() + m, sizeof(i64), cudaMemcpyDeviceToHost, c->stream));
  FVG_CUDA(cudaStreamSynchronize(c->stream));
  if (!forced && (double)tot[0] < 0.5 * (double)nnz) return nullptr;  // most entries outside the head
  hd->E = tot[0];
  hd->poff.alloc(sizeof(i32) * (Q + 1), c->stream);
  k_head_off<<<grid_n(Q + 1), 256, 0, c->stream>>>(hoff.as<i64>(), m, Q, hd->poff.as<i32>());
  check_launch("head_off");
  count_launch(c);
  DevCRS& tail = hd->cold;
  tail.m = m;
  tail.n = n;
  tail.nnz = tot[1];
  tail.off.alloc(sizeof(i32) * (m + 1), c->stream);
  k_i64_to_i32<<<grid_n(m + 1), 256, 0, c->stream>>>(tof.as<i64>(), tail.off.as<i32>(), m + 1);
  check_launch("tail_off");
  count_launch(c);
  alloc_padded(c, tail.idx, tail.nnz, 4);
  alloc_padded(c, tail.val[master], tail.nnz, dtype_size(master));
  const SidePlanes spt = side_planes(c, a.val, a.lo, master, tail.val, tail.lo, tail.nnz);
  auto fill = [&](auto tag) {
    using T = decltype(tag);
    k_tail_fill<T><<<grid_n(32 * m), 256, 0, c->stream>>>(a.off.as<i32>(), a.idx.as<i32>(), a.val[master].as<T>(), m,
                                                         dslot.as<i32>(), tof.as<i64>(), tail.idx.as<i32>(),
                                                         tail.val[master].as<T>(), spt);
    check_launch("tail_fill");
    count_launch(c);
  };
  if (master == FVG_F64) fill(double{});
  else if (master == FVG_F32) fill(float{});
  else fill(bf16{});
  tail.max_row = 0;
  hd->group = (np + grid - 1) / grid;  // a CTA's whole share of the stretches
  if (!stream_layout(c, *hd)) return nullptr;
  FVG_CUDA(cudaStreamSynchronize(c->stream));  // host vectors go out of scope
  return hd;
}

}  // namespace

DevPanels* panels_for(fvg_ctx* c, fvg_matrix* M) {
  if (M->panel_rows == 0) return nullptr;
  if (M->pan) return M->pan.get();
  if (M->pan_tried) return nullptr;
  transpose_of(c, M);
  // a forced layout that cannot be built throws here, on every call
  std::unique_ptr<DevPanels> pn = panel_build(c, *M->AT, M->master, M->panel_rows, M->panel_min);
  M->pan_tried = true;
  M->pan = std::move(pn);
  return M->pan.get();
}

void panel_ensure_plane(fvg_ctx* c, fvg_matrix* M, DevPanels& pn, int dt) {
  if (!pn.rec[dt].p) {
    if (dt == FVG_F32) fill_records<FVG_F32>(c, M, pn);
    else fill_records<FVG_BF16>(c, M, pn);
  }
  sum_buffers(c, pn, pn.ypan, pn.partials, sizeof(float));
  crs_ensure_plane(c, pn.cold, dt, pn.master);
  crs_sched(c, pn.cold, kWarpTile);  // the cold product's work items
}

i64 panel_scratch_bytes(fvg_ctx* c, DevPanels& pn, int storage) { return crs_pass_scratch_bytes(c, pn.cold, storage); }

void panel_trans_mv(fvg_ctx* c, DevPanels& pn, int storage, const float* r, int y_dt, void* y, void* scratch,
                    int prof_key) {
  if (storage == FVG_F64) fail(FVG_ERR_INTERNAL, "the panel product runs on FP32 or BF16 values");
  if (y_dt != FVG_F64 && y_dt != FVG_F32) fail(FVG_ERR_INTERNAL, "panel product output must be FP64 or FP32");
  ProfScope pr(c, prof_key);
  // cold columns (and zeros for the hot ones) by the transposed CRS kernel
  crs_pass(c, pn.cold, storage, FVG_F32, r, y_dt, y, EPI_STORE, nullptr, scratch, P_NKEYS);
  if (storage == FVG_F32) launch_stream<FVG_F32>(c, pn, r, pn.ypan.p, pn.partials.p);
  else launch_stream<FVG_BF16>(c, pn, r, pn.ypan.p, pn.partials.p);
  const unsigned cg = (unsigned)std::max<i64>(1, std::min<i64>((pn.nhot + 31) / 32, 8 * c->num_sms));
  const int ct = 32 * kSumWarps;
  if (y_dt == FVG_F64)
    k_panel_colsum<double><<<cg, ct, 0, c->stream>>>(pn.ypan.as<float>(), pn.hot_cols.as<i32>(), pn.nhot, pn.npanels,
                                                     (double*)y);
  else
    k_panel_colsum<float><<<cg, ct, 0, c->stream>>>(pn.ypan.as<float>(), pn.hot_cols.as<i32>(), pn.nhot, pn.npanels,
                                                    (float*)y);
  check_launch("k_panel_colsum");
  count_launch(c);
}

}  // namespace fvg

namespace fvg {

DevPanels* head_for(fvg_ctx* c, fvg_matrix* M) {
  if (M->head_cols == 0) return nullptr;
  if (M->head) return M->head.get();
  if (M->head_tried) return nullptr;
  transpose_of(c, M);
  std::unique_ptr<DevPanels> hd = head_build(c, M->A, *M->AT, M->master, M->head_cols);
  M->head_tried = true;
  M->head = std::move(hd);
  return M->head.get();
}

i64 head_scratch_bytes(fvg_ctx* c, DevPanels& hd, int storage) { return crs_pass_scratch_bytes(c, hd.cold, storage); }

void head_logreg_pass(fvg_ctx* c, DevPanels& hd, int storage, const float* w, const LogregEpi& lr, void* scratch,
                      int prof_key) {
  if (storage == FVG_F64) fail(FVG_ERR_INTERNAL, "the head pass runs on FP32 or BF16 values");
  ProfScope pr(c, prof_key);
  if (storage == FVG_F32) launch_stream<FVG_F32>(c, hd, w, hd.ypan.p, hd.partials.p);
  else launch_stream<FVG_BF16>(c, hd, w, hd.ypan.p, hd.partials.p);
  LogregEpi t = lr;
  t.ybase = hd.ypan.as<float>();
  crs_pass(c, hd.cold, storage, FVG_F32, w, FVG_F32, nullptr, EPI_LOGREG, &t, scratch, P_NKEYS);
}

}  // namespace fvg

// ------------------------------------------------------------ split storage
namespace fvg {

void panel_ensure_split(fvg_ctx* c, fvg_matrix* M, DevPanels& pn) {
  if (!pn.rec[FVG_SPLIT].p) fill_records<FVG_SPLIT>(c, M, pn);
  crs_ensure_split(c, pn.cold, pn.master);
  sum_buffers(c, pn, pn.ypan2, pn.partials2, sizeof(float2));
}

i64 panel_split_scratch_bytes(fvg_ctx* c, DevPanels& pn, bool y_df) {
  return crs_split_scratch_bytes(c, pn.cold, y_df);
}

void panel_trans_mv_split(fvg_ctx* c, DevPanels& pn, const void* r, double* y, void* scratch) {
  // cold columns (and zeros for the hot ones) by the transposed CRS kernel
  crs_pass_split(c, pn.cold, r, false, y, scratch, P_NKEYS);
  launch_stream<FVG_SPLIT>(c, pn, r, pn.ypan2.p, pn.partials2.p);
  const unsigned cg = (unsigned)std::max<i64>(1, std::min<i64>((pn.nhot + 31) / 32, 2 * c->num_sms));
  k_panel_colsum_split<<<cg, 1024, 0, c->stream>>>(pn.ypan2.as<float2>(), pn.hot_cols.as<i32>(), pn.nhot,
                                                    pn.npanels, y);
  check_launch("k_panel_colsum_split");
  count_launch(c);
}

void head_pass_split(fvg_ctx* c, DevPanels& hd, const void* w, void* wtx, void* scratch) {
  launch_stream<FVG_SPLIT>(c, hd, w, hd.ypan2.p, hd.partials2.p);
  crs_pass_split(c, hd.cold, w, true, wtx, scratch, P_NKEYS);
}

}  // namespace fvg
