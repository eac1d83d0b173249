// Multi-vector CRS products: Y = A X for a block of up to 128 columns of a
// row-major X (crs_matrix_spmm_impl, crs_matrix.hpp:2036-2050), with
// optional fused epilogues:
//  * logistic (batched binary training): R = dloss(A W + b) * sw per (row,
//    model) and per-model loss / bias sums (gradient.hpp:15-53);
//  * softmax (multinomial training): P = (softmax(A W + b) - onehot(label))
//    * sw per row (softmax_gradient_descent.hpp:140-235).
//
// The kernel walks the same warp work items as the CRS SpMV (tiles of short
// rows, pieces of long rows, at most 512 nonzeros each).  For every nonzero
// the warp reads one row of X: lane L takes columns L, L+32, ... (CPL columns
// per lane), so a row of X is read with coalesced 128-byte accesses.  Column
// ids and values are loaded 32 at a time, one per lane, and broadcast with
// shuffles.  Pieces of long rows leave 32*CPL partial sums each; the
// finalize kernel adds them in piece order.  Loss and bias sums of the
// logistic epilogue are compensated per lane, then combined per CTA and
// across CTAs in a fixed order (deterministic).
#include <type_traits>

#include "device_common.cuh"

namespace fvg {

constexpr int kSpmmMaxCols = 128;  // columns per launch (four per lane)
constexpr int EPI_SOFTMAX = 2;

struct SpmmK {
  const i32* off;
  const i32* idx;
  const void* val;
  const Item* items;
  i64 nitems;
  const void* X;  // first column of the block; row stride ldx
  i64 ldx;
  int kb;         // columns in this block
  void* Y;        // EPI_STORE output, row stride ldy
  i64 ldy;
  void* partials;  // [npieces][32*CPL] accumulator type
  // epilogues
  const double* label;  // logistic: +-1; softmax: class id
  const double* sw;
  const float* label_f;
  const float* sw_f;
  int icpt;
  const double* bias;  // [kb] intercepts
  void* R;             // epilogue output (accumulator type), row stride ldr
  i64 ldr;
  double* cta_part;  // logistic: [grid][64][2] loss, bias
  int loss;          // GLM loss kind of the per-model epilogue
  double eps;
  // Stacked datasets (logistic epilogue): rows [seg_row[d], seg_row[d+1])
  // belong to dataset d, whose intercepts sit at bias + d * ldb.  Every warp
  // leaves one loss / bias partial per dataset in seg_part[d][warp] (zero
  // for the datasets it saw no row of); nseg = 0: one dataset, per-CTA
  // partials in cta_part.
  const i32* seg_row;
  int nseg;
  i64 ldb;
  double* seg_part;
  const int* gate;  // the launch does nothing while *gate == 0 (null: always runs)
  // Column masks of stacked datasets (null: every column): bit c of
  // mask[d * mstride + mword] set = column c of dataset d is computed;
  // masked columns are neither gathered nor written (their outputs keep
  // what they held) and their loss / bias sums are left out.
  const unsigned long long* mask;
  i64 mstride;
  int mword;
};

__device__ __forceinline__ unsigned long long mask_of(const SpmmK& p, int d) {
  return p.mask ? __ldcg(p.mask + (i64)d * p.mstride + p.mword) : ~0ull;
}
// column c (< 64 whenever a mask is given) is computed under mask word mw;
// all-ones = no mask
__device__ __forceinline__ bool col_on(unsigned long long mw, int c) {
  return mw == ~0ull || (c < 64 && ((mw >> c) & 1ull));
}
// any of the n columns c .. c + n - 1
__device__ __forceinline__ bool cols_on(unsigned long long mw, int c, int n) {
  return mw == ~0ull || (c < 64 && ((mw >> c) & ((1ull << n) - 1)) != 0);
}

__device__ __forceinline__ bool gated_off(const int* gate) { return gate && __ldcg(gate) == 0; }

// Lane layouts of the block's columns.  Strided (VEC = false): lane L owns
// columns L, L+32, ...; every load is one element.  Packed (VEC = true):
// lane L owns columns CPL*L .. CPL*L+CPL-1 and reads / writes them with one
// vector access (needs ldx, the output stride and kb to be multiples of CPL
// and CPL-aligned bases).  Each column's sum runs over the nonzeros in the
// same order in both layouts; only the softmax denominator's lane partials
// group the classes differently.
template <bool VEC, int CPL> __device__ __forceinline__ int colof(int lane, int q) {
  return VEC ? lane * CPL + q : lane + 32 * q;
}

// CPL consecutive elements at an aligned address
template <class XT, int CPL> struct VecLd;
template <int CPL> struct VecLd<float, CPL> {
  static __device__ __forceinline__ void ld(const float* x, float (&o)[CPL]) {
    if constexpr (CPL == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(x));
      o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else if constexpr (CPL == 2) {
      const float2 v = __ldg(reinterpret_cast<const float2*>(x));
      o[0] = v.x; o[1] = v.y;
    } else {
      o[0] = __ldg(x);
    }
  }
};
template <int CPL> struct VecLd<double, CPL> {
  static __device__ __forceinline__ void ld(const double* x, double (&o)[CPL]) {
#pragma unroll
    for (int h = 0; h < CPL; h += 2) {
      if constexpr (CPL >= 2) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(x + h));
        o[h] = v.x; o[h + 1] = v.y;
      } else {
        o[0] = __ldg(x);
      }
    }
  }
};

// CPL consecutive elements stored at an aligned address
template <class T, int CPL> __device__ __forceinline__ void vec_st(T* y, const T (&v)[CPL]) {
  if constexpr (sizeof(T) == 4 && CPL == 4) {
    *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (sizeof(T) == 4 && CPL == 2) {
    *reinterpret_cast<float2*>(y) = make_float2(v[0], v[1]);
  } else if constexpr (sizeof(T) == 8 && CPL >= 2) {
#pragma unroll
    for (int h = 0; h < CPL; h += 2) *reinterpret_cast<double2*>(y + h) = make_double2(v[h], v[h + 1]);
  } else {
#pragma unroll
    for (int q = 0; q < CPL; q++) y[q] = v[q];
  }
}

template <class VT, class XT, class AT, int CPL, bool VEC>
__device__ __forceinline__ void row_dot(const SpmmK& p, i32 e0, i32 e1, int lane, AT (&a)[CPL]) {
  const XT* X = (const XT*)p.X;
  const VT* val = (const VT*)p.val;
#pragma unroll
  for (int q = 0; q < CPL; q++) a[q] = 0;
  const bool mine = !VEC || lane * CPL < p.kb;
  for (i32 e = e0; e < e1; e += 32) {
    const int cnt = min(32, e1 - e);
    i32 mi = 0;
    AT mv = 0;
    if (lane < cnt) {
      mi = __ldcs(p.idx + e + lane);
      mv = ld_val<VT, AT>(val + e + lane);
    }
#pragma unroll 4
    for (int t = 0; t < cnt; t++) {
      const i32 col = __shfl_sync(0xffffffffu, mi, t);
      const AT v = __shfl_sync(0xffffffffu, mv, t);
      if constexpr (VEC) {
        if (mine) {
          XT x[CPL];
          VecLd<XT, CPL>::ld(X + (long long)col * (int)p.ldx + lane * CPL, x);
#pragma unroll
          for (int q = 0; q < CPL; q++) a[q] += v * (AT)x[q];
        }
      } else {
        const XT* xr = X + (long long)col * (int)p.ldx + lane;
#pragma unroll
        for (int q = 0; q < CPL; q++)
          if (lane + 32 * q < p.kb) a[q] += v * (AT)__ldg(xr + 32 * q);
      }
    }
  }
}

template <class AT> __device__ __forceinline__ AT exp_acc(AT x);
template <> __device__ __forceinline__ double exp_acc<double>(double x) { return exp(x); }
template <> __device__ __forceinline__ float exp_acc<float>(float x) { return expf(x); }
template <class AT> __device__ __forceinline__ AT log_acc(AT x);
template <> __device__ __forceinline__ double log_acc<double>(double x) { return log(x); }
template <> __device__ __forceinline__ float log_acc<float>(float x) { return logf(x); }

template <class AT, class YT, int EPI, int CPL, bool VEC, class S>
__device__ __forceinline__ void spmm_epi(const SpmmK& p, i32 row, const AT (&a)[CPL], const AT (&b)[CPL], int lane,
                                         S (&ls)[CPL], S (&bs)[CPL], unsigned long long mw = ~0ull) {
#define ON(q) (colof<VEC, CPL>(lane, q) < p.kb && col_on(mw, colof<VEC, CPL>(lane, q)))
  if (EPI == EPI_STORE) {
    YT* y = (YT*)p.Y + (i64)row * p.ldy;
    if constexpr (VEC) {
      if (mw != ~0ull) {
#pragma unroll
        for (int q = 0; q < CPL; q++)
          if (ON(q)) y[colof<VEC, CPL>(lane, q)] = (YT)a[q];
      } else if (lane * CPL < p.kb) {
        YT o[CPL];
#pragma unroll
        for (int q = 0; q < CPL; q++) o[q] = (YT)a[q];
        vec_st<YT, CPL>(y + lane * CPL, o);
      }
    } else {
#pragma unroll
      for (int q = 0; q < CPL; q++)
        if (ON(q)) y[colof<VEC, CPL>(lane, q)] = (YT)a[q];
    }
    return;
  }
  // softmax without labels: the probability matrix alone (compute_probability_matrix)
  const bool has_label = (sizeof(AT) == 8) ? p.label != nullptr : p.label_f != nullptr;
  AT lab = 0, w = 1;
  bool has_sw = false;
  if (has_label) {
    if constexpr (sizeof(AT) == 8) {
      lab = p.label[row];
      has_sw = p.sw != nullptr;
      if (has_sw) w = p.sw[row];
    } else {
      lab = p.label_f[row];
      has_sw = p.sw_f != nullptr;
      if (has_sw) w = p.sw_f[row];
    }
  }
  AT* r = (AT*)p.R + (i64)row * p.ldr;
  AT out[CPL];
  if (EPI == EPI_LOGREG) {
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      out[q] = 0;
      if (!ON(q)) continue;
      AT loss, d;
      glm_row<AT>(p.loss, (AT)p.eps, a[q] + b[q], lab, loss, d);
      if (has_sw) d = d * w;
      out[q] = d;
      ls[q].add(loss);
      bs[q].add(d);
    }
  } else {  // EPI_SOFTMAX: compute_exp_matrix, compute_softmax_probability, compute_error_inplace
    AT z[CPL], mx = -INFINITY;
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      z[q] = a[q] + b[q];
      if (ON(q)) mx = fmax(mx, z[q]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    // the label's margin z_label - max, for the cross-entropy
    AT zy = 0;
    if (has_label)
#pragma unroll
      for (int q = 0; q < CPL; q++)
        if (ON(q) && lab == (AT)colof<VEC, CPL>(lane, q)) zy = z[q] - mx;
    AT sum = 0;
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      z[q] = ON(q) ? exp_acc<AT>(z[q] - mx) : (AT)0;
      sum += z[q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    // cross-entropy -log p[label] = log(sum) - (z_label - max), unweighted,
    // into lane 0's first partial (the L-BFGS line search's loss)
    if (has_label && p.cta_part) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) zy += __shfl_xor_sync(0xffffffffu, zy, o);
      if (lane == 0) ls[0].add(log_acc<AT>(sum) - zy);
    }
    const AT inv = (AT)1 / sum;
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      AT pr = inv * z[q];
      if (has_label) {
        pr -= (lab == (AT)colof<VEC, CPL>(lane, q)) ? (AT)1 : (AT)0;
        if (has_sw) pr *= w;
      }
      out[q] = pr;
    }
  }
  if constexpr (VEC) {
    if (lane * CPL < p.kb) vec_st<AT, CPL>(r + lane * CPL, out);
  } else {
#pragma unroll
    for (int q = 0; q < CPL; q++)
      if (ON(q)) r[colof<VEC, CPL>(lane, q)] = out[q];
  }
#undef ON
}

template <class VT, class XT, class AT, class YT, int EPI, int CPL, bool VEC>
__global__ void __launch_bounds__(kThreads, 4) k_spmm(const SpmmK p) {
  using Sum = typename SumOf<AT>::type;
  constexpr int NC = 32 * CPL;
  if (gated_off(p.gate)) return;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const i64 gw = (i64)blockIdx.x * (kThreads / 32) + wib;
  const i64 nw = (i64)gridDim.x * (kThreads / 32);
  AT b[CPL];
#pragma unroll
  for (int q = 0; q < CPL; q++) {
    const int c = colof<VEC, CPL>(lane, q);
    b[q] = (EPI != EPI_STORE && p.icpt && c < p.kb) ? (AT)p.bias[c] : (AT)0;
  }
  Sum ls[CPL], bs[CPL];
  for (i64 it = gw; it < p.nitems; it += nw) {
    const Item item = p.items[it];
    AT a[CPL];
    if (item.r1 < 0) {  // piece of a long row
      row_dot<VT, XT, AT, CPL, VEC>(p, item.e0, item.e1, lane, a);
      AT* part = (AT*)p.partials + (i64)(-1 - item.r1) * NC;
#pragma unroll
      for (int q = 0; q < CPL; q++) part[colof<VEC, CPL>(lane, q)] = a[q];
    } else {
      for (i32 r = item.r0; r < item.r1; r++) {
        row_dot<VT, XT, AT, CPL, VEC>(p, __ldg(p.off + r), __ldg(p.off + r + 1), lane, a);
        spmm_epi<AT, YT, EPI, CPL, VEC>(p, r, a, b, lane, ls, bs);
      }
    }
  }
  if constexpr (EPI == EPI_LOGREG || EPI == EPI_SOFTMAX) if (EPI == EPI_LOGREG || p.cta_part) {
    __shared__ double red[kThreads / 32][NC][2];
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      red[wib][colof<VEC, CPL>(lane, q)][0] = ls[q].total();
      red[wib][colof<VEC, CPL>(lane, q)][1] = bs[q].total();
    }
    __syncthreads();
    if (threadIdx.x < 2 * NC) {
      const int col = threadIdx.x % NC, qq = threadIdx.x / NC;
      double t = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; w++) t += red[w][col][qq];
      p.cta_part[((i64)blockIdx.x * NC + col) * 2 + qq] = t;
    }
  }
}

struct SpmmFin {
  SpmmK k;
  const i32* long_rows;
  const i32* long_piece0;
  i64 nlong;
  i64 ncta;
  double* fin_part;  // [gridDim][NC][2]
  double* out;       // [kb][2]: loss, bias
  double* gbias;     // [kb] or null: where each column's bias lands
  unsigned* ticket;
  double* seg_fpart;  // stacked datasets: [nseg][warps][NC][2] of this kernel
};

// ------------------------------------------------ stacked-dataset partials
// A warp meets its rows in increasing order, so the datasets it visits come
// in order too: SegWalk keeps the current one, and when a row of a later
// dataset arrives it stores the warp's loss / bias sums of the current one
// in its slot, zeros in the slots of the datasets skipped, and loads the
// next dataset's intercepts.  finish() stores the last sums and zeros the
// remaining slots: every warp writes each of its nseg slots exactly once, so
// the reduction reads all of them in warp order without a memset.
template <class AT, int QN> struct SegWalk {
  using Sum = typename SumOf<AT>::type;
  int d = 0;
  i32 end = 0;
  double* slots;  // this warp's slot of dataset 0; slot d at + d * stride
  i64 stride;
  __device__ __forceinline__ SegWalk(const SpmmK& p, double* base, i64 warp, i64 nwarps, int nc)
      : end(p.nseg > 0 ? __ldg(p.seg_row + 1) : 0x7fffffff), slots(base ? base + warp * nc * 2 : nullptr),
        stride(nwarps * nc * 2) {}
  __device__ __forceinline__ void put(int dd, const int (&col)[QN], Sum (&ls)[QN], Sum (&bs)[QN]) {
    if (!slots) return;
    double* s = slots + dd * stride;
#pragma unroll
    for (int q = 0; q < QN; q++) {
      s[2 * col[q]] = ls[q].total();
      s[2 * col[q] + 1] = bs[q].total();
      ls[q] = Sum();
      bs[q] = Sum();
    }
  }
  __device__ __forceinline__ void zero(int dd, const int (&col)[QN]) {
    if (!slots) return;
    double* s = slots + dd * stride;
#pragma unroll
    for (int q = 0; q < QN; q++) {
      s[2 * col[q]] = 0.0;
      s[2 * col[q] + 1] = 0.0;
    }
  }
  // row r (warp-uniform) is next; true when the dataset changed
  __device__ __forceinline__ bool to_row(const SpmmK& p, i32 r, const int (&col)[QN], Sum (&ls)[QN], Sum (&bs)[QN]) {
    if (r < end) return false;
    put(d, col, ls, bs);
    d++;
    while (r >= __ldg(p.seg_row + d + 1)) zero(d++, col);
    end = __ldg(p.seg_row + d + 1);
    return true;
  }
  // the dataset of row r wherever it lies (schedules whose items are not in
  // row order; no sums are kept then)
  __device__ __forceinline__ void seek(const SpmmK& p, i32 r) {
    int lo = 0, hi = p.nseg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(p.seg_row + mid) <= r) lo = mid;
      else hi = mid - 1;
    }
    d = lo;
    end = __ldg(p.seg_row + d + 1);
  }
  __device__ __forceinline__ void finish(const SpmmK& p, const int (&col)[QN], Sum (&ls)[QN], Sum (&bs)[QN]) {
    if (!slots) return;
    put(d, col, ls, bs);
    for (int dd = d + 1; dd < p.nseg; dd++) zero(dd, col);
  }
};

// Long rows (a warp each): add the pieces' partials in piece order, apply the
// epilogue; then (logistic) the last CTA reduces all loss / bias partials per
// column in a fixed order.
//
// The hot rows of a transposed matrix have thousands of pieces, and the
// latency of their loads bounds the kernel: the row's warp alone keeps 32 in
// flight.  For a row of more than kFinShare pieces the whole CTA copies them
// through a ring of tiles in shared memory, from which the row's warp adds
// them in the same order; the rows are dealt across the CTAs, so neighbouring
// hot rows meet different ones.  2,000 pieces of 32 columns: 34 us, 95 us
// by one warp.
constexpr int kFinShare = 64;
constexpr int kFinTile = 8192;  // bytes
constexpr int kFinTiles = 3;

__device__ __forceinline__ void copy16_async(void* to, const void* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}

template <class AT, class YT, int EPI, int CPL, bool VEC>
__global__ void __launch_bounds__(kThreads) k_spmm_fin(const SpmmFin f) {
  using Sum = typename SumOf<AT>::type;
  constexpr int NC = 32 * CPL;
  const SpmmK& p = f.k;
  if (gated_off(p.gate)) return;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const bool track = p.nseg > 0;                  // stacked datasets
  const bool seg = EPI == EPI_LOGREG && track;    // per-dataset loss slots
  AT b[CPL];
  auto load_bias = [&](const double* bias) {
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      const int c = colof<VEC, CPL>(lane, q);
      b[q] = (EPI != EPI_STORE && p.icpt && c < p.kb) ? (AT)bias[c] : (AT)0;
    }
  };
  load_bias(p.bias);
  Sum ls[CPL], bs[CPL];
  int cols[CPL];
#pragma unroll
  for (int q = 0; q < CPL; q++) cols[q] = colof<VEC, CPL>(lane, q);
  const i64 gw = (i64)blockIdx.x * (kThreads / 32) + wib, nw = (i64)gridDim.x * (kThreads / 32);
  SegWalk<AT, CPL> sw(p, seg ? f.seg_fpart : nullptr, gw, nw, NC);
  unsigned long long mw = mask_of(p, 0);
  constexpr int kWarps = kThreads / 32;
  __shared__ i32 s_piece[kWarps][2];  // the pieces of each warp's row, if shared
  __shared__ __align__(16) AT s_tile[kFinTiles][kFinTile / sizeof(AT)];
  constexpr int kPer = kFinTile / (int)sizeof(AT) / NC;  // pieces of a tile
  // a row's pieces [q0, q1) one after the other, loaded kBatch at a time
  auto add_pieces = [&](i32 q0, i32 q1, AT (&a)[CPL]) {
    constexpr int kBatch = 32 / CPL;
    i32 pc = q0;
    for (; pc + kBatch <= q1; pc += kBatch) {
      AT v[kBatch][CPL];
      const AT* part = (const AT*)p.partials + (i64)pc * NC;
#pragma unroll
      for (int u = 0; u < kBatch; u++)
#pragma unroll
        for (int q = 0; q < CPL; q++) v[u][q] = __ldcg(part + u * NC + colof<VEC, CPL>(lane, q));
#pragma unroll
      for (int u = 0; u < kBatch; u++)
#pragma unroll
        for (int q = 0; q < CPL; q++) a[q] += v[u][q];
    }
    for (; pc < q1; pc++) {
      const AT* part = (const AT*)p.partials + (i64)pc * NC;
#pragma unroll
      for (int q = 0; q < CPL; q++) a[q] += __ldcg(part + colof<VEC, CPL>(lane, q));
    }
  };
  for (i64 i0 = 0; i0 < f.nlong; i0 += nw) {
    const i64 i = i0 + (i64)wib * gridDim.x + blockIdx.x;
    i32 q0 = 0, q1 = 0, row = 0;
    bool live = i < f.nlong;
    if (live) {
      q0 = f.long_piece0[i];
      q1 = f.long_piece0[i + 1];
      row = f.long_rows[i];
      if (track && sw.to_row(p, row, cols, ls, bs)) {
        if (EPI == EPI_LOGREG) load_bias(p.bias + sw.d * p.ldb);
        mw = mask_of(p, sw.d);
      }
      live = mw != 0;
    }
    const bool shared = live && q1 - q0 > kFinShare;
    if (lane == 0) {
      s_piece[wib][0] = q0;
      s_piece[wib][1] = shared ? q1 : q0;
    }
    AT a[CPL];
#pragma unroll
    for (int q = 0; q < CPL; q++) a[q] = 0;
    if (live && !shared) add_pieces(q0, q1, a);
    __syncthreads();
    for (int w = 0; w < kWarps; w++) {
      const i32 b0 = s_piece[w][0], n = s_piece[w][1] - b0;
      if (n == 0) continue;
      const i32 nt = (n + kPer - 1) / kPer;
      auto fetch = [&](i32 t) {
        if (t < nt) {
          const i32 bytes = min(n - t * kPer, kPer) * NC * (int)sizeof(AT);
          const char* from = (const char*)p.partials + (i64)(b0 + t * kPer) * NC * sizeof(AT);
          for (i32 o = threadIdx.x * 16; o < bytes; o += kThreads * 16)
            copy16_async((char*)s_tile[t % kFinTiles] + o, from + o);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      for (i32 t = 0; t < kFinTiles - 1; t++) fetch(t);
      for (i32 t = 0; t < nt; t++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kFinTiles - 2) : "memory");
        __syncthreads();  // tile t is there, tile t - 1 is read
        fetch(t + kFinTiles - 1);
        if (w == wib) {
          const AT* tile = s_tile[t % kFinTiles];
          const i32 cnt = min(n - t * kPer, kPer);
#pragma unroll 8
          for (i32 u = 0; u < cnt; u++)
#pragma unroll
            for (int q = 0; q < CPL; q++) a[q] += tile[u * NC + colof<VEC, CPL>(lane, q)];
        }
      }
      __syncthreads();
    }
    if (live) spmm_epi<AT, YT, EPI, CPL, VEC>(p, row, a, b, lane, ls, bs, mw);
    __syncthreads();  // s_piece is written by the next round
  }
  if (track && !seg) return;
  if (seg && p.nseg > 1) {
    sw.finish(p, cols, ls, bs);
    return;
  }
  if constexpr (EPI == EPI_LOGREG || EPI == EPI_SOFTMAX) if (EPI == EPI_LOGREG || p.cta_part) {
    __shared__ double red[kThreads / 32][NC][2];
    __shared__ double half[2][2 * NC];
    __shared__ bool last;
#pragma unroll
    for (int q = 0; q < CPL; q++) {
      red[wib][colof<VEC, CPL>(lane, q)][0] = ls[q].total();
      red[wib][colof<VEC, CPL>(lane, q)][1] = bs[q].total();
    }
    __syncthreads();
    if (threadIdx.x < 2 * NC) {
      const int col = threadIdx.x % NC, qq = threadIdx.x / NC;
      double t = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; w++) t += red[w][col][qq];
      (seg ? f.seg_fpart : f.fin_part)[((i64)blockIdx.x * NC + col) * 2 + qq] = t;
    }
    if (seg) return;  // one stacked dataset: a slot per CTA
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(f.ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    if constexpr (EPI == EPI_SOFTMAX) {
      // the cross-entropy sits in column 0's loss partials: thread t adds
      // CTAs t, t + 256, ... of both kernels, then a fixed tree
      CSum t;
      for (i64 bb = threadIdx.x; bb < f.ncta; bb += kThreads) t.add(__ldcg(&p.cta_part[(bb * NC) * 2]));
      for (i64 bb = threadIdx.x; bb < gridDim.x; bb += kThreads) t.add(__ldcg(&f.fin_part[(bb * NC) * 2]));
      double tl = 0.0, tb = 0.0;
      block_csum2(t.total(), 0.0, &tl, &tb);
      if (threadIdx.x == 0) {
        f.out[0] = tl;
        f.out[1] = 0.0;
        *f.ticket = 0u;
      }
      return;
    } else {
    // (column, quantity) pairs over the threads, two halves of the partials
    // each; 2*NC pairs must fit in half the CTA
    static_assert(EPI != EPI_LOGREG || 4 * NC <= kThreads, "logistic epilogue: too many columns per launch");
    const int pair = threadIdx.x % (2 * NC), hf = threadIdx.x / (2 * NC);
    const int col = pair % NC, qq = pair / NC;
    CSum t;
    if (hf < 2) {
      for (i64 bb = hf; bb < f.ncta; bb += 2) t.add(__ldcg(&p.cta_part[(bb * NC + col) * 2 + qq]));
      for (i64 bb = hf; bb < gridDim.x; bb += 2) t.add(__ldcg(&f.fin_part[(bb * NC + col) * 2 + qq]));
      half[hf][pair] = t.total();
    }
    __syncthreads();
    if (threadIdx.x < 2 * NC && col < p.kb) {
      const double tot = half[0][pair] + half[1][pair];
      if (qq == 0) {
        f.out[2 * col] = tot;
      } else {
        f.out[2 * col + 1] = p.icpt ? tot : 0.0;
        if (f.gbias) f.gbias[col] = p.icpt ? tot : 0.0;
      }
    }
    if (threadIdx.x == 0) *f.ticket = 0u;
    }
  }
}

// ------------------------------------------------ grouped lane layout
// For the store, logistic and softmax epilogues with aligned rows of X: lane
// (group g, sub-lane s) of G groups of LPR = 32 / G lanes reads columns
// s*CPL .. s*CPL+CPL-1 of a row of X with one load (CPL = 8 FP32 values,
// 32 bytes, or 2 FP64 values, 16 bytes), and group g takes nonzeros g,
// g+G, g+2G, ... of every 32-entry chunk, so a warp gathers G rows of X per
// step.  FP32 products are accumulated with packed two-lane FMAs
// (fma.rn.f32x2: each half rounds like a scalar FMA).  At the end of a row
// the groups' sums meet in a fixed butterfly that leaves lane (g, s) with the
// QG = CPL / G columns s*CPL + g*QG ... of the row (reduce-scatter), which it
// runs the epilogue on.  A launch covers NC = LPR * CPL columns; pieces and
// the per-CTA partials use the column order of the finalize kernel with
// NC / 32 columns a lane.  Each column's sum is the group sums added in the
// butterfly's fixed order (deterministic; it differs from the
// one-nonzero-at-a-time order only by rounding).
template <class XT, int G> struct GLay {
  static constexpr int CPL = sizeof(XT) == 4 ? 8 : 2;
  static constexpr int LPR = 32 / G;
  static constexpr int NC = LPR * CPL;
  static constexpr int QG = CPL / G;
  static_assert(G >= 1 && G <= CPL && NC <= 128, "groups per warp");
};

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// acc = v * x + acc on both FP32 halves
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long v, unsigned long long x) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(v), "l"(x));
}

// A chunk of 32 entries staged for the warp: the column (the row of X to
// gather) and the value, both zero past the chunk's end.  8 bytes an entry
// with FP32 values: the SM's shared-memory / L1 data path carries the gathers
// (8 passes a step of 32 lanes x 32 bytes) and two thirds of it were busy; a
// staged row offset (16 bytes) took 8 passes of it to write and 2 a step to
// read.
template <class AT> struct alignas(2 * sizeof(AT)) StageE {
  i32 col;
  AT v;
};

// The largest of the lanes' values (a NaN is ignored, as fmax does).
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// The entries a warp takes next: lane L holds entry pos + L, loaded while the
// chunk before is multiplied.  A chunk starts where the one before ended,
// whatever row it belongs to, so 32 entries are fetched without a look at the
// row bounds; at an item's end the next item's first ones.  pos tells a chunk
// that comes after skipped rows that it has to load for itself.
template <class AT> struct EntryPre {
  i32 pos = -1;
  i32 col = 0;
  AT v = 0;
};
template <class VT, class AT>
__device__ __forceinline__ void pre_fetch(const SpmmK& p, EntryPre<AT>& pre, i32 e, i32 end, int lane) {
  pre.pos = e < end ? e : -1;  // an item without entries leaves nothing for one that starts at the same place
  if (e + lane < end) {
    pre.col = __ldcs(p.idx + e + lane);
    pre.v = ld_val<VT, AT>((const VT*)p.val + e + lane);
  }
}

// Entries [e0, e1) of one row (or piece) of `item`, `next` the item the warp
// takes after it.  Group grp of the warp takes entries grp, grp + G, ... of
// each chunk of 32.  FP32: the gathers of kStep steps are issued together, in
// the last chunk under a predicate: a loop over the steps left it to the
// compiler how many were under way, and the last chunk's went one by one,
// padding included.  1M rows x 100 entries, 32 columns, BF16 values (with the
// 8-byte stage): softmax pass 908 -> 780 us, transposed pass 722 -> 702 us.
//
// HOW:
//   kBatch4  four steps' gathers together;
//   kAhead   two, and the entries fetched a chunk ahead: plain products with
//            FP32 values up to 64 columns (300 000 rows x 50 entries, 64
//            columns: 217 us without, 192 with; 128 columns of 100 000 rows:
//            151 without, 176 with) and FP64 ones up to 32 (150 000 rows x 60
//            entries, 32 columns: 545 without, 540 with; 64 columns: 955
//            without, 1,011 with).  BF16 values are faster without (60 000 rows
//            x 20 entries, 64 columns: 55 without, 58 with), and the epilogues'
//            registers and the FP64 results of the transposed pass leave no
//            room for it (64 a thread): 796 -> 832, 702 -> 797 us;
//   kBatch2  two: rows of a few entries, whose batch of four is half empty.
// The rule for plain FP32 sums is in launch_grouped_l.
enum { kBatch4, kAhead, kBatch2 };
template <class VT, class XT, class AT, int G, int HOW>
__device__ __forceinline__ void row_dot_g(const SpmmK& p, i32 e0, i32 e1, int lane, AT (&a)[GLay<XT, G>::CPL],
                                          StageE<AT>* st, bool lane_on, EntryPre<AT>& pre, const Item& item,
                                          const Item& next) {
  using L = GLay<XT, G>;
  constexpr int CPL = L::CPL;
  constexpr bool PACK = sizeof(XT) == 4 && sizeof(AT) == 4, PRE = HOW == kAhead;
  constexpr int kStep = HOW == kBatch4 ? 4 : 2;
  static_assert(32 / G >= kStep, "whole batches of steps in a chunk");
  const int sub = lane % L::LPR, grp = lane / L::LPR;
  const char* X = (const char*)((const XT*)p.X + sub * CPL);
  const unsigned ldx = (unsigned)p.ldx * sizeof(XT);  // row stride of X in bytes: launch_grouped keeps it within 32 bits
  const VT* val = (const VT*)p.val;
  const bool mine = lane_on && sub * CPL < p.kb;
  unsigned long long acc[CPL / 2];  // packed FP32 pairs
#pragma unroll
  for (int q = 0; q < CPL; q++) a[q] = 0;
#pragma unroll
  for (int q = 0; q < CPL / 2; q++) acc[q] = 0ull;
  for (i32 e = e0; e < e1; e += 32) {
    const int cnt = min(32, e1 - e);
    StageE<AT> se;
    se.col = 0;
    se.v = 0;
    if constexpr (PRE) {
      if (pre.pos != e) pre_fetch<VT, AT>(p, pre, e, item.e1, lane);
      if (lane < cnt) {
        se.col = pre.col;
        se.v = pre.v;
      }
    } else if (lane < cnt) {
      se.col = __ldcs(p.idx + e + lane);
      se.v = ld_val<VT, AT>(val + e + lane);
    }
    __syncwarp();
    st[lane] = se;
    if constexpr (PRE) {
      if (e + cnt < item.e1) pre_fetch<VT, AT>(p, pre, e + cnt, item.e1, lane);
      else pre_fetch<VT, AT>(p, pre, next.e0, next.e1, lane);
    }
    __syncwarp();
    // lanes whose columns are not computed skip the chunk
    if (!mine) continue;
    if constexpr (!PACK) {
      auto step = [&](int k) {
        const StageE<AT> t = st[k * G + grp];
        XT x[CPL];
        VecLd<XT, CPL>::ld((const XT*)(X + (unsigned long long)(unsigned)t.col * ldx), x);
#pragma unroll
        for (int q = 0; q < CPL; q++) a[q] += t.v * (AT)x[q];
      };
      const int whole = cnt / G;
#pragma unroll 4
      for (int k = 0; k < whole; k++) step(k);
      if (whole * G + grp < cnt) step(whole);  // the padding is no entry: 0 * infinity would be one
    } else {
      // the lane's 8 FP32 columns in one 32-byte load, as 4 packed pairs
      static_assert(!PACK || CPL == 8, "one 32-byte load a lane");
      auto steps = [&](int k0, auto full) {
        StageE<AT> t[kStep];
        unsigned long long x[kStep][4];
#pragma unroll
        for (int u = 0; u < kStep; u++) t[u] = st[(k0 + u) * G + grp];
#pragma unroll
        for (int u = 0; u < kStep; u++) {
          const char* row = X + (unsigned long long)(unsigned)t[u].col * ldx;
          if constexpr (decltype(full)::value) {
            asm volatile("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(x[u][0]), "=l"(x[u][1]), "=l"(x[u][2]), "=l"(x[u][3])
                         : "l"(row));
          } else {
            const int on = (k0 + u) * G + grp < cnt;
            asm volatile(
                "{ .reg .pred p; setp.ne.s32 p, %5, 0;\n"
                " mov.b64 %0, 0; mov.b64 %1, 0; mov.b64 %2, 0; mov.b64 %3, 0;\n"
                " @p ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4]; }"
                : "=&l"(x[u][0]), "=&l"(x[u][1]), "=&l"(x[u][2]), "=&l"(x[u][3])
                : "l"(row), "r"(on));
          }
        }
#pragma unroll
        for (int u = 0; u < kStep; u++) {
          const unsigned long long vv = pack2((float)t[u].v, (float)t[u].v);
#pragma unroll
          for (int q = 0; q < 4; q++) fma2(acc[q], vv, x[u][q]);
        }
      };
      if (cnt == 32) {
#pragma unroll
        for (int k = 0; k < 32 / G; k += kStep) steps(k, std::true_type());
      } else {
        for (int k = 0; k * G < cnt; k += kStep) steps(k, std::false_type());
      }
    }
  }
  if constexpr (PACK) {
#pragma unroll
    for (int q = 0; q < CPL / 2; q++) {
      float lo, hi;
      unpack2(acc[q], lo, hi);
      a[2 * q] = lo;
      a[2 * q + 1] = hi;
    }
  }
  // reduce-scatter over the groups: at offset o the lane keeps the half of
  // its columns picked by bit o of its lane id and sends the other half
#pragma unroll
  for (int o = 16, h = CPL / 2; o >= L::LPR; o >>= 1, h >>= 1) {
    const bool hi = (lane & o) != 0;
#pragma unroll
    for (int q = 0; q < h; q++) {
      const AT keep = hi ? a[h + q] : a[q];
      const AT send = hi ? a[q] : a[h + q];
      a[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
}

// CTAs per SM: four (64 registers a thread), three for the transposed pass of
// the trainings (FP32 arithmetic, FP64 results) from 64 columns on, whose rows
// of X of 256 bytes and more gain from fewer warps sharing the L1: 107 -> 98
// us at 200 000 x 20 000, 10M entries, 64 columns (32 columns: 702 -> 780).
template <class XT, class YT, int EPI, int G>
constexpr int kGroupedCtas = EPI == EPI_STORE && sizeof(XT) == 4 && sizeof(YT) == 8 && G <= 4 ? 3 : 4;

template <class VT, class XT, class AT, class YT, int EPI, int G, int HOW>
__global__ void __launch_bounds__(kThreads, kGroupedCtas<XT, YT, EPI, G>) k_spmm_g(const SpmmK p) {
  using L = GLay<XT, G>;
  using Sum = typename SumOf<AT>::type;
  constexpr int CPL = L::CPL, NC = L::NC, QG = L::QG;
  if (gated_off(p.gate)) return;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int c0 = (lane % L::LPR) * CPL + (lane / L::LPR) * QG;  // first of the lane's epilogue columns
  const i64 gw = (i64)blockIdx.x * (kThreads / 32) + wib;
  const i64 nw = (i64)gridDim.x * (kThreads / 32);
  const bool track = p.nseg > 0;                // stacked datasets
  const bool seg = EPI == EPI_LOGREG && track;  // per-dataset loss slots
  int cols[QG];
#pragma unroll
  for (int q = 0; q < QG; q++) cols[q] = c0 + q;
  AT b[QG];
  auto load_bias = [&](const double* bias) {
#pragma unroll
    for (int q = 0; q < QG; q++) b[q] = (EPI != EPI_STORE && p.icpt && cols[q] < p.kb) ? (AT)bias[cols[q]] : (AT)0;
  };
  load_bias(p.bias);
  Sum ls[QG], bs[QG];
  SegWalk<AT, QG> walk(p, seg ? p.seg_part : nullptr, gw, nw, NC);
  const int lsh = (lane % L::LPR) * CPL;  // the lane's gathered columns: lsh .. lsh + CPL - 1
  __shared__ StageE<AT> stage[kThreads / 32][32];
  unsigned long long mw = mask_of(p, 0);
  AT lab = 0, w = 1;
  constexpr bool PRE = HOW == kAhead;  // entries fetched ahead: see row_dot_g
  EntryPre<AT> pre;
  Item next{0, 0, 0, 0};
  if (PRE && gw < p.nitems) next = p.items[gw];
  for (i64 it = gw; it < p.nitems; it += nw) {
    const Item item = PRE ? next : p.items[it];
    if (PRE) next = it + nw < p.nitems ? p.items[it + nw] : Item{0, 0, 0, 0};
    AT a[CPL];
    // the store epilogue keeps no per-dataset sums, so its items may come in
    // any order (slab-ordered pieces): each item looks its dataset up
    if (EPI == EPI_STORE && track) {
      walk.seek(p, item.r0);
      mw = mask_of(p, walk.d);
    }
    if (item.r1 < 0) {  // piece of a long row (item.r0)
      if (EPI != EPI_STORE && track && walk.to_row(p, item.r0, cols, ls, bs)) {
        if (EPI == EPI_LOGREG) load_bias(p.bias + walk.d * p.ldb);
        mw = mask_of(p, walk.d);
      }
      if (mw == 0) continue;  // the finalize skips the row too
      row_dot_g<VT, XT, AT, G, HOW>(p, item.e0, item.e1, lane, a, stage[wib], cols_on(mw, lsh, CPL), pre, item,
                                    next);
      AT* part = (AT*)p.partials + (i64)(-1 - item.r1) * NC;
#pragma unroll
      for (int q = 0; q < QG; q++) part[cols[q]] = a[q];
      continue;
    }
    for (i32 r = item.r0; r < item.r1; r++) {
      if (track && walk.to_row(p, r, cols, ls, bs)) {
        if (EPI == EPI_LOGREG) load_bias(p.bias + walk.d * p.ldb);
        mw = mask_of(p, walk.d);
      }
      if (mw == 0) continue;  // no column of this dataset is computed
      row_dot_g<VT, XT, AT, G, HOW>(p, __ldg(p.off + r), __ldg(p.off + r + 1), lane, a, stage[wib], cols_on(mw, lsh, CPL), pre, item,
                                    next);
      if constexpr (EPI == EPI_STORE) {
        YT* y = (YT*)p.Y + (i64)r * p.ldy;
#pragma unroll
        for (int q = 0; q < QG; q++)
          if (cols[q] < p.kb && col_on(mw, cols[q])) y[cols[q]] = (YT)a[q];
      } else {
        // labels: always with the logistic epilogue; the softmax one runs
        // without them for the probability matrix alone
        const bool has_label = (sizeof(AT) == 8) ? p.label != nullptr : p.label_f != nullptr;
        bool has_sw = false;
        if (has_label) {
          if constexpr (sizeof(AT) == 8) {
            lab = p.label[r];
            has_sw = p.sw != nullptr;
            if (has_sw) w = p.sw[r];
          } else {
            lab = p.label_f[r];
            has_sw = p.sw_f != nullptr;
            if (has_sw) w = p.sw_f[r];
          }
        }
        AT* rr = (AT*)p.R + (i64)r * p.ldr;
        if constexpr (EPI == EPI_LOGREG) {
#pragma unroll
          for (int q = 0; q < QG; q++) {
            if (cols[q] >= p.kb || !col_on(mw, cols[q])) continue;
            AT loss, d;
            if constexpr (sizeof(AT) == 4) {
              if (p.loss == LOSS_LOGISTIC) logistic_row_1exp(a[q] + b[q], lab, loss, d);
              else glm_row<AT>(p.loss, (AT)p.eps, a[q] + b[q], lab, loss, d);
            } else {
              glm_row<AT>(p.loss, (AT)p.eps, a[q] + b[q], lab, loss, d);
            }
            if (has_sw) d = d * w;
            rr[cols[q]] = d;
            ls[q].add(loss);
            bs[q].add(d);
          }
        } else {  // softmax over the row's classes, every class held by one lane
          AT z[QG], mx = -INFINITY;
#pragma unroll
          for (int q = 0; q < QG; q++) {
            z[q] = a[q] + b[q];
            if (cols[q] < p.kb) mx = fmax(mx, z[q]);
          }
          mx = warp_max(mx);
          AT zy = 0, sum = 0;
#pragma unroll
          for (int q = 0; q < QG; q++) {
            if (has_label && cols[q] < p.kb && lab == (AT)cols[q]) zy = z[q] - mx;
            z[q] = cols[q] < p.kb ? exp_acc<AT>(z[q] - mx) : (AT)0;
            sum += z[q];
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
          // cross-entropy -log p[label] = log(sum) - (z_label - max), unweighted
          if (has_label && p.cta_part) {
            // the label's lane alone holds a value other than 0
            const unsigned own = __ballot_sync(0xffffffffu, zy != (AT)0);
            zy = __shfl_sync(0xffffffffu, zy, own ? __ffs(own) - 1 : 0);
            if (lane == 0) ls[0].add(log_acc<AT>(sum) - zy);
          }
          const AT inv = (AT)1 / sum;
#pragma unroll
          for (int q = 0; q < QG; q++) {
            if (cols[q] >= p.kb) continue;
            AT pr = inv * z[q];
            if (has_label) {
              pr -= (lab == (AT)cols[q]) ? (AT)1 : (AT)0;
              if (has_sw) pr *= w;
            }
            rr[cols[q]] = pr;
          }
        }
      }
    }
  }
  if (track && !seg) return;
  if constexpr (EPI == EPI_LOGREG || EPI == EPI_SOFTMAX) {
    if (EPI == EPI_SOFTMAX && !p.cta_part) return;
    if (seg && p.nseg > 1) {
      walk.finish(p, cols, ls, bs);
      return;
    }
    // one dataset (stacked or not): the CTA's warps added in order
    __shared__ double red[kThreads / 32][NC][2];
#pragma unroll
    for (int q = 0; q < QG; q++) {
      red[wib][cols[q]][0] = ls[q].total();
      red[wib][cols[q]][1] = bs[q].total();
    }
    __syncthreads();
    if (threadIdx.x < 2 * NC) {
      const int col = threadIdx.x % NC, qq = threadIdx.x / NC;
      double t = 0;
#pragma unroll
      for (int w8 = 0; w8 < kThreads / 32; w8++) t += red[w8][col][qq];
      (seg ? p.seg_part : p.cta_part)[((i64)blockIdx.x * NC + col) * 2 + qq] = t;
    }
  }
}

// Stacked datasets: loss / bias sums of dataset blockIdx.x from the slots of
// the main kernel (nw1 slots: its warps, or its CTAs when one dataset is
// stacked) and of the finalize kernel (nw2), in a fixed order.  A compensated
// FP64 add costs five FP64 instructions, so the slots are spread over
// gridDim.z CTAs: CTA (d, y, z) takes the 32 (column, quantity) pairs of y in
// 8 stripes, stripe s the slots z*8 + s, + 8 * gridDim.z, ...; the last CTA of
// (d, y) adds the CTAs' sums in order.  out[2 * (d * ldo + col) + q]; the bias
// sums also go to gb[grow[d] * ldg + col].  One dataset of 200,000 rows, 64
// models, averaged over the launches of a training (half of them gated off):
// 1.8 us; one CTA per 32 pairs over a slot per warp took 27.8 us.
constexpr int kSegZ = 16;  // most CTAs per (dataset, 32 pairs)
template <int NC>
__global__ void __launch_bounds__(256) k_spmm_seg_reduce(const double* __restrict__ s1, i64 nw1,
                                                         const double* __restrict__ s2, i64 nw2, int kout, int icpt,
                                                         double* __restrict__ out, i64 ldo, double* __restrict__ gb,
                                                         const i64* __restrict__ grow, i64 ldg, const int* gate,
                                                         const unsigned long long* mask, i64 mstride, int mword,
                                                         double* __restrict__ rpart, unsigned* __restrict__ tickets) {
  constexpr int P = 2 * NC, S = 8;
  static_assert(P % 32 == 0, "pairs per CTA");
  __shared__ double part[S][33];
  __shared__ bool last;
  if (gated_off(gate)) return;
  const int d = blockIdx.x, dy = d * gridDim.y + blockIdx.y, Z = gridDim.z;
  const int pl = threadIdx.x & 31, st = threadIdx.x >> 5;
  const int pr = blockIdx.y * 32 + pl;
  CSum t;
  const double* b1 = s1 + (i64)d * nw1 * P + pr;
  const double* b2 = s2 + (i64)d * nw2 * P + pr;
  for (i64 w = blockIdx.z * S + st; w < nw1 + nw2; w += S * Z) t.add(w < nw1 ? __ldcg(b1 + w * P) : __ldcg(b2 + (w - nw1) * P));
  part[st][pl] = t.total();
  __syncthreads();
  if (st != 0) return;
  double tot = 0.0;
#pragma unroll
  for (int q = 0; q < S; q++) tot += part[q][pl];
  if (Z > 1) {
    double* rp = rpart + (i64)dy * kSegZ * 32;
    rp[blockIdx.z * 32 + pl] = tot;
    __threadfence();
    __syncwarp();
    if (pl == 0) last = atomicAdd(tickets + dy, 1u) == (unsigned)Z - 1;
    __syncwarp();
    if (!last) return;
    __threadfence();
    tot = 0.0;
    for (int z = 0; z < Z; z++) tot += __ldcg(rp + z * 32 + pl);
    if (pl == 0) tickets[dy] = 0u;
  }
  const int col = pr >> 1, qq = pr & 1;
  if (col >= kout) return;
  if (mask && !col_on(__ldcg(mask + (i64)d * mstride + mword), col)) return;  // not evaluated: keep
  if (qq == 0) {
    out[2 * ((i64)d * ldo + col)] = tot;
  } else {
    out[2 * ((i64)d * ldo + col) + 1] = icpt ? tot : 0.0;
    if (gb) gb[grow[d] * ldg + col] = icpt ? tot : 0.0;
  }
}

// ------------------------------------------------------------ host side
static size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

template <class VT, class XT, class AT, class YT, int EPI, int CPL, bool VEC>
static int spmm_grid(fvg_ctx* c) {
  return occupancy_blocks((const void*)k_spmm<VT, XT, AT, YT, EPI, CPL, VEC>, kThreads) * c->num_sms;
}

static int spmm_fin_grid(fvg_ctx* c, i64 nlong) {
  return (int)std::max<i64>(1, std::min<i64>(nlong, 2 * c->num_sms));  // a CTA each while they last: rows are shared by its warps
}

// Scratch of one block pass (sized for 128 columns): ticket, per-CTA
// partials of the main and finalize kernels, long-row piece partials.
i64 spmm_scratch_bytes(fvg_ctx* c, DevCRS& a, int storage, i64 slab) {
  const Sched& s = slab > 0 ? crs_sched_slabs(c, a, storage, slab) : pass_sched(c, a, storage);
  const size_t at = storage == FVG_F64 ? 8 : 4;
  const i64 grid = 8 * (i64)c->num_sms;  // occupancy upper bound (8 CTAs of 256 threads per SM)
  return (i64)(al256(256) + al256(sizeof(double) * 2 * kSpmmMaxCols * grid) +
               al256(sizeof(double) * 2 * kSpmmMaxCols * spmm_fin_grid(c, s.nlong)) +
               al256(at * kSpmmMaxCols * std::max<i64>(s.npieces, 1)));
}

template <class VT, class XT, class AT, class YT, int EPI, int CPL, bool VEC>
static void launch_spmm_l(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, SpmmK p, double* out, double* gbias,
                          char* scratch) {
  const int grid =
      (int)std::max<i64>(1, std::min<i64>(spmm_grid<VT, XT, AT, YT, EPI, CPL, VEC>(c), (s.nitems + 7) / 8));
  const int fg = spmm_fin_grid(c, s.nlong);
  unsigned* ticket = (unsigned*)scratch;
  double* cta = (double*)(scratch + al256(256));
  double* fin = (double*)((char*)cta + al256(sizeof(double) * 2 * kSpmmMaxCols * 8 * (i64)c->num_sms));
  p.partials = (char*)fin + al256(sizeof(double) * 2 * kSpmmMaxCols * fg);
  p.off = a.off.as<i32>();
  p.idx = a.idx.as<i32>();
  p.val = a.val[storage].p;
  p.items = s.items.as<Item>();
  p.nitems = s.nitems;
  // softmax: the cross-entropy is reduced only when the caller asks for it
  const bool reduce = EPI == EPI_LOGREG || (EPI == EPI_SOFTMAX && out);
  p.cta_part = reduce ? cta : nullptr;
  if (s.nitems > 0) {
    k_spmm<VT, XT, AT, YT, EPI, CPL, VEC><<<grid, kThreads, 0, c->stream>>>(p);
    check_launch("k_spmm");
    count_launch(c);
  }
  if (s.nlong > 0 || reduce) {
    SpmmFin f;
    f.k = p;
    f.long_rows = s.long_rows.as<i32>();
    f.long_piece0 = s.long_piece0.as<i32>();
    f.nlong = s.nlong;
    f.ncta = s.nitems > 0 ? grid : 0;
    f.fin_part = fin;
    f.out = out;
    f.gbias = gbias;
    f.ticket = ticket;
    k_spmm_fin<AT, YT, EPI, CPL, VEC><<<fg, kThreads, 0, c->stream>>>(f);
    check_launch("k_spmm_fin");
    count_launch(c);
  }
}

static bool aligned_to(const void* ptr, size_t b) { return ((uintptr_t)ptr % b) == 0; }

// Scratch of a stacked-dataset pass (SpmmSeg::slots): the reduction's tickets
// (zeroed once by spmm_seg_init) and its CTAs' sums, then the slots.
constexpr int kSegY = 2 * kSpmmMaxCols / 32;  // 32-pair groups of the widest block
static i64 seg_ticket_bytes(int nseg) { return (i64)al256(sizeof(unsigned) * kSegY * (size_t)nseg); }
static i64 seg_part_bytes(int nseg) { return (i64)sizeof(double) * kSegY * kSegZ * 32 * nseg; }
static double* seg_parts(const SpmmSeg& sg) { return (double*)((char*)sg.slots + seg_ticket_bytes(sg.nseg)); }
static double* seg_slots(const SpmmSeg& sg) {
  return (double*)((char*)sg.slots + seg_ticket_bytes(sg.nseg) + seg_part_bytes(sg.nseg));
}

// Grouped layout launch: k_spmm_g and its finalize kernel (NC / 32
// columns a lane); for stacked datasets the slot reduction is left to
// crs_spmm_seg_finish.
template <class VT, class XT, class AT, class YT, int EPI, int G, int HOW>
static void launch_grouped_how(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, SpmmK p, double* out,
                             double* gbias, char* scratch, SpmmSeg* sg) {
  using L = GLay<XT, G>;
  constexpr int NC = L::NC, CF = NC / 32;
  const int grid = (int)std::max<i64>(
      1, std::min<i64>(occupancy_blocks((const void*)k_spmm_g<VT, XT, AT, YT, EPI, G, HOW>, kThreads) * c->num_sms,
                       (s.nitems + 7) / 8));
  const int fg = spmm_fin_grid(c, s.nlong);
  unsigned* ticket = (unsigned*)scratch;
  double* cta = (double*)(scratch + al256(256));
  double* fin = (double*)((char*)cta + al256(sizeof(double) * 2 * kSpmmMaxCols * 8 * (i64)c->num_sms));
  p.partials = (char*)fin + al256(sizeof(double) * 2 * kSpmmMaxCols * fg);
  p.off = a.off.as<i32>();
  p.idx = a.idx.as<i32>();
  p.val = a.val[storage].p;
  p.items = s.items.as<Item>();
  p.nitems = s.nitems;
  // softmax: the cross-entropy is reduced only when the caller asks for it
  const bool reduce = EPI == EPI_LOGREG || (EPI == EPI_SOFTMAX && out);
  p.cta_part = reduce ? cta : nullptr;
  const bool track = sg && sg->nseg > 0;
  const bool seg = EPI == EPI_LOGREG && track;
  // slots of a stacked dataset: a warp each, or with one dataset a CTA each
  const i64 per = track && sg->nseg == 1 ? 1 : kThreads / 32;
  const i64 nw1 = grid * per, nw2 = fg * per;
  double* const slots = seg ? seg_slots(*sg) : nullptr;
  if (track) {
    if (!sg->seg_row || (seg && !sg->slots) || sg->nseg > 65535)
      fail(FVG_ERR_INTERNAL, "stacked-dataset pass without its row bounds or slots");
    if (sg->mask && p.kb > 64) fail(FVG_ERR_INTERNAL, "column masks cover 64 columns");
    p.nseg = sg->nseg;
    p.seg_row = sg->seg_row;
    p.ldb = sg->ldb;
    p.seg_part = slots;
    p.gate = sg->gate;
    p.mask = sg->mask;
    p.mstride = sg->mstride;
    p.mword = sg->mword;
  }
  if (s.nitems > 0 || seg) {
    k_spmm_g<VT, XT, AT, YT, EPI, G, HOW><<<grid, kThreads, 0, c->stream>>>(p);
    check_launch("k_spmm_g");
    count_launch(c);
  }
  if (s.nlong > 0 || reduce) {
    SpmmFin f;
    f.k = p;
    f.long_rows = s.long_rows.as<i32>();
    f.long_piece0 = s.long_piece0.as<i32>();
    f.nlong = s.nlong;
    f.ncta = s.nitems > 0 ? grid : 0;
    f.fin_part = fin;
    f.out = out;
    f.gbias = gbias;
    f.ticket = ticket;
    f.seg_fpart = seg ? slots + (i64)sg->nseg * nw1 * NC * 2 : nullptr;
    k_spmm_fin<AT, YT, EPI, CF, true><<<fg, kThreads, 0, c->stream>>>(f);
    check_launch("k_spmm_fin");
    count_launch(c);
  }
  if (seg) {
    sg->nw1 = nw1;
    sg->nw2 = nw2;
    sg->nc = NC;
    sg->icpt = p.icpt;
  }
}

// How the gathers of plain sums (up to 64 FP32 or 32 FP64 columns) are issued.
// Two steps at a time where rows are short: a batch of four is then mostly
// predicates (300,000 rows x 5 entries, two / four: BF16 values, 8 columns 103
// / 117 us, 64 columns 112 / 127; FP32 values, 8 columns 104 / 113 with entries
// ahead; 13 entries, BF16, 8 columns 99 / 108, 64 columns 136 / 136).
// Entries ahead for FP32 values, except where the columns are scattered
// (DevCRS::spread) over more of X than L2 keeps beside the entries: the rows of
// X then come from HBM, and four gathers under way do more than early entries
// (300,000 power-law rows x 40 entries, 64 columns, ahead / four: X of 77 MB
// 341 / 315 us, 128 MB 428 / 389; 40 columns, 48 MB 246 / 246).
constexpr i64 kShortRows = 7, kShortRows16 = 15;
constexpr i64 kSpreadX = 64ll << 20;
template <class VT, class XT, class AT, class YT, int EPI, int G>
static void launch_grouped_l(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, SpmmK p, double* out,
                             double* gbias, char* scratch, SpmmSeg* sg) {
  auto launch = [&](auto how) {
    launch_grouped_how<VT, XT, AT, YT, EPI, G, decltype(how)::value>(c, a, s, storage, p, out, gbias, scratch, sg);
  };
  if constexpr (EPI == EPI_STORE && sizeof(YT) == sizeof(AT) && sizeof(AT) == 8 && G >= 2) {
    launch(std::integral_constant<int, kAhead>());
  } else if constexpr (EPI == EPI_STORE && sizeof(YT) == sizeof(AT) && sizeof(AT) == 4 && G >= 4) {
    const bool scattered = a.spread && a.n * p.ldx * (i64)sizeof(XT) > kSpreadX;
    constexpr i64 kShort = sizeof(VT) == 2 && G == 8 ? kShortRows16 : kShortRows;
    if (a.nnz < kShort * a.m) launch(std::integral_constant<int, kBatch2>());
    else if (sizeof(VT) == 4 && !scattered) launch(std::integral_constant<int, kAhead>());
    else launch(std::integral_constant<int, kBatch4>());
  } else {
    launch(std::integral_constant<int, kBatch4>());
  }
}

// Grouped layout when its 16-byte accesses are aligned; false: not taken.
template <class VT, class XT, class AT, class YT, int EPI>
static bool launch_grouped(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, const SpmmK& p, double* out,
                           double* gbias, char* scratch, SpmmSeg* sg = nullptr) {
  // vector loads: column blocks and strides in whole vectors (the FP32
  // lanes read 8 columns, the FP64 ones 2), 16-byte aligned bases
  constexpr int VW = 16 / (int)sizeof(XT);
  bool ok = p.kb % VW == 0 && p.ldx % VW == 0 && aligned_to(p.X, 16) && p.ldx * (i64)sizeof(XT) < (i64)1 << 32;
  if (EPI == EPI_STORE) ok = ok && p.ldy % VW == 0 && aligned_to(p.Y, 16);
  else ok = ok && p.ldr % VW == 0 && aligned_to(p.R, 16);
  if (!ok) return false;
  if constexpr (sizeof(XT) == 4) {
    // FP32: 8 columns a lane read with one 32-byte load: whole 8-column
    // groups, 32-byte aligned rows
    if (p.kb % 8 != 0 || p.ldx % 8 != 0 || p.kb > 128 || !aligned_to(p.X, 32)) return false;
    if (p.kb <= 32) {
      launch_grouped_l<VT, XT, AT, YT, EPI, 8>(c, a, s, storage, p, out, gbias, scratch, sg);
      return true;
    }
    if (p.kb <= 64) {
      launch_grouped_l<VT, XT, AT, YT, EPI, 4>(c, a, s, storage, p, out, gbias, scratch, sg);
      return true;
    }
    // the logistic epilogue's finalize reduction takes at most 64 columns
    if constexpr (EPI != EPI_LOGREG) {
      launch_grouped_l<VT, XT, AT, YT, EPI, 2>(c, a, s, storage, p, out, gbias, scratch, sg);
      return true;
    }
    return false;
  } else {
    if (p.kb > 64) return false;
    if (p.kb <= 32) launch_grouped_l<VT, XT, AT, YT, EPI, 2>(c, a, s, storage, p, out, gbias, scratch, sg);
    else launch_grouped_l<VT, XT, AT, YT, EPI, 1>(c, a, s, storage, p, out, gbias, scratch, sg);
    return true;
  }
}

// Packed lane layout when every access it makes is aligned: the block's
// width and the strides of X and of the output are multiples of CPL and the
// bases are aligned to CPL elements.
template <class VT, class XT, class AT, class YT, int EPI, int CPL>
static void launch_spmm(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, SpmmK p, double* out, double* gbias,
                        char* scratch) {
  bool vec = CPL >= 2 && p.kb % CPL == 0 && p.ldx % CPL == 0 && aligned_to(p.X, CPL * sizeof(XT));
  if (EPI == EPI_STORE) vec = vec && p.ldy % CPL == 0 && aligned_to(p.Y, CPL * sizeof(YT));
  else vec = vec && p.ldr % CPL == 0 && aligned_to(p.R, CPL * sizeof(AT));
  if constexpr (CPL >= 2) {
    if (vec) {
      launch_spmm_l<VT, XT, AT, YT, EPI, CPL, true>(c, a, s, storage, p, out, gbias, scratch);
      return;
    }
  }
  launch_spmm_l<VT, XT, AT, YT, EPI, CPL, false>(c, a, s, storage, p, out, gbias, scratch);
}

template <class VT, class XT, class AT, class YT>
static void launch_store(fvg_ctx* c, DevCRS& a, const Sched& s, int storage, const SpmmK& p, char* sc) {
  if (p.kb <= 32) launch_spmm<VT, XT, AT, YT, EPI_STORE, 1>(c, a, s, storage, p, nullptr, nullptr, sc);
  else if (p.kb <= 64) launch_spmm<VT, XT, AT, YT, EPI_STORE, 2>(c, a, s, storage, p, nullptr, nullptr, sc);
  else launch_spmm<VT, XT, AT, YT, EPI_STORE, 4>(c, a, s, storage, p, nullptr, nullptr, sc);
}

// Y[:, c0:c0+kb] = A X[:, c0:c0+kb] (X, Y pointers already offset to c0).
void crs_spmm_block(fvg_ctx* c, DevCRS& a, int storage, const void* X, i64 ldx, int kb, int y_dt, void* Y, i64 ldy,
                    void* scratch, const int* gate, i64 slab) {
  if (kb < 1 || kb > kSpmmMaxCols) fail(FVG_ERR_INTERNAL, "spmm block width out of range");
  if (!a.val[storage].p) fail(FVG_ERR_INTERNAL, "missing value plane for the requested storage");
  const Sched& s = slab > 0 ? crs_sched_slabs(c, a, storage, slab) : pass_sched(c, a, storage);
  SpmmK p = {};
  p.X = X;
  p.ldx = ldx;
  if (ldx > 0x7fffffffll) fail(FVG_ERR_INVALID_ARG, "dense operand row stride beyond 2^31 - 1");
  p.kb = kb;
  p.Y = Y;
  p.ldy = ldy;
  p.gate = gate;
  char* sc = (char*)scratch;
  if (storage == FVG_F64) {
    if (!launch_grouped<double, double, double, double, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc))
      launch_store<double, double, double, double>(c, a, s, storage, p, sc);
  } else if (storage == FVG_F32) {
    if (y_dt == FVG_F64) {
      if (!launch_grouped<float, float, float, double, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc))
        launch_store<float, float, float, double>(c, a, s, storage, p, sc);
    } else if (!launch_grouped<float, float, float, float, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc)) {
      launch_store<float, float, float, float>(c, a, s, storage, p, sc);
    }
  } else {
    if (y_dt == FVG_F64) {
      if (!launch_grouped<bf16, float, float, double, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc))
        launch_store<bf16, float, float, double>(c, a, s, storage, p, sc);
    } else if (!launch_grouped<bf16, float, float, float, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc)) {
      launch_store<bf16, float, float, float>(c, a, s, storage, p, sc);
    }
  }
}

// Y = A X over stacked datasets (rows [seg_row[d], seg_row[d+1]) of A belong
// to dataset d) with the column masks and the gate of sg; masked columns of
// Y keep what they held.  X, Y and their strides 16-byte aligned, kb a
// multiple of 8 (of 2 for FP64) and at most 64.
void crs_spmm_store_seg(fvg_ctx* c, DevCRS& a, int storage, const void* X, i64 ldx, int kb, void* Y, i64 ldy,
                        void* scratch, SpmmSeg& sg, i64 slab) {
  if (kb < 1 || kb > 64 || sg.nseg < 1) fail(FVG_ERR_INTERNAL, "stacked store: block width or datasets out of range");
  if (!a.val[storage].p) fail(FVG_ERR_INTERNAL, "missing value plane for the requested storage");
  const Sched& s = slab > 0 ? crs_sched_slabs(c, a, storage, slab) : pass_sched(c, a, storage);
  SpmmK p = {};
  p.X = X;
  p.ldx = ldx;
  if (ldx > 0x7fffffffll) fail(FVG_ERR_INVALID_ARG, "dense operand row stride beyond 2^31 - 1");
  p.kb = kb;
  p.Y = Y;
  p.ldy = ldy;
  char* sc = (char*)scratch;
  bool ok;
  if (storage == FVG_F64)
    ok = launch_grouped<double, double, double, double, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc, &sg);
  else if (storage == FVG_F32)
    ok = launch_grouped<float, float, float, double, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc, &sg);
  else
    ok = launch_grouped<bf16, float, float, double, EPI_STORE>(c, a, s, storage, p, nullptr, nullptr, sc, &sg);
  if (!ok) fail(FVG_ERR_INTERNAL, "stacked store needs 16-byte aligned rows");
}

// Batched GLM forward pass over a block of kb <= 64 models: R = dloss(A W +
// b) * sw per (row, model) for the loss kind `loss`; out[2j] = loss of model
// j, out[2j+1] = its bias sum (0 without intercept), also written to gbias[j]
// when given.
void crs_spmm_logreg_block(fvg_ctx* c, DevCRS& a, int storage, const void* W, i64 ldw, int kb, const double* label,
                           const double* sw, const float* label_f, const float* sw_f, int icpt, const double* bias,
                           void* R, i64 ldr, double* out, double* gbias, void* scratch, int loss, double eps) {
  if (kb < 1 || kb > 64) fail(FVG_ERR_INTERNAL, "spmm block width out of range");
  const Sched& s = pass_sched(c, a, storage);
  SpmmK p = {};
  p.X = W;
  p.ldx = ldw;
  if (ldw > 0x7fffffffll) fail(FVG_ERR_INVALID_ARG, "dense operand row stride beyond 2^31 - 1");
  p.kb = kb;
  p.label = label;
  p.sw = sw;
  p.label_f = label_f;
  p.sw_f = sw_f;
  p.icpt = icpt;
  p.bias = bias;
  p.R = R;
  p.ldr = ldr;
  p.loss = loss;
  p.eps = eps;
  char* sc = (char*)scratch;
  FVG_CUDA(cudaMemsetAsync(sc, 0, 256, c->stream));
  if (storage == FVG_F64) {
    if (!launch_grouped<double, double, double, double, EPI_LOGREG>(c, a, s, storage, p, out, gbias, sc))
      launch_spmm<double, double, double, double, EPI_LOGREG, 2>(c, a, s, storage, p, out, gbias, sc);
  } else if (storage == FVG_F32) {
    if (!launch_grouped<float, float, float, float, EPI_LOGREG>(c, a, s, storage, p, out, gbias, sc))
      launch_spmm<float, float, float, float, EPI_LOGREG, 2>(c, a, s, storage, p, out, gbias, sc);
  } else if (!launch_grouped<bf16, float, float, float, EPI_LOGREG>(c, a, s, storage, p, out, gbias, sc)) {
    launch_spmm<bf16, float, float, float, EPI_LOGREG, 2>(c, a, s, storage, p, out, gbias, sc);
  }
}

// Warp slots of a stacked-dataset pass: main kernel (at most 8 CTAs an SM)
// and finalize kernel, NC = the launch's columns, two doubles each.
i64 spmm_seg_slot_bytes(fvg_ctx* c, int nseg, int kb) {
  const i64 nc = kb <= 32 ? 32 : (kb <= 64 ? 64 : 128);
  const i64 warps = (8 * (i64)c->num_sms + 2 * (i64)c->num_sms) * (kThreads / 32);
  const int ns = std::max(nseg, 1);
  return seg_ticket_bytes(ns) + seg_part_bytes(ns) + ns * warps * nc * 2 * (i64)sizeof(double);
}

void spmm_seg_init(fvg_ctx* c, void* slots, int nseg) {
  FVG_CUDA(cudaMemsetAsync(slots, 0, (size_t)seg_ticket_bytes(std::max(nseg, 1)), c->stream));
}

void crs_spmm_logreg_seg(fvg_ctx* c, DevCRS& a, int storage, const void* W, i64 ldw, int kb, const double* label,
                         const double* sw, const float* label_f, const float* sw_f, int icpt, const double* bias,
                         void* R, i64 ldr, void* scratch, SpmmSeg& sg, int loss, double eps) {
  if (kb < 1 || kb > 64 || sg.nseg < 1) fail(FVG_ERR_INTERNAL, "stacked pass: block width or datasets out of range");
  const Sched& s = pass_sched(c, a, storage);
  SpmmK p = {};
  p.X = W;
  p.ldx = ldw;
  if (ldw > 0x7fffffffll) fail(FVG_ERR_INVALID_ARG, "dense operand row stride beyond 2^31 - 1");
  p.kb = kb;
  p.label = label;
  p.sw = sw;
  p.label_f = label_f;
  p.sw_f = sw_f;
  p.icpt = icpt;
  p.bias = bias;
  p.R = R;
  p.ldr = ldr;
  p.loss = loss;
  p.eps = eps;
  char* sc = (char*)scratch;
  bool ok;
  if (storage == FVG_F64)
    ok = launch_grouped<double, double, double, double, EPI_LOGREG>(c, a, s, storage, p, nullptr, nullptr, sc, &sg);
  else if (storage == FVG_F32)
    ok = launch_grouped<float, float, float, float, EPI_LOGREG>(c, a, s, storage, p, nullptr, nullptr, sc, &sg);
  else
    ok = launch_grouped<bf16, float, float, float, EPI_LOGREG>(c, a, s, storage, p, nullptr, nullptr, sc, &sg);
  if (!ok) fail(FVG_ERR_INTERNAL, "stacked pass needs 16-byte aligned rows");
}

// Per-dataset loss / bias sums of the last crs_spmm_logreg_seg pass (after
// the backward product, which writes the bias rows of the gradient as 0).
void crs_spmm_seg_finish(fvg_ctx* c, const SpmmSeg& sg) {
  if (sg.nw1 <= 0) fail(FVG_ERR_INTERNAL, "stacked-dataset reduction without its pass");
  const double* s1 = seg_slots(sg);
  const double* s2 = s1 + (i64)sg.nseg * sg.nw1 * sg.nc * 2;
  // at least 64 slots a CTA: 8 a thread
  const unsigned z = (unsigned)std::max<i64>(1, std::min<i64>(kSegZ, (sg.nw1 + sg.nw2) / 64));
  auto launch = [&](auto nc) {
    constexpr int NC = decltype(nc)::value;
    k_spmm_seg_reduce<NC><<<dim3(sg.nseg, 2 * NC / 32, z), 256, 0, c->stream>>>(
        s1, sg.nw1, s2, sg.nw2, sg.kout, sg.icpt, sg.out, sg.ldo, sg.gb, sg.grow, sg.ldg, sg.gate, sg.mask,
        sg.mstride, sg.mword, seg_parts(sg), (unsigned*)sg.slots);
  };
  if (sg.nc == 32) launch(std::integral_constant<int, 32>{});
  else if (sg.nc == 64) launch(std::integral_constant<int, 64>{});
  else launch(std::integral_constant<int, 128>{});
  check_launch("k_spmm_seg_reduce");
  count_launch(c);
}

// Multinomial forward pass, K <= 128 classes: P = (softmax(A W + icpt) -
// onehot(label)) * sw, row-major [m][ldp] of the accumulator type; with
// loss_out (device, 2 * K doubles) also the cross-entropy sum in loss_out[0].
void crs_spmm_softmax(fvg_ctx* c, DevCRS& a, int storage, const void* W, i64 ldw, int K, const double* label,
                      const double* sw, const float* label_f, const float* sw_f, int icpt, const double* icpt_v,
                      void* P, i64 ldp, void* scratch, double* loss_out) {
  if (K < 1 || K > kSpmmMaxCols) fail(FVG_ERR_INTERNAL, "softmax block width out of range");
  const Sched& s = pass_sched(c, a, storage);
  SpmmK p = {};
  p.X = W;
  p.ldx = ldw;
  if (ldw > 0x7fffffffll) fail(FVG_ERR_INVALID_ARG, "dense operand row stride beyond 2^31 - 1");
  p.kb = K;
  p.label = label;
  p.sw = sw;
  p.label_f = label_f;
  p.sw_f = sw_f;
  p.icpt = icpt;
  p.bias = icpt_v;
  p.R = P;
  p.ldr = ldp;
  char* sc = (char*)scratch;
  FVG_CUDA(cudaMemsetAsync(sc, 0, 256, c->stream));
  if (storage == FVG_F64) {
    if (!launch_grouped<double, double, double, double, EPI_SOFTMAX>(c, a, s, storage, p, loss_out, nullptr, sc))
      launch_spmm<double, double, double, double, EPI_SOFTMAX, 4>(c, a, s, storage, p, loss_out, nullptr, sc);
  } else if (storage == FVG_F32) {
    if (!launch_grouped<float, float, float, float, EPI_SOFTMAX>(c, a, s, storage, p, loss_out, nullptr, sc))
      launch_spmm<float, float, float, float, EPI_SOFTMAX, 4>(c, a, s, storage, p, loss_out, nullptr, sc);
  } else if (!launch_grouped<bf16, float, float, float, EPI_SOFTMAX>(c, a, s, storage, p, loss_out, nullptr, sc)) {
    launch_spmm<bf16, float, float, float, EPI_SOFTMAX, 4>(c, a, s, storage, p, loss_out, nullptr, sc);
  }
}

// Y = A X, X row-major num_col x k, Y row-major num_row x k, in blocks of 128
// columns.
void crs_spmm(fvg_ctx* c, DevCRS& a, int storage, int x_dt, const void* X, i64 k, void* Y) {
  ProfScope pr(c, P_SPMM);
  if (a.m == 0 || k == 0) return;
  if (storage == FVG_F64 && x_dt != FVG_F64) fail(FVG_ERR_INVALID_ARG, "FP64 values need FP64 vectors");
  DBuf sc;
  sc.alloc((size_t)spmm_scratch_bytes(c, a, storage), c->stream);
  const size_t es = (size_t)dtype_size(x_dt);
  for (i64 c0 = 0; c0 < k; c0 += kSpmmMaxCols) {
    const int kb = (int)std::min<i64>(kSpmmMaxCols, k - c0);
    crs_spmm_block(c, a, storage, (const char*)X + c0 * es, k, kb, x_dt, (char*)Y + c0 * es, k, sc.p);
  }
}

}  // namespace fvg
