// Device helpers shared by the product kernels: fixed-order block sums,
// compensated accumulators, the per-row logistic loss/gradient and value
// widening.
#pragma once

#include "fvg_internal.cuh"
#include "logistic64.cuh"

namespace fvg {

template <class T> __device__ __forceinline__ T block_sum256(T v) {
  __shared__ T red[8];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  T t = 0;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 8; q++) t += red[q];
  }
  return t;  // valid in thread 0
}

// ---------------------------------------------------- Euclidean norms
// The reference scales by the largest magnitude first (vector_operations.hpp:
// 227-264), which takes two passes.  Here the squares are summed in three
// ranges whose scaling (a power of two, exact) keeps them within FP64, after
// J. L. Blue ("A portable Fortran program to find the Euclidean norm of a
// vector", ACM TOMS 4(1), 1978): the exponent picks the range, one fused
// multiply-add per element.  An infinity makes the norm NaN, and so does a NaN
// beside an element other than 0; with zeros only it leaves 0 (the largest
// magnitude ignores it).
__device__ __forceinline__ void norm_add(double& tiny, double& mid, double& huge, double g) {
  const int ex = (__double2hiint(g) >> 20) & 0x7ff;  // biased exponent
  if (ex >= 1023 - 480 && ex <= 1023 + 480) {
    mid = fma(g, g, mid);
  } else if (ex < 1023 - 480) {
    const double x = g * 0x1p+600;
    tiny = fma(x, x, tiny);
  } else if (ex < 0x7ff) {
    const double x = g * 0x1p-600;
    huge = fma(x, x, huge);
  } else {
    huge += g - g;          // NaN
    if (g == g) mid += 1.0;  // an infinity: an element other than 0
  }
}
__device__ __forceinline__ double norm_of(double tiny, double mid, double huge) {
  if (huge != huge) return tiny > 0.0 || mid > 0.0 ? huge : 0.0;
  if (huge > 0.0) return sqrt(huge + mid * 0x1p-600 * 0x1p-600) * 0x1p+600;
  if (mid > 0.0) return sqrt(mid + tiny * 0x1p-600 * 0x1p-600);
  return sqrt(tiny) * 0x1p-600;
}

// ---------------------------------------------------- compensated sums
// Neumaier, FP64 (the FP64 path).  The larger summand is told by the high
// words: with equal exponents either order leaves the same remainder.  Four
// FP64 instructions and no branch, where an FP64 comparison and two branches
// made it up to eight: 1,000,000 hinge rows 42 us instead of 52, logistic
// rows 111 instead of 119.
struct CSum {
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double v) {
    const double t = s + v;
    const bool sb = (__double2hiint(s) & 0x7fffffff) >= (__double2hiint(v) & 0x7fffffff);
    const double big = sb ? s : v, small = sb ? v : s;
    c += (big - t) + small;
    s = t;
  }
  __device__ __forceinline__ double total() const { return s + c; }
};
struct FSum {  // Kahan in FP32 (the FP32-arithmetic path keeps the FP64 unit idle)
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double total() const { return (double)s - (double)c; }
};
template <class AT> struct SumOf { using type = CSum; };
template <> struct SumOf<float> { using type = FSum; };

// Fixed-order block reduction of two compensated sums (256 threads).
__device__ __forceinline__ void block_csum2(double a, double b, double* out_a, double* out_b) {
  __shared__ double ra[256], rb[256];
  __syncthreads();
  ra[threadIdx.x] = a;
  rb[threadIdx.x] = b;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      ra[threadIdx.x] += ra[threadIdx.x + st];
      rb[threadIdx.x] += rb[threadIdx.x + st];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *out_a = ra[0];
    *out_b = rb[0];
  }
}

// ------------------------------------------------------- logistic math
// logistic_gradient<T>::compute_dloss for one row (gradient.hpp:24-50) in
// FP64 with one exponential, e = exp(-|z|): between the reference's
// thresholds log(1 + exp(-z)) = log(1 + e) (+ |z| when z < 0) and
// 1 / (1 + exp(z)) = e / (1 + e) (z > 0) or 1 / (1 + e).  GB300's FP64 unit
// makes every FP64 instruction count (two exponentials and FP64 range tests:
// 1.6x the time of this form), so the rarely met ranges are recognised from
// the high word and tested exactly only there (NaN included).
__device__ __forceinline__ bool dbl_at_least(double v, int hi) {  // |v|'s high word >= hi
  return (__double2hiint(v) & 0x7fffffff) >= hi;
}
__device__ __forceinline__ void logistic_row(double wtx, double lab, double& loss, double& d) {
  const double z = lab * wtx;
  const double neg = -lab;
  const double az = __hiloint2double(__double2hiint(z) & 0x7fffffff, __double2loint(z));
  const double e = dbl_at_least(az, 0x4085e000) ? exp(-az) : logi::exp_neg(az);  // 700 and above
  const bool up = __double2hiint(z) >= 0;  // z >= 0
  if (dbl_at_least(z, 0x40320000) && z > 18.0) {
    loss = e;
    d = e * neg;
  } else if (dbl_at_least(z, 0x40320000) && z < -18.0) {
    loss = az;
    d = neg;
  } else {
    double q;
    logi::log_and_quotient(1.0 + e, up ? e : 1.0, loss, q);
    if (!up) loss += az;
    d = neg * q;
  }
  if (dbl_at_least(d, 0x426d1a94)) {  // 1e12 and above
    if (d > 1e12) d = 1e12;
    else if (d < -1e12) d = -1e12;
  }
}
// FP32 variant for the BF16/FP32-storage path (log1p form keeps small
// losses that log(1+e) would round away in single precision).
__device__ __forceinline__ void logistic_row(float wtx, float lab, float& loss, float& d) {
  float z = lab * wtx;
  float neg = -lab;
  if (z > 18.0f) {
    float e = expf(-z);
    loss = e;
    d = e * neg;
  } else if (z < -18.0f) {
    loss = -z;
    d = neg;
  } else {
    loss = log1pf(expf(-z));
    d = neg / (1.0f + expf(z));
  }
  if (d > 1e12f) d = 1e12f;
  else if (d < -1e12f) d = -1e12f;
}

// The FP32 logistic row of the multi-model products with one exponential:
// e = exp(-|z|), 1 / (1 + exp(z)) = (z > 0 ? e : 1) / (1 + e) and
// log(1 + exp(-z)) = max(-z, 0) + log1p(e).  Every branch of
// gradient.hpp:24-50 is the same function: beyond |z| = 18 the reference's
// e and -z differ from these forms by less than e / 2 relative (below FP32
// resolution), so the result differs from logistic_row(float) by rounding.
__device__ __forceinline__ void logistic_row_1exp(float wtx, float lab, float& loss, float& d) {
  const float z = lab * wtx;
  const float e = expf(-fabsf(z));
  loss = fmaxf(-z, 0.0f) + log1pf(e);
  d = -lab * __fdividef(z > 0.0f ? e : 1.0f, 1.0f + e);
  if (d > 1e12f) d = 1e12f;
  else if (d < -1e12f) d = -1e12f;
}

// ------------------------------------------------------ GLM loss kinds
// compute_dloss of the GLM family for one row (ml/glm/gradient.hpp):
// 0 logistic_gradient, 1 linear_gradient (55-87), 2 hinge_gradient
// (89-121), 3 epsilon_insensitive (123-159), 4 squared_epsilon_insensitive
// (161-202).  MAX_LOSS / MIN_LOSS clip at ±1e12, HINGE_THRESHOLD = 1
// (gradient.hpp:8-10).  The squared loss comes back halved per row: the
// reference halves a rank's sum (70-73) and scaling by 0.5 is exact, so the
// halves add up to the same value.  The kind is uniform across a launch.
enum GlmLossKind { LOSS_LOGISTIC = 0, LOSS_SQUARED = 1, LOSS_HINGE = 2, LOSS_EPS = 3, LOSS_SQEPS = 4 };

template <class AT> __device__ __forceinline__ AT clip_dloss(AT d) {
  return d > (AT)1e12 ? (AT)1e12 : (d < (AT)-1e12 ? (AT)-1e12 : d);
}

template <class AT>
__device__ __forceinline__ void glm_row(int kind, AT eps, AT wtx, AT lab, AT& loss, AT& d) {
  if (kind == LOSS_LOGISTIC) {
    logistic_row(wtx, lab, loss, d);
  } else if (kind == LOSS_SQUARED) {
    const AT e = wtx - lab;
    loss = (AT)0.5 * (e * e);
    d = clip_dloss(e);
  } else if (kind == LOSS_HINGE) {
    const AT z = wtx * lab;
    const bool in = z <= (AT)1;
    loss = in ? (AT)1 - z : (AT)0;
    d = in ? -lab : (AT)0;
  } else {
    const AT z = lab - wtx;  // positive: the prediction is below the label
    const AT e = fabs(z) - eps;
    if (kind == LOSS_EPS) {
      loss = e > 0 ? e : (AT)0;
      d = z > eps ? (AT)-1 : ((wtx - lab) > eps ? (AT)1 : (AT)0);
    } else {
      loss = e > 0 ? e * e : (AT)0;
      d = z > eps ? (AT)-2 * (z - eps) : (z < -eps ? (AT)2 * (-z - eps) : (AT)0);
      d = clip_dloss(d);
    }
  }
}

template <class VT> __device__ __forceinline__ float to_f(VT v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }

template <class VT, class AT> __device__ __forceinline__ AT to_acc(VT v) { return (AT)to_f<VT>(v); }
template <> __device__ __forceinline__ double to_acc<double, double>(double v) { return v; }

// Streaming (evict-first) load of one value, widened to the accumulator.
template <class VT, class AT> __device__ __forceinline__ AT ld_val(const VT* q);
template <> __device__ __forceinline__ double ld_val<double, double>(const double* q) { return __ldcs(q); }
template <> __device__ __forceinline__ float ld_val<float, float>(const float* q) { return __ldcs(q); }
template <> __device__ __forceinline__ float ld_val<bf16, float>(const bf16* q) {
  return __uint_as_float((unsigned)__ldcs(reinterpret_cast<const unsigned short*>(q)) << 16);
}

}  // namespace fvg
