// FP64 loss and derivative of a logistic row without the general exp, log and
// division: a warp's FP64 instruction takes its scheduler 64 clocks, and the
// three calls took over 100 of them a row.
//
// exp and log are table driven, after P. T. P. Tang ("Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15(2), 1989; "... of the logarithm function ...", ACM
// TOMS 16(4), 1990); the quotient is Newton's iteration from the logarithm's
// reciprocal with P. Markstein's final correction (IBM J. Res. Dev. 34(1),
// 1990).  The tables hold a high and a low part, computed by the compiler in
// double-double arithmetic.
#pragma once

#include <cstdint>

namespace fvg {
namespace logi {

// ---------------------------------------------- double-double, constant folding
struct DD {
  double h, l;
};
constexpr DD fast_sum(double a, double b) {  // |a| >= |b|
  const double s = a + b;
  return DD{s, b - (s - a)};
}
constexpr DD two_sum(double a, double b) {
  const double s = a + b, v = s - a;
  return DD{s, (a - (s - v)) + (b - v)};
}
constexpr DD two_prod(double a, double b) {  // Dekker's splitting
  const double c = 134217729.0;
  const double ca = c * a, cb = c * b;
  const double ah = ca - (ca - a), al = a - ah, bh = cb - (cb - b), bl = b - bh;
  const double p = a * b;
  return DD{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr DD add(DD a, DD b) {
  const DD s = two_sum(a.h, b.h), t = two_sum(a.l, b.l);
  const DD u = fast_sum(s.h, s.l + t.h);
  return fast_sum(u.h, u.l + t.l);
}
constexpr DD mul(DD a, DD b) {
  const DD p = two_prod(a.h, b.h);
  return fast_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr DD div(DD a, DD b) {
  const double q0 = a.h / b.h;
  const DD r = add(a, mul(DD{-q0, 0.0}, b));
  const double q1 = r.h / b.h;
  const DD r2 = add(r, mul(DD{-q1, 0.0}, b));
  return add(fast_sum(q0, q1), DD{r2.h / b.h, 0.0});
}
// -log(x), 1/2 <= x <= 1, as 2 atanh((1 - x) / (1 + x))
constexpr DD neg_log(double x) {
  const DD y = div(DD{1.0 - x, 0.0}, two_sum(1.0, x)), y2 = mul(y, y);
  DD s{0.0, 0.0};
  for (int k = 35; k >= 0; k--) s = add(mul(s, y2), div(DD{2.0, 0.0}, DD{2.0 * k + 1.0, 0.0}));
  return mul(s, y);
}
constexpr DD exp_series(DD x) {  // 0 <= x < 0.7
  DD s{1.0, 0.0};
  for (int k = 28; k >= 1; k--) s = add(DD{1.0, 0.0}, div(mul(s, x), DD{(double)k, 0.0}));
  return s;
}

constexpr int kBits = 7;  // 128 intervals
constexpr int kN = 1 << kBits;
struct ExpTable {
  double t[kN][2];  // 2^(j / 128)
};
struct alignas(16) LogTable {
  double t[kN + 1][4];  // r = 1 / (1 + j / 128) in eight bits, -log(r) in two parts, unused
};
constexpr DD kLn2 = neg_log(0.5);
constexpr ExpTable exp_table() {
  ExpTable e{};
  for (int j = 0; j < kN; j++) {
    const DD v = exp_series(mul(kLn2, DD{j * (1.0 / kN), 0.0}));
    e.t[j][0] = v.h;
    e.t[j][1] = v.l;
  }
  return e;
}
constexpr LogTable log_table() {
  LogTable g{};
  for (int j = 0; j <= kN; j++) {
    const double r = (double)(int)(256.0 / (1.0 + j * (1.0 / kN)) + 0.5) / 256.0;
    const DD v = neg_log(r);
    g.t[j][0] = r;
    g.t[j][1] = v.h;
    g.t[j][2] = v.l;
  }
  return g;
}
// ln 2 / 128 in two parts, the first of 32 bits: its product with the integer
// quotient is exact
constexpr double kStepHi = (double)(int64_t)(kLn2.h / kN * 549755813888.0) / 549755813888.0;
constexpr double kStepLo = (kLn2.h / kN - kStepHi) + kLn2.l / kN;
constexpr double kInvStep = kN / kLn2.h;

alignas(16) static __device__ const ExpTable d_exp = exp_table();
static __device__ const LogTable d_log = log_table();

// exp(-a), 0 <= a <= 700
__device__ __forceinline__ double exp_neg(double a) {
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the nearest integer
  const double kd = fma(a, -kInvStep, magic);
  const int n = __double2loint(kd);
  const double k = kd - magic;
  const double r = fma(k, -kStepLo, fma(k, -kStepHi, -a));  // |r| <= ln 2 / 256
  const double2 t = __ldg((const double2*)d_exp.t + (n & (kN - 1)));
  double p = fma(r, 1.0 / 120, 1.0 / 24);
  p = fma(p, r, 1.0 / 6);
  p = fma(p, r, 0.5);
  p = fma(p, r * r, r);  // e^r - 1
  const double v = t.x + fma(t.x, p, t.y);
  return __hiloint2double(__double2hiint(v) + ((n >> kBits) << 20), __double2loint(v));
}

// log(u) and num / u, 1 <= u <= 2
__device__ __forceinline__ void log_and_quotient(double u, double num, double& lg, double& q) {
  const unsigned j = min((unsigned)(__double2hiint(u) - 0x3ff00000 + (1 << (19 - kBits))) >> (20 - kBits), (unsigned)kN);
  const double2 rl = __ldg((const double2*)d_log.t[j]);
  const double lo = __ldg(&d_log.t[j][2]);
  const double s = fma(u, rl.x, -1.0);  // u r = 1 + s, |s| <= 2^-7: exact, r has eight bits
  double p = fma(s, -1.0 / 8, 1.0 / 7);
  p = fma(p, s, -1.0 / 6);
  p = fma(p, s, 0.2);
  p = fma(p, s, -0.25);
  p = fma(p, s, 1.0 / 3);
  p = fma(p, s, -0.5);
  const double h = rl.y + s;
  lg = h + ((s - (h - rl.y)) + fma(s * s, p, lo));
  double y = fma(-rl.x, s, rl.x);     // 1 / u to 2^-14
  y = fma(y, fma(-u, y, 1.0), y);     // 2^-28
  y = fma(y, fma(-u, y, 1.0), y);     // FP64
  q = num * y;
  q = fma(fma(-u, q, num), y, q);
}

}  // namespace logi
}  // namespace fvg
