// pa_sincos.cuh -- FP64 sine and cosine for the FP64 forms, whose kernels the
// FP64 pipe bounds (2 lanes per clock and SM: every FP64 instruction of a warp
// holds it for 16 clocks).
//
// x = k (2 pi / 256) + r, |r| <= pi / 256: k by adding and subtracting 1.5 2^52,
// r by two fused multiply-adds with 2 pi / 256 as the sum of two doubles (Cody
// and Waite).  sin r and cos r - 1 are their Taylor sums to r^7 and r^6 (the rest
// is below 1e-21 of r and 2e-20); the angle sum with sin and cos of k (2 pi /
// 256), from a table of two doubles each, makes 18 FP64 operations, where the
// library's sincos takes more than twice as many.  Against 113-bit values, 10^6
// arguments up to 2^25: at most 5.8e-17 and 2.7e-17 rms (0.29 units in the last
// place rms); the library's 1.3e-16 and 3.2e-17 (0.36).  Pass A of the FP64
// search, two detectors, N = 43082: 15.1 -> 14.0 us a spindown; FP64 followup,
// 100 points of N = 86164: 2.39 -> 2.12 ms.
// Larger |x|, infinities and NaN go to the library's.
#pragma once
#include <cuda_runtime.h>

namespace pa {

struct TrigEntry {
  double s, c, sl, cl;  // sin and cos of k (2 pi / 256), and what their doubles leave
};
struct TrigTab {
  TrigEntry e[256];
};

// Sums and products of two doubles each, exact to about 2^-104 (Dekker, Knuth),
// for the compiler to form the table with.
namespace trig_detail {
struct DD {
  double h, l;
};
constexpr DD norm(double a, double b) {
  const double s = a + b;
  return DD{s, b - (s - a)};
}
constexpr DD sum(double a, double b) {
  const double s = a + b, bb = s - a;
  return DD{s, (a - (s - bb)) + (b - bb)};
}
constexpr DD prod(double a, double b) {
  const double p = a * b;
  const double ta = 134217729.0 * a, ah = ta - (ta - a), al = a - ah;
  const double tb = 134217729.0 * b, bh = tb - (tb - b), bl = b - bh;
  return DD{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr DD add(DD a, DD b) {
  const DD s = sum(a.h, b.h);
  return norm(s.h, s.l + (a.l + b.l));
}
constexpr DD mul(DD a, DD b) {
  const DD p = prod(a.h, b.h);
  return norm(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr DD div(DD a, double b) {  // b a small integer
  const double q = a.h / b;
  const DD p = prod(q, b);
  return norm(q, ((a.h - p.h) - p.l + a.l) / b);
}
// x^first/first! - x^(first+2)/(first+2)! + ...
constexpr DD series(DD x, int first) {
  DD t{1., 0.};
  for (int j = 1; j <= first; ++j) t = div(mul(t, x), (double)j);
  DD s = t;
  const DD x2 = mul(x, x);
  for (int j = first + 2; j <= first + 28; j += 2) {
    t = div(mul(t, x2), -(double)((j - 1) * j));
    s = add(s, t);
  }
  return s;
}
constexpr TrigTab make() {
  TrigTab t{};
  for (int k = 0; k < 256; ++k) {
    // within an eighth of a turn of the nearest quarter, where the series and
    // the signs are exact
    const int q = ((k + 32) / 64) & 3, m = k - 64 * ((k + 32) / 64);
    const DD x = div(mul(DD{3.141592653589793116, 1.2246467991473531772e-16}, DD{(double)m, 0.}), 128.);
    const DD s = series(x, 1), c = series(x, 0);
    const DD ns{-s.h, -s.l}, nc{-c.h, -c.l};
    const DD sn = q == 0 ? s : (q == 1 ? c : (q == 2 ? ns : nc));
    const DD cs = q == 0 ? c : (q == 1 ? ns : (q == 2 ? nc : s));
    t.e[k].s = sn.h;
    t.e[k].sl = sn.l;
    t.e[k].c = cs.h;
    t.e[k].cl = cs.l;
  }
  return t;
}
constexpr TrigTab kTab = make();
}  // namespace trig_detail

static __device__ const __align__(16) TrigTab c_trig = trig_detail::kTab;

// (a call: the compiler would issue a rare branch's FP64 operations for every
// number)
static __device__ __noinline__ void sincos_any(double x, double* s, double* c) { sincos(x, s, c); }

__device__ __forceinline__ void sincos_fast(double x, double* s, double* c) {
  if (((unsigned)__double2hiint(x) & 0x7fffffffu) >= 0x41800000u) {  // |x| >= 2^25, NaN
    sincos_any(x, s, c);
    return;
  }
  constexpr double kInv = 40.74366543152521;                             // 256 / 2 pi
  constexpr double kStep = 0.02454369260617026;                         // 2 pi / 256
  constexpr double kStepLo = 9.567553118338697e-19;                     // its rest
  const double t = fma(x, kInv, 6755399441055744.0);                    // 1.5 2^52
  const double k = t - 6755399441055744.0;
  const double2* e = reinterpret_cast<const double2*>(&c_trig.e[__double2loint(t) & 255]);
  const double2 hi = __ldg(e), lo = __ldg(e + 1);
  double r = fma(-k, kStep, x);
  r = fma(-k, kStepLo, r);
  const double r2 = r * r;
  const double sr = fma(r2 * r, fma(r2, fma(r2, -1. / 5040., 1. / 120.), -1. / 6.), r);
  const double cm = r2 * fma(r2, fma(r2, -1. / 720., 1. / 24.), -.5);
  *s = hi.x + fma(hi.y, sr, fma(hi.x, cm, lo.x));
  *c = hi.y + fma(-hi.x, sr, fma(hi.y, cm, lo.y));
}

}  // namespace pa
