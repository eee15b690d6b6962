// pa_followup_f32.cuh -- the followup's sums in the mixed form (FP32 sums, the
// phase in 64-bit fixed point), included by pa_followup.cu only.
//
// For a point (f, s, delta, alpha) and a detector at R(i) the phase in turns is
//   [f i + s i^2]/2pi + (f + oms + 2 s i)/2pi shft(i),   shft = n . R(i).
// A GB300 runs FP64 at 1/64 of the FP32 rate; with shft and the last product in
// FP64 per point and sample the kernel was held by that pipe (5 operations
// each: 10.4 ms for 4096 points of three detectors, N = 86164).  Here a chunk
// of 1024 samples from sample b on has R(b + j) = R0 + V j + A j^2 + r(j) with
// FP64 R0, V, A (the parabola through its first, middle and last sample, formed
// once on the host) and an FP32 rest r, which the smooth motion of a detector
// leaves at 1e-6 and less.  The phase of the chunk is then, exactly,
//   P0 + P1 j + P2 j^2 + W n.r + (2 s/2pi) j (n.r + n.A j^2),   W = (f + oms + 2 s b)/2pi,
// with P0, P1, P2 in 64-bit fixed point from FP64 values of the point and chunk
// (17 FP64 operations per 1024 samples), advanced from sample to sample by
// integer additions, and a last part of less than 2^-8 turns in FP32, whose
// rounding is below that of the angle itself.  Where W n.r is more than that, it
// is formed from integer rests, or in FP64 per sample (form_of).
//
// The amplitude modulations are a = sum_k A_k u_k(i), b = sum_k B_k u_k(i) with
// u = (1, cos w, sin w, cos 2w, sin 2w), w = omr i, and five coefficients per
// point and detector.  The sums are taken over x u_k, the same for all points:
//   U_k = sum x u_k cos(phase),  W_k = sum x u_k sin(phase),
// so that Xa = sum_k A_k (U_k - i W_k), Xb likewise, and sum a^2 = A.G.A with
// the FP64 matrix G of the u_k (no sum over samples).  The adjoint needs, beside
// these, the moments of the phase's gradient g(i) = x (ka a Im_a + kb b Im_b):
// sum g j^m (m <= 3) and sum g r, per chunk; the derivatives of all four
// parameters follow from them in FP64, about a centre of time and position: sum g
// is 0 (Im conj(X) X), so that its rounding need not be multiplied by either.
//
// What bounds it: per sample of two points 26 packed-FP32 operations (two cycles
// a warp and scheduler each) and 2 x 15 integer ones on the half-rate ALU (two
// cycles each), about 56 cycles on either pipe, so that both run beside each
// other.  4096 points of three detectors, N = 86164: F 11.04 -> 1.71 ms, F and
// gradient 21.8 -> 3.76 ms (F: issue slots 64 % busy, FMA pipe 57 %, ALU 50 %; the
// adjoint 63, 60 and 39 %); 81 points of two detectors, N = 43082: 172 -> 79 us.
// F errs by 3.8e-8 against 64 bits where the FP64 phase per sample had 4.3e-8, the
// gradient by 4.5e-8 (6.2e-8 without the centre, 7e-8 per sample).
#pragma once
#include <stdint.h>

#include "pa_f32x2.cuh"

namespace fu32 {

using pa::add2;
using pa::dup;
using pa::f2;
using pa::fma2;
using pa::mul2;
using pa::pk;
using pa::upk;

constexpr int kChunk = 1024;
constexpr int kThreads = 256;
constexpr int kU = 5;                      // functions u_k
// floats per point and chunk: U, W; moments of g {sum g j^0..3, g r, (rough) g j
// r_0}, and after those of all points two more, {(rough) g j r_1, g j r_2}
constexpr int kPartF = 2 * kU, kPartA = 8, kPartA2 = 2;
// most of each term of the FP32 part of the phase, in turns (two of them: the
// sine's polynomial is used on pi/4 + 0.0245 rad)
constexpr double kMaxRest = 1. / 512.;
// most of W n.r, in turns, that the integer rests hold (30 bits: 64 turns to 6e-8)
constexpr double kMaxTurns = 64.;

// What the form of the phase is chosen by: the largest |r| and |A| (NaN: some
// position is) and whether sum g j r is below the rounding of sum g i R
// (k_final_adj).
struct Bounds {
  double rest, curv;
  int adj_fast, pad;
};

// The motion of a detector over a chunk from sample b on; unit: of the integer
// rests; b - ic, b^2 - ic^2, R0 - Rc and b R0 - ic Rc with the centre (ic, Rc).
struct Chunk {
  double R0[3], V[3], A[3];
  double unit, db, db2, dR[3], dbR[3];
  Bounds top;
};

// The sample and the position that the adjoint's sums are taken from: sum g is 0
// over all samples and detectors (Im conj(X) X), so that any constant may be
// taken off i and R, and with these the rounding of g is not multiplied by a
// time of N samples and the distance of the Sun.
struct Centre {
  double i, R[3];
};

// The form of the phase of a point over a chunk (the same operations wherever it
// is asked for; larger |f + oms|, |s| or bounds never give a faster form):
//   fast   W n.r and the j^3 term in FP32
//   rough  W n.r by 32-bit integer rests, the j^3 term and W's change in FP32;
//          the adjoint adds sum g j r
//   slow   FP64 per sample
// Rough costs six integer multiplications a sample and point more.  It is for
// positions that a parabola over 1024 samples leaves too far behind (dt = 8 s
// above 63 Hz, dt = 4 s above 500 Hz, an ephemeris that is not smooth) and for
// the adjoint of short data; slow for jumps of 64 turns, NaN and spindowns of
// more than 1e-2 rad a sample^2.  1024 points of two detectors, N = 10771, dt = 8
// s, 100 Hz, F and gradient: rough 123 and 235 us, slow 365 and 1361 us (fast, at
// 30 Hz: 103 and 182 us); 43082 samples of three at dt = 4 s, 1 kHz: 382 and 840 us,
// slow 1593 and 7040 us.
enum { kSlow = 0, kRough = 1, kFast = 2 };
__host__ __device__ __forceinline__ double mul_rn(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;  // (host code is built without contraction)
#endif
}
__host__ __device__ __forceinline__ int form_of(double fo, double st2, const Bounds& h, int N, bool adj) {
  const double s2 = fabs(st2), t = mul_rn(fma(s2, (double)N, fabs(fo)), h.rest);
  if (!(mul_rn(mul_rn(s2, h.curv), (double)kChunk * kChunk * kChunk) <= kMaxRest)) return kSlow;
  if (t <= kMaxRest && (!adj || h.adj_fast)) return kFast;
  return t <= kMaxTurns && mul_rn(mul_rn(s2, h.rest), (double)kChunk) <= kMaxRest ? kRough : kSlow;
}

struct Gram {
  double g[kU][kU];  // sum_i u_k(i) u_l(i)
};

// Per-point constants (the phase and its derivatives in FP64).
struct Point {
  double f, s, fo, st2;          // f, s; (f + oms)/2pi, 2s/2pi
  double n[3], nD[3], nA[3];     // source vector, its derivatives by delta and alpha
  unsigned long long ffx, sfx;   // f/2pi, s/2pi in 64-bit fixed-point turns
  double A, B;                   // sum a^2/sig2, sum b^2/sig2
  double dA[2], dB[2];           // their derivatives by delta, alpha
  double xr, xi, yr, yi;         // Xa, Xb of the last forward pass
  double ka, kb, qa, qb;         // factors of dF/dX, dF/dA (adjoint)
  int active, fast;              // fast: over every chunk, forward and adjoint
};

// coefficients per point and detector: A, B, dA/ddelta, dB/ddelta
constexpr int kCoef = 4 * kU;

// d/dalpha of the five coefficients q (the angle enters as alpha - w)
__device__ __forceinline__ void d_alpha(const double* q, double* o) {
  o[0] = 0.;
  o[1] = -q[2];
  o[2] = q[1];
  o[3] = -2. * q[4];
  o[4] = 2. * q[3];
}

// v = G q
__device__ __forceinline__ void gram_mul(const Gram& G, const double* q, double* v) {
#pragma unroll
  for (int k = 0; k < kU; k++) {
    v[k] = G.g[k][0] * q[0];
#pragma unroll
    for (int l = 1; l < kU; l++) v[k] = fma(G.g[k][l], q[l], v[k]);
  }
}
__device__ __forceinline__ double dot5(const double* p, const double* v) {
  return fma(p[0], v[0], p[1] * v[1]) + fma(p[2], v[2], fma(p[3], v[3], p[4] * v[4]));
}

// a = k0 (2c^2 - 1) + k1 2cs + k2 c + k3 s + q0 with c, s = cos, sin(beta - w)
// as coefficients of u
__device__ __forceinline__ void harmonics(double k0, double k1, double k2, double k3, double q0, double cb, double sb,
                                          double* q) {
  const double c2 = cb * cb - sb * sb, s2 = 2. * sb * cb;
  q[0] = q0;
  q[1] = k2 * cb + k3 * sb;
  q[2] = k2 * sb - k3 * cb;
  q[3] = k0 * c2 + k1 * s2;
  q[4] = k0 * s2 - k1 * c2;
}

// Point set-up; with a mask, the active points into list[0 .. *nlist).  Eight
// lanes a point, lane d taking detector d (one after the other their FP64
// chains took 25 us of a call of a few points).  GRAD: also what the adjoint
// needs.
template <bool GRAD>
__global__ void __launch_bounds__(64) k_prep(const double* __restrict__ pts, int n,
                                             const unsigned char* __restrict__ mask, Point* __restrict__ point,
                                             double* __restrict__ coef, FuDets dets, Gram G, int nifo, double oms,
                                             Bounds top, int N, int* __restrict__ list,
                                             int* __restrict__ nlist) {
  static_assert(PA_MAX_DETECTORS == 8, "eight lanes a point");
  const int d = threadIdx.x & 7;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  // (whole warps stay for the shuffles; lanes of no point repeat the last one)
  const bool live = k < n && (!mask || mask[k]);
  const int kk = min(k, n - 1);
  const double f = pts[4 * kk + 0], s = pts[4 * kk + 1], de = pts[4 * kk + 2], al = pts[4 * kk + 3];
  // (odd lanes take delta's, even ones alpha's)
  double s_, c_;
  sincos((d & 1) ? de : al, &s_, &c_);
  const double so = __shfl_xor_sync(0xffffffffu, s_, 1), co = __shfl_xor_sync(0xffffffffu, c_, 1);
  const double sa = (d & 1) ? so : s_, ca = (d & 1) ? co : c_, sd = (d & 1) ? s_ : so, cd = (d & 1) ? c_ : co;
  // A, B and their derivatives by delta, alpha: sums over the detectors
  double o6[6] = {0., 0., 0., 0., 0., 0.};
  const double c2d = cd * cd, w2 = 2. - c2d, sc = sd * cd, dw2 = 2. * sc, dsc = cd * cd - sd * sd;
  if (d < nifo) {
    const double* K = dets.d[d].amod;
    const double cb = ca * dets.d[d].cphir + sa * dets.d[d].sphir;
    const double sb = sa * dets.d[d].cphir - ca * dets.d[d].sphir;
    const double is2 = dets.d[d].inv_sig2;
    double q[kCoef], o[kU];
    harmonics(K[0] * w2, K[1] * w2, K[2] * sc, K[3] * sc, K[4] * c2d, cb, sb, q);
    harmonics(K[5] * sd, K[6] * sd, K[7] * cd, K[8] * cd, 0., cb, sb, q + kU);
    double va[kU], vb[kU];
    gram_mul(G, q, va);
    gram_mul(G, q + kU, vb);
    o6[0] = is2 * dot5(q, va);
    o6[1] = is2 * dot5(q + kU, vb);
    if (GRAD) {
      harmonics(K[0] * dw2, K[1] * dw2, K[2] * dsc, K[3] * dsc, -K[4] * dw2, cb, sb, q + 2 * kU);
      harmonics(K[5] * cd, K[6] * cd, -K[7] * sd, -K[8] * sd, 0., cb, sb, q + 3 * kU);
      o6[2] = 2. * is2 * dot5(q + 2 * kU, va);
      o6[3] = 2. * is2 * dot5(q + 3 * kU, vb);
      d_alpha(q, o);
      o6[4] = 2. * is2 * dot5(o, va);
      d_alpha(q + kU, o);
      o6[5] = 2. * is2 * dot5(o, vb);
    }
    if (live) {
      double* Q = coef + ((size_t)k * nifo + d) * kCoef;
#pragma unroll
      for (int t = 0; t < (GRAD ? kCoef : 2 * kU); t++) Q[t] = q[t];
    }
  }
#pragma unroll
  for (int t = 0; t < (GRAD ? 6 : 2); t++)
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) o6[t] += __shfl_xor_sync(0xffffffffu, o6[t], off);
  if (d || k >= n) return;
  if (!live) {
    point[k].active = 0;
    return;
  }
  Point c;
  c.active = 1;
  c.f = f;
  c.s = s;
  c.fo = (f + oms) * kInv2Pi;
  c.st2 = 2. * s * kInv2Pi;
  c.ffx = fu_turns_fixed(f * kInv2Pi);
  c.sfx = fu_turns_fixed(s * kInv2Pi);
  c.n[0] = ca * cd;
  c.n[1] = sa * cd;
  c.n[2] = sd;
  c.nD[0] = -ca * sd;
  c.nD[1] = -sa * sd;
  c.nD[2] = cd;
  c.nA[0] = -sa * cd;
  c.nA[1] = ca * cd;
  c.nA[2] = 0.;
  c.fast = form_of(c.fo, c.st2, top, N, true) == kFast;
  c.A = o6[0];
  c.B = o6[1];
  c.dA[0] = o6[2];
  c.dB[0] = o6[3];
  c.dA[1] = o6[4];
  c.dB[1] = o6[5];
  c.xr = c.xi = c.yr = c.yi = c.ka = c.kb = c.qa = c.qb = 0.;
  point[k] = c;
  if (list) list[atomicAdd(nlist, 1)] = k;
}

// The points selected by need[] into list[0 .. *nlist).
__global__ void k_list(const unsigned char* __restrict__ need, int n, int* __restrict__ list, int* __restrict__ nlist) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n && need[k]) list[atomicAdd(nlist, 1)] = k;
}

// Phase of one point over a chunk; rough form: 2 pi W is left out of w, and W n_k
// unit in 64-bit fixed-point turns, mh 2^32 + ml with a signed ml.
struct Phase {
  unsigned long long P0, P1, P2;  // turns 2^64, with an eighth of a turn added to P0
  int mh[3], ml[3];
  float w, dw, c3, n[3];          // radians: 2 pi W, its step over 32 samples, j^3 term; source vector
};

__device__ __forceinline__ void chunk_phase(const Point& c, const Chunk& h, int base, Phase* o) {
  const double b = (double)base;
  const double W = fma(c.st2, b, c.fo);
  const double S = fma(c.n[0], h.R0[0], fma(c.n[1], h.R0[1], c.n[2] * h.R0[2]));
  const double v = fma(c.n[0], h.V[0], fma(c.n[1], h.V[1], c.n[2] * h.V[2]));
  const double a = fma(c.n[0], h.A[0], fma(c.n[1], h.A[1], c.n[2] * h.A[2]));
  const unsigned long long ub = (unsigned long long)base;
  o->P0 = c.ffx * ub + c.sfx * (ub * ub) + fu_turns_fixed(W * S) + (1ull << 61);
  o->P1 = c.ffx + 2 * c.sfx * ub + fu_turns_fixed(fma(W, v, c.st2 * S));
  o->P2 = c.sfx + fu_turns_fixed(fma(W, a, c.st2 * v));
  const float twopi = 6.283185307179586f;
  const float st = (float)c.st2 * twopi;
  o->w = (float)W * twopi;
  o->dw = st * 32.f;
  o->c3 = st * (float)a;
#pragma unroll
  for (int t = 0; t < 3; t++) o->n[t] = (float)c.n[t];
}
__device__ __forceinline__ void chunk_rough(const Point& c, const Chunk& h, int base, Phase* o) {
  const double W = fma(c.st2, (double)base, c.fo);
  o->w = 0.f;
#pragma unroll
  for (int t = 0; t < 3; t++) {
    const unsigned long long m = fu_turns_fixed(W * c.n[t] * h.unit);
    o->ml[t] = (int)(unsigned)m;
    o->mh[t] = (int)(unsigned)(m >> 32) + (o->ml[t] < 0 ? 1 : 0);
  }
}

// sine and cosine of (quadrant, angle) pairs of two points: polynomials fitted on
// |x| <= 0.8 (least squares, weighted again and again by the error itself towards
// the least largest one).  With their FP32 coefficients they err by 5e-9 and 2e-9
// there and by 7e-9 up to 0.81, where two terms of kMaxRest lead; 4e-8 and 5e-8
// with FP32 arithmetic
__device__ __forceinline__ void sincos2(f2 x, unsigned qa, unsigned qb, f2* sn, f2* cs) {
  const f2 z = mul2(x, x);
  const f2 s = fma2(mul2(x, z), fma2(z, fma2(z, dup(-1.948277497e-4f), dup(8.331875317e-3f)), dup(-1.666664928e-1f)), x);
  const f2 c = fma2(
      z, fma2(z, fma2(z, fma2(z, dup(2.437514377e-5f), dup(-1.388660166e-3f)), dup(4.166661948e-2f)), dup(-0.5f)), dup(1.f));
  float sa, sb, ca, cb;
  upk(s, sa, sb);
  upk(c, ca, cb);
  auto turn = [](unsigned q, float s_, float c_, float* so, float* co) {
    const bool swap = (q & 0x40000000u) != 0u;
    *so = __uint_as_float(__float_as_uint(swap ? c_ : s_) ^ (q & 0x80000000u));
    *co = __uint_as_float(__float_as_uint(swap ? s_ : c_) ^ ((q ^ (q << 1)) & 0x80000000u));
  };
  turn(qa, sa, ca, &sa, &ca);
  turn(qb, sb, cb, &sb, &cb);
  *sn = pk(sa, sb);
  *cs = pk(ca, cb);
}

// Sum over the warp of eight values per lane; the sum of value
// warp_sum8_index(lane) is returned (the same in the four lanes of a group).
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane) {
#pragma unroll
  for (int off = 16, m = 4; off >= 4; off >>= 1, m >>= 1) {
    const bool hi = (lane & off) != 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k < m) {
        const float send = hi ? v[2 * k] : v[2 * k + 1], keep = hi ? v[2 * k + 1] : v[2 * k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
  }
  float t = v[0];
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  return t;
}
__device__ __forceinline__ int warp_sum8_index(int lane) {
  return ((lane >> 4) & 1) | ((lane >> 2) & 2) | (lane & 4);
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The sums of one point over a chunk in the slow form: forward U, W as the
// others; adjoint the four derivatives' phase parts, from the centre.
template <bool ADJ>
__device__ __noinline__ void sums_slow(const Point& c, const float* __restrict__ seeds, const double* __restrict__ pos,
                                       const float4* s0, const float4* s1, int base, int cnt, const Centre& ctr, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  float acc[2 * kU] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  double g4[4] = {0., 0., 0., 0.};
  auto dot = [](const double* n, double x, double y, double z) { return n[0] * x + n[1] * y + n[2] * z; };
  const double hc = ctr.i + dot(c.n, ctr.R[0], ctr.R[1], ctr.R[2]), h2c = (2. * hc - ctr.i) * ctr.i;
  const double omc = (c.fo + c.st2 * ctr.i) * 6.283185307179586476925286766559;
  const double dc = omc * dot(c.nD, ctr.R[0], ctr.R[1], ctr.R[2]), ac = omc * dot(c.nA, ctr.R[0], ctr.R[1], ctr.R[2]);
  for (int j = lane; j < cnt; j += 32) {
    const int i = base + j;
    const double di = (double)i, r0 = pos[3 * (size_t)j], r1 = pos[3 * (size_t)j + 1], r2 = pos[3 * (size_t)j + 2];
    const double shft = dot(c.n, r0, r1, r2);
    const unsigned long long ui = (unsigned long long)i;
    const unsigned long long t = c.ffx * ui + c.sfx * (ui * ui) + fu_turns_fixed(fma(c.st2, di, c.fo) * shft);
    float sn, co;
    sincospif((float)(int)(t >> 32) * 4.656612873077393e-10f, &sn, &co);
    const float4 p = s0[j], q = s1[j];
    const float xu[kU] = {p.x, p.y, p.z, p.w, q.x};
    if (!ADJ) {
#pragma unroll
      for (int k = 0; k < kU; k++) {
        acc[k] += co * xu[k];
        acc[kU + k] += sn * xu[k];
      }
    } else {
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int k = 0; k < kU; k++) {
        a += seeds[k] * xu[k];
        b += seeds[kU + k] * xu[k];
      }
      const double g = (double)(a * co + b * sn);
      const double om = (c.fo + c.st2 * di) * 6.283185307179586476925286766559;
      g4[0] += g * (di + shft - hc);
      g4[1] += g * (di * di + 2. * di * shft - h2c);
      g4[2] += g * (om * dot(c.nD, r0, r1, r2) - dc);
      g4[3] += g * (om * dot(c.nA, r0, r1, r2) - ac);
    }
  }
  if (!ADJ) {
#pragma unroll
    for (int k = 0; k < 2 * kU; k++) {
      float v = acc[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) out[k] = v;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double v = warp_sum_d(g4[k]);
      if (lane == 0) reinterpret_cast<double*>(out)[k] = v;
    }
  }
}

// The sums of 2 NPK points (places w0 on) over a chunk in the fast or the rough
// form, a warp's lanes over the samples, two points in the halves of packed
// registers.  What belongs to points of another form is computed and not written.
template <bool ADJ, bool ROUGH, int NPK>
__device__ __forceinline__ void sums_fp32(const float4* s0, const float4* s1, const int* ri, const Phase* ph,
                                          const int* idx, const int* form, const float* __restrict__ seeds,
                                          int w0, int cnt, int n, int nifo, int d, int P, int p, float* __restrict__ part) {
  constexpr int NP = 2 * NPK;
  const int lane = threadIdx.x & 31;
  unsigned long long t[NP], dt[NP], ddt[NP];
  f2 nv[NPK][3], w[NPK], dw[NPK], c3[NPK];
  f2 al[ADJ ? kU : 1], be[ADJ ? kU : 1];
  int mh[ROUGH ? NP : 1][3], ml[ROUGH ? NP : 1][3];
#pragma unroll
  for (int q = 0; q < NP; q++) {
    const Phase& h = ph[w0 + q];
    const unsigned long long u = (unsigned long long)lane;
    t[q] = h.P0 + h.P1 * u + h.P2 * (u * u);
    dt[q] = h.P1 * 32ull + h.P2 * (64ull * u + 1024ull);
    ddt[q] = h.P2 * 2048ull;
    if (ROUGH)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        mh[q][k] = h.mh[k];
        ml[q][k] = h.ml[k];
      }
  }
#pragma unroll
  for (int g = 0; g < NPK; g++) {
    const Phase &a = ph[w0 + 2 * g], &b = ph[w0 + 2 * g + 1];
#pragma unroll
    for (int k = 0; k < 3; k++) nv[g][k] = pk(a.n[k], b.n[k]);
    dw[g] = pk(a.dw, b.dw);
    w[g] = fma2(dw[g], dup((float)lane * 0.03125f), pk(a.w, b.w));
    c3[g] = pk(a.c3, b.c3);
  }
  if (ADJ) {
    const int ka = idx[w0], kb = idx[w0 + 1] < 0 ? ka : idx[w0 + 1];
    const float *sa = seeds + ((size_t)ka * nifo + d) * 2 * kU, *sb = seeds + ((size_t)kb * nifo + d) * 2 * kU;
#pragma unroll
    for (int k = 0; k < kU; k++) {
      al[k] = pk(sa[k], sb[k]);
      be[k] = pk(sa[kU + k], sb[kU + k]);
    }
  }
  constexpr int NA = ADJ ? (ROUGH ? 10 : 7) : 2 * kU;
  f2 acc[NPK][NA];
#pragma unroll
  for (int g = 0; g < NPK; g++)
#pragma unroll
    for (int k = 0; k < NA; k++) acc[g][k] = 0ull;
  float jf = (float)lane;
  const int its = (cnt + 31) >> 5;
  for (int it = 0; it < its; it++) {
    const int j = it * 32 + lane;
    const float4 a = s0[j], b = s1[j];
    const float j3 = jf * jf * jf;
    int rr[3];
    if (ROUGH)
#pragma unroll
      for (int k = 0; k < 3; k++) rr[k] = ri[k * kChunk + j];
#pragma unroll
    for (int g = 0; g < NPK; g++) {
      const f2 nr = fma2(nv[g][2], dup(b.w), fma2(nv[g][1], dup(b.z), mul2(nv[g][0], dup(b.y))));
      const f2 rho = fma2(c3[g], dup(j3), mul2(w[g], nr));
      w[g] = add2(w[g], dw[g]);
      unsigned qa = (unsigned)(t[2 * g] >> 32), qb = (unsigned)(t[2 * g + 1] >> 32);
      if (ROUGH)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          qa += (unsigned)(mh[2 * g][k] * rr[k]) + (unsigned)__mulhi(ml[2 * g][k], rr[k]);
          qb += (unsigned)(mh[2 * g + 1][k] * rr[k]) + (unsigned)__mulhi(ml[2 * g + 1][k], rr[k]);
        }
      // the turns of a quadrant in two's complement: 2^32 per quarter turn
      const f2 ang = fma2(pk((float)(int)((qa << 2) ^ 0x80000000u), (float)(int)((qb << 2) ^ 0x80000000u)),
                          dup(3.6572951981e-10f), rho);  // pi/2 2^-32
#pragma unroll
      for (int q = 2 * g; q < 2 * g + 2; q++) {
        t[q] += dt[q];
        dt[q] += ddt[q];
      }
      f2 sn, cs;
      sincos2(ang, qa, qb, &sn, &cs);
      const float xu[kU] = {a.x, a.y, a.z, a.w, b.x};
      if (!ADJ) {
#pragma unroll
        for (int k = 0; k < kU; k++) {
          acc[g][k] = fma2(cs, dup(xu[k]), acc[g][k]);
          acc[g][kU + k] = fma2(sn, dup(xu[k]), acc[g][kU + k]);
        }
      } else {
        f2 ca = mul2(al[0], dup(xu[0])), cb = mul2(be[0], dup(xu[0]));
#pragma unroll
        for (int k = 1; k < kU; k++) {
          ca = fma2(al[k], dup(xu[k]), ca);
          cb = fma2(be[k], dup(xu[k]), cb);
        }
        const f2 gv = fma2(cs, ca, mul2(sn, cb));
        const f2 g1 = mul2(gv, dup(jf)), g2 = mul2(g1, dup(jf));
        acc[g][0] = add2(acc[g][0], gv);
        acc[g][1] = add2(acc[g][1], g1);
        acc[g][2] = add2(acc[g][2], g2);
        acc[g][3] = fma2(g2, dup(jf), acc[g][3]);
        acc[g][4] = fma2(gv, dup(b.y), acc[g][4]);
        acc[g][5] = fma2(gv, dup(b.z), acc[g][5]);
        acc[g][6] = fma2(gv, dup(b.w), acc[g][6]);
        if constexpr (ROUGH) {
          acc[g][7] = fma2(g1, dup(b.y), acc[g][7]);
          acc[g][8] = fma2(g1, dup(b.z), acc[g][8]);
          acc[g][9] = fma2(g1, dup(b.w), acc[g][9]);
        }
      }
    }
    jf += 32.f;
  }
  // the sums of all points as groups of eight values, NV a point
  constexpr int PART = ADJ ? kPartA : kPartF, NV = ADJ && ROUGH ? kPartA + kPartA2 : PART, VAL = NP * NV;
  float v[(VAL + 7) / 8 * 8];
#pragma unroll
  for (int k = VAL; k < (VAL + 7) / 8 * 8; k++) v[k] = 0.f;
#pragma unroll
  for (int g = 0; g < NPK; g++)
#pragma unroll
    for (int k = 0; k < NV; k++) {
      float x = 0.f, y = 0.f;
      if (k < NA) upk(acc[g][k < NA ? k : 0], x, y);
      v[(2 * g) * NV + k] = x;
      v[(2 * g + 1) * NV + k] = y;
    }
#pragma unroll
  for (int g = 0; g < (VAL + 7) / 8; g++) {
    float e[8];
#pragma unroll
    for (int k = 0; k < 8; k++) e[k] = v[8 * g + k];
    const float s = warp_sum8(e, lane);
    const int q = 8 * g + warp_sum8_index(lane), pt = q / NV, m = q - pt * NV;
    if ((lane & 3) == 0 && q < VAL) {
      const int k = idx[w0 + pt];
      if (k >= 0 && form[w0 + pt] == (ROUGH ? kRough : kFast)) {
        const size_t at = (size_t)k * P + p;
        part[m < PART ? at * PART + m : (size_t)n * P * PART + at * kPartA2 + (m - PART)] = s;
      }
    }
  }
}

// (a call: its registers are not the fast form's)
template <bool ADJ>
__device__ __noinline__ void sums_rough(const float4* s0, const float4* s1, const int* ri, const Phase* ph,
                                        const int* idx, const int* form, const float* __restrict__ seeds, int w0,
                                        int cnt, int n, int nifo, int d, int P, int p, float* __restrict__ part) {
  sums_fp32<ADJ, true, 1>(s0, s1, ri, ph, idx, form, seeds, w0, cnt, n, nifo, d, P, p, part);
}

// Sums of a chunk (of one detector) for 32 (forward) or 16 (adjoint) points,
// blockIdx.x = group of points * chunks + chunk: the chunk's samples {x u_0 .. x u_4, r} are staged in shared
// memory (32 KB, and 12 KB of integer rests where a point needs them), each warp
// takes four (two) points at once with its lanes over the samples, two points in
// the halves of packed registers; a sample read from shared memory serves all of
// them.  The adjoint holds ten more factors a point, so it takes two points at 80
// registers, three CTAs per SM (3.83 ms; 3.87 with 124 registers and two CTAs;
// 4.00 with 64 points to a CTA).  FAST: every point is fast over every chunk, for the
// adjoint of points that the host has seen; the other forms' code and the choice
// among them take 1 us of a kernel that runs for 5 to 10, and registers (4096 points:
// F and gradient 3.83 -> 3.76 ms).  The forward sums gain nothing by it (1.72 ms,
// 1.80 without the other forms, with other registers spilled).
template <bool ADJ, bool FAST>
__global__ void __launch_bounds__(kThreads, ADJ ? 3 : 2)
    k_sums(const float4* __restrict__ samp, const int* __restrict__ rough, const Chunk* __restrict__ chunk,
           const double* __restrict__ pos, const Point* __restrict__ point, const float* __restrict__ seeds,
           const int* __restrict__ list, const int* __restrict__ nlist, int n, int N, int nifo, int nch,
           const Centre ctr, float* __restrict__ part) {
  constexpr int NPK = ADJ ? 1 : 2, NP = 2 * NPK, PTS = 8 * NP;
  __shared__ __align__(16) float4 s0[kChunk], s1[kChunk];
  __shared__ __align__(16) int ri[FAST ? 4 : 3 * kChunk];
  __shared__ Phase ph[PTS];
  __shared__ int idx[PTS], form[PTS];
  const int cnt_pts = list ? *nlist : n;
  const int P = nifo * nch, p = blockIdx.x % P, d = p / nch, base = (p - d * nch) * kChunk;
  const int first = (int)(blockIdx.x / P) * PTS;
  if (first >= cnt_pts) return;
  const int cnt = min(kChunk, N - base);
  auto copy16 = [](void* to, const void* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
  };
  {
    const float4* src = samp + (size_t)p * 2 * kChunk;
    for (int k = threadIdx.x; k < kChunk; k += kThreads) {
      copy16(&s0[k], src + k);
      copy16(&s1[k], src + kChunk + k);
    }
  }
  bool is_rough = false;
  if (threadIdx.x < PTS) {
    // (places past the last point repeat it; they are not written)
    const int q = min(first + (int)threadIdx.x, cnt_pts - 1);
    const int k = list ? list[q] : q;
    idx[threadIdx.x] = first + (int)threadIdx.x < cnt_pts ? k : -1;
    chunk_phase(point[k], chunk[p], base, &ph[threadIdx.x]);
    const int fm = FAST || point[k].fast ? kFast : form_of(point[k].fo, point[k].st2, chunk[p].top, N, ADJ);
    form[threadIdx.x] = fm;
    is_rough = fm == kRough;
    if (is_rough) chunk_rough(point[k], chunk[p], base, &ph[threadIdx.x]);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (FAST) {
    __syncthreads();
  } else if (__syncthreads_or(is_rough)) {
    const int* src = rough + (size_t)p * 3 * kChunk;
    for (int k = 4 * threadIdx.x; k < 3 * kChunk; k += 4 * kThreads) copy16(&ri[k], src + k);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
  }
  const int w0 = (threadIdx.x >> 5) * NP;
  if (idx[w0] < 0) return;
  unsigned any = 0;  // bit f: a point of form f
#pragma unroll
  for (int q = 0; q < NP; q++)
    if (idx[w0 + q] >= 0) any |= 1u << form[w0 + q];
  if (FAST || (any >> kFast & 1))
    sums_fp32<ADJ, false, NPK>(s0, s1, ri, ph, idx, form, seeds, w0, cnt, n, nifo, d, P, p, part);
  if (FAST) return;
  if (any >> kRough & 1) {
#pragma unroll 1
    for (int q = w0; q < w0 + NP; q += 2)
      if ((idx[q] >= 0 && form[q] == kRough) || (idx[q + 1] >= 0 && form[q + 1] == kRough))
        sums_rough<ADJ>(s0, s1, ri, ph, idx, form, seeds, q, cnt, n, nifo, d, P, p, part);
  }
  if (any >> kSlow & 1) {
    for (int q = 0; q < NP; q++) {
      const int k = idx[w0 + q];
      if (k < 0 || form[w0 + q] != kSlow) continue;
      sums_slow<ADJ>(point[k], ADJ ? seeds + ((size_t)k * nifo + d) * 2 * kU : nullptr, pos + ((size_t)d * N + base) * 3,
                     s0, s1, base, cnt, ctr, part + ((size_t)k * P + p) * (ADJ ? kPartA : kPartF));
    }
  }
}

// CTAs of k_sums for n points
inline unsigned sum_grid(bool adj, int n, int P) {
  const int pts = adj ? 16 : 32;
  return (unsigned)P * (unsigned)((n + pts - 1) / pts);
}

// Sum of floats to about 48 bits: s + e (TwoSum)
__device__ __forceinline__ void comp_add(float& s, float& e, float v) {
  const float t = __fadd_rn(s, v);
  const float bb = __fsub_rn(t, s);
  e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(v, bb)));
  s = t;
}

// F and fstat_out (followup.c:508-529) per point, and the seeds of the adjoint
// pass.  One warp per point: lanes (value m, group g of chunks) sum the chunks
// in a fixed order, compensated; then lane d combines detector d.
__global__ void __launch_bounds__(256)
    k_final(const float* __restrict__ part, const double* __restrict__ pts, Point* __restrict__ point,
            const double* __restrict__ coef, FuDets dets, const int* __restrict__ list, const int* __restrict__ nlist,
            int n, int nifo, int nch, double* __restrict__ totals, double* __restrict__ Fo, double* __restrict__ out,
            const double* __restrict__ seed, float* __restrict__ seeds) {
  __shared__ double sums[8][PA_MAX_DETECTORS][2 * kU];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + warp;
  if (q >= (list ? *nlist : n)) return;
  const int k = list ? list[q] : q;
  const int m = lane % (2 * kU), g = lane / (2 * kU);  // three groups of ten lanes
  for (int d = 0; d < nifo; d++) {
    const float* src = part + ((size_t)k * nifo + d) * nch * kPartF;
    float s = 0.f, e = 0.f;
    if (g < 3)
      for (int c = g; c < nch; c += 3) comp_add(s, e, src[(size_t)c * kPartF + m]);
    const double v = (double)s + (double)e;
    const double v1 = __shfl_down_sync(0xffffffffu, v, 2 * kU), v2 = __shfl_down_sync(0xffffffffu, v, 4 * kU);
    if (lane < 2 * kU) sums[warp][d][lane] = v + v1 + v2;
  }
  __syncwarp();
  double xr = 0., xi = 0., yr = 0., yi = 0.;
  if (lane < nifo) {
    const double* Q = coef + ((size_t)k * nifo + lane) * kCoef;
    const double* S = sums[warp][lane];
    const double is2 = dets.d[lane].inv_sig2;
    for (int t = 0; t < kU; t++) {
      xr += Q[t] * S[t];
      xi -= Q[t] * S[kU + t];
      yr += Q[kU + t] * S[t];
      yi -= Q[kU + t] * S[kU + t];
    }
    xr *= is2;
    xi *= is2;
    yr *= is2;
    yi *= is2;
  }
  xr = warp_sum_d(xr);
  xi = warp_sum_d(xi);
  yr = warp_sum_d(yr);
  yi = warp_sum_d(yi);
  const double iA = 1. / point[k].A, iB = 1. / point[k].B, sd = seed ? seed[k] : 1.;
  const double ka = 2. * sd * iA, kb = 2. * sd * iB;
  for (int t = lane; t < nifo * 2 * kU; t += 32) {
    const int d = t / (2 * kU), r = t - d * 2 * kU;
    totals[((size_t)k * nifo + d) * 2 * kU + r] = sums[warp][d][r];
    // g = x (ka a Im_a + kb b Im_b), Im = -(xr sin + xi cos), as coefficients
    // of x u_k cos and x u_k sin
    const double* Q = coef + ((size_t)k * nifo + d) * kCoef;
    const int u = r < kU ? r : r - kU;
    seeds[((size_t)k * nifo + d) * 2 * kU + r] =
        (float)(r < kU ? -(ka * xi * Q[u] + kb * yi * Q[kU + u]) : -(ka * xr * Q[u] + kb * yr * Q[kU + u]));
  }
  if (lane) return;
  const double Fa = (xr * xr + xi * xi) * iA, Fb = (yr * yr + yi * yi) * iB, F = Fa + Fb;
  if (Fo) Fo[k] = F;
  if (out) {
    double* o = out + (size_t)k * 11;
    o[5] = -F;
    o[0] = 2 * xr * iA;
    o[1] = 2 * yr * iB;
    o[2] = -2 * xi * iA;
    o[3] = -2 * yi * iB;
    o[4] = sqrt(2 * (F - 2));
    for (int j = 0; j < 4; j++) o[6 + j] = pts[4 * k + j];
    o[10] = 2 * sqrt(xr * xr + yr * yr + xi * xi + yi * yi);
  }
  Point& c = point[k];
  c.xr = xr;
  c.xi = xi;
  c.yr = yr;
  c.yi = yi;
  c.ka = ka;
  c.kb = kb;
  c.qa = -sd * Fa * iA;
  c.qb = -sd * Fb * iB;
}

// The gradient.  Per chunk, sum g (R - Rc) and sum g (i R - ic Rc) with the
// centre (ic, Rc), from the moments of g (fast form: without sum g j r, at most
// 2048 of the chunk's rest times sum |g|: below FP32 rounding, adj_fast), with
// sum g (i - ic) and sum g (i^2 - ic^2); then, with Q0 and Q1 the first two over
// all samples and detectors,
//   dF/df = sum g i + n.Q0, dF/ds = sum g i^2 + 2 n.Q1,
//   dF/dangle = (f + oms) n'.Q0 + 2 s n'.Q1 + the amplitudes' part.
// One warp a point, two to a block: the FP64 pipe of an SM bounds it, and blocks of
// eight left a call of a few points to a few SMs (39 points of two detectors, N =
// 33390: 25 -> 16 us; the call 116 -> 113 us).
constexpr int kAdjPts = 2;
__global__ void __launch_bounds__(32 * kAdjPts)
    k_final_adj(const float* __restrict__ part, const Point* __restrict__ point, const double* __restrict__ coef,
                const Chunk* __restrict__ chunk, FuDets dets, const int* __restrict__ list,
                const int* __restrict__ nlist, int n, int N, int nifo, int nch, double oms,
                const double* __restrict__ totals, double* __restrict__ grad) {
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * kAdjPts + (threadIdx.x >> 5);
  if (q >= (list ? *nlist : n)) return;
  const int k = list ? list[q] : q;
  const Point& c = point[k];
  const int P = nifo * nch;
  double o[4] = {0., 0., 0., 0.};
  double m1 = 0., m2 = 0., Q0[3] = {0., 0., 0.}, Q1[3] = {0., 0., 0.};
  for (int p = lane; p < P; p += 32) {
    const int d = p / nch, form = c.fast ? kFast : form_of(c.fo, c.st2, chunk[p].top, N, true);
    const double is2 = dets.d[d].inv_sig2;
    const float* src = part + ((size_t)k * P + p) * kPartA;
    if (form == kSlow) {
#pragma unroll
      for (int t = 0; t < 4; t++) o[t] += is2 * reinterpret_cast<const double*>(src)[t];
      continue;
    }
    const float4 a = reinterpret_cast<const float4*>(src)[0], e = reinterpret_cast<const float4*>(src)[1];
    const Chunk& H = chunk[p];
    const double b = (double)((p - d * nch) * kChunk);
    const double g0 = is2 * (double)a.x, g1 = is2 * (double)a.y, g2 = is2 * (double)a.z, g3 = is2 * (double)a.w;
    const double h[3] = {is2 * (double)e.x, is2 * (double)e.y, is2 * (double)e.z};
    m1 += fma(H.db, g0, g1);
    m2 += fma(H.db2, g0, fma(2. * b, g1, g2));
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const double z = fma(g1, H.V[t], fma(g2, H.A[t], h[t]));
      Q0[t] += fma(g0, H.dR[t], z);
      Q1[t] += fma(g0, H.dbR[t], fma(b, z, fma(g1, H.R0[t], fma(g2, H.V[t], g3 * H.A[t]))));
    }
    if (form == kRough) {
      const float2 r = reinterpret_cast<const float2*>(part + (size_t)n * P * kPartA)[(size_t)k * P + p];
      Q1[0] += is2 * (double)e.w;
      Q1[1] += is2 * (double)r.x;
      Q1[2] += is2 * (double)r.y;
    }
  }
  auto dot = [](const double* x, const double* y) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
  const double om0 = c.f + oms, s2 = 2. * c.s;
  o[0] += m1 + dot(c.n, Q0);
  o[1] += m2 + 2. * dot(c.n, Q1);
  o[2] += om0 * dot(c.nD, Q0) + s2 * dot(c.nD, Q1);
  o[3] += om0 * dot(c.nA, Q0) + s2 * dot(c.nA, Q1);
  // amplitudes: sum x Re(conj(X) E) da/dangle, E = cos - i sin
  if (lane < nifo) {
    const double* Q = coef + ((size_t)k * nifo + lane) * kCoef;
    const double* S = totals + ((size_t)k * nifo + lane) * 2 * kU;
    const double is2 = dets.d[lane].inv_sig2;
    double aa[kU], bb[kU];
    d_alpha(Q, aa);
    d_alpha(Q + kU, bb);
    double gd = 0., ga = 0.;
    for (int t = 0; t < kU; t++) {
      const double a = c.ka * (c.xr * S[t] - c.xi * S[kU + t]), b = c.kb * (c.yr * S[t] - c.yi * S[kU + t]);
      gd += Q[2 * kU + t] * a + Q[3 * kU + t] * b;
      ga += aa[t] * a + bb[t] * b;
    }
    o[2] += is2 * gd;
    o[3] += is2 * ga;
  }
#pragma unroll
  for (int t = 0; t < 4; t++) o[t] = warp_sum_d(o[t]);
  if (lane) return;
  o[2] += c.qa * c.dA[0] + c.qb * c.dB[0];
  o[3] += c.qa * c.dA[1] + c.qb * c.dB[1];
  for (int t = 0; t < 4; t++) grad[(size_t)k * 4 + t] = o[t];
}

}  // namespace fu32
