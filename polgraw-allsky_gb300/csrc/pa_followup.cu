// pa_followup.cu -- the followup path of libpolgraw_gb300.so: the
// demodulated network F-statistic of followup/src/followup.c (Fstatnet,
// :413-535, with the sky set-up of evaluate_simplex, :986-1009) at batches
// of arbitrary points (f, s, delta, alpha), its adjoint gradient, a batched
// gradient ascent, and the reference simplex amoeba (:971-1174) with its
// evaluations batched on the device.
//
// The mixed form (FP32 sums, the phase in 64-bit fixed point) is in
// pa_followup_f32.cuh; the FP64 form is here:
//   xd  [nifo][N]      xDat
//   pos [nifo][N][3]   DetSSB (x y z interleaved, as the input file)
//   cm, sm [N]         cos/sin(omr i) (init.c:464-475)
// Per evaluated point k:
//   cand[k]            scalars of the point (phase terms, seeds)
//   coef[k][d][20]     modvir factors of detector d and their sky derivatives
//   part[k][p][6|4]    partial sums of chunk p (fixed order)
//
// Work split: chunk p covers kChunk samples of one detector; a CTA stages
// its chunk in shared memory and each warp runs kCandPerWarp points over it
// (lanes stride the samples), then reduces across lanes and writes one
// partial per point and chunk.  A second kernel sums the partials of a
// point in a fixed order, so results do not depend on the batch.
// Nothing here waits on another CTA or kernel.
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/polgraw_gb300.h"
#include "pa_f32x2.cuh"
#include "pa_sincos.cuh"
#include "pa_trace.h"

namespace {

constexpr int kChunk = 1024;      // samples per chunk (shared-memory stage)
constexpr int kThreads = 256;     // 8 warps
constexpr int kCandPerWarp = 4;   // points per warp per chunk
constexpr int kCandPerCta = 8 * kCandPerWarp;
constexpr int kCoef = 20;         // modvir factors per point and detector
constexpr double kInv2Pi = 0.15915494309189533577;  // 1/(2 pi), rounded to double

// x mod 1 as a 64-bit fixed-point fraction (x 2^64 mod 2^64), exactly, with
// integer operations on the bits of x: x = m 2^(e-1075), so the fraction is
// m shifted by e - 1011, negated for x < 0.
__device__ __forceinline__ unsigned long long fu_turns_fixed(double x) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((bits >> 52) & 0x7ff);
  if (e == 0) return 0ull;
  const unsigned long long m = (bits & 0xfffffffffffffull) | 0x10000000000000ull;
  const int sh = e - 1011;
  unsigned long long t;
  if (sh >= 64) t = 0ull;
  else if (sh >= 0) t = m << sh;
  else if (sh > -64) t = m >> (-sh);
  else t = 0ull;
  return (bits >> 63) ? (0ull - t) : t;
}

thread_local std::string g_fu_create_error;

// Per-detector inputs of the modvir() formula (settings.c:281-325).
struct FuDet {
  double amod[9];
  double cphir, sphir, inv_sig2;
};

struct FuDets {
  FuDet d[PA_MAX_DETECTORS];
};

#include "pa_followup_f32.cuh"

// Per-point scalars of the FP64 form.
struct FuCand {
  double f, s;          // sgnlo[0], sgnlo[1] (radians)
  double nS[3];         // source unit vector
  double nD[3], nA[3];  // d nS / d delta, d nS / d alpha
  double om0, s2;       // f + oms, 2 s (d phase / d shft = om0 + s2 i)
  // adjoint seeds: conj(X) parts and the factors of dF/dX, dF/dA
  double xar, xai, xbr, xbi, ka, kb, qa, qb;
  int active;
  int pad;
};

// ---------------------------------------------------------------------
// Point set-up: sin/cos of the sky angles, source vector and derivatives,
// per-detector modvir factors.  One thread per point.
//   a = 2 A1 c^2 + A2 c s + A3 c + A4 s + A0      (modvir aa)
//   b = 2 B1 c^2 + B2 c s + B3 c + B4 s + B0      (modvir bb)
//   da/ddelta = D1 c^2 + D2 c s + D3 c + D4 s + D0, db/ddelta likewise (E)
// with c, s the rotated sidereal cos/sin of the sample; d/dalpha acts on
// (c, s) only: dc/dalpha = -s, ds/dalpha = c.
// ---------------------------------------------------------------------
__global__ void k_fu_prep(const double* __restrict__ pts, int n, const unsigned char* __restrict__ mask,
                          FuCand* __restrict__ cand, double* __restrict__ coef, FuDets dets, int nifo, double oms) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  FuCand c;
  c.active = mask ? (int)mask[k] : 1;
  const double f = pts[4 * k + 0], s = pts[4 * k + 1], de = pts[4 * k + 2], al = pts[4 * k + 3];
  double sa, ca, sd, cd;
  sincos(al, &sa, &ca);
  sincos(de, &sd, &cd);
  c.f = f;
  c.s = s;
  c.nS[0] = ca * cd;
  c.nS[1] = sa * cd;
  c.nS[2] = sd;
  c.nD[0] = -ca * sd;
  c.nD[1] = -sa * sd;
  c.nD[2] = cd;
  c.nA[0] = -sa * cd;
  c.nA[1] = ca * cd;
  c.nA[2] = 0.;
  c.om0 = f + oms;
  c.s2 = 2. * s;
  c.xar = c.xai = c.xbr = c.xbi = c.ka = c.kb = c.qa = c.qb = 0.;
  c.pad = 0;
  cand[k] = c;
  const double c2d = cd * cd, c2sd = sd * cd;
  const double dc2d = -2. * sd * cd, dc2sd = cd * cd - sd * sd;
  for (int d = 0; d < nifo; d++) {
    const double* K = dets.d[d].amod;
    const double cosalfr = ca * dets.d[d].cphir + sa * dets.d[d].sphir;
    const double sinalfr = sa * dets.d[d].cphir - ca * dets.d[d].sphir;
    double* q = coef + ((size_t)k * nifo + d) * kCoef;
    q[0] = cosalfr;
    q[1] = sinalfr;
    // a
    q[2] = K[0] * (2. - c2d);                // A1
    q[3] = 2. * K[1] * (2. - c2d);           // A2
    q[4] = K[2] * c2sd;                      // A3
    q[5] = K[3] * c2sd;                      // A4
    q[6] = -K[0] * (2. - c2d) + K[4] * c2d;  // A0
    // b
    q[7] = K[5] * sd;                        // B1
    q[8] = 2. * K[6] * sd;                   // B2
    q[9] = K[7] * cd;                        // B3
    q[10] = K[8] * cd;                       // B4
    q[11] = -K[5] * sd;                      // B0
    // da/ddelta
    q[12] = -2. * K[0] * dc2d;               // D1 (c^2)
    q[13] = -2. * K[1] * dc2d;               // D2 (c s)
    q[14] = K[2] * dc2sd;                    // D3 (c)
    q[15] = K[3] * dc2sd;                    // D4 (s)
    q[16] = (K[0] + K[4]) * dc2d;            // D0
    // db/ddelta = E1 c^2 + E2 c s + E3 c + E4 s + E0
    // (E3 = -K7 sd and E4 = -K8 sd are formed in the adjoint kernel)
    q[17] = 2. * K[5] * cd;                  // E1
    q[18] = 2. * K[6] * cd;                  // E2
    q[19] = -K[5] * cd;                      // E0
  }
}

// Makes the adjoint pass run for the points selected by need[] with the
// constants and seeds their last forward pass left in cand[].
__global__ void k_fu_select(FuCand* __restrict__ cand, int n, const unsigned char* __restrict__ need) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) cand[k].active = (int)need[k];
}

struct Sample {
  double x, cm, sm;
  double r0, r1, r2;
  double di;             // the sample index as FP64
};

// The phase of sample i for point c (followup.c:460-462 order, no
// contraction): phi = f (i + shft) + (s i) i + (oms + 2 s i) shft
__device__ __forceinline__ void fu_phase(const FuCand& c, double oms, double di, double shft, double* sn, double* cs) {
  const double phi = __dadd_rn(__dadd_rn(__dmul_rn(c.f, __dadd_rn(di, shft)), __dmul_rn(__dmul_rn(c.s, di), di)),
                               __dmul_rn(__dadd_rn(oms, __dmul_rn(__dmul_rn(2., c.s), di)), shft));
  pa::sincos_fast(phi, sn, cs);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------
// Forward sums (ADJ = false): per point and chunk
//   sum x a e^{-i phi}, sum x b e^{-i phi}, sum a^2, sum b^2   (x 1/sig2)
// Adjoint sums (ADJ = true): per point and chunk, the four components of
//   dF/dtheta = sum [ dphi/dtheta x (ka a Im(conj(Xa)E) + kb b Im(conj(Xb)E))
//                   + da/dtheta (x ka Re(conj(Xa)E) + 2 qa a) + (b terms) ]
//   (x 1/sig2), with E = e^{-i phi}, ka = 2 seed/A, qa = -seed |Xa|^2/A^2.
// ---------------------------------------------------------------------
// Two CTAs per SM: the FP64 pipe bounds the kernel with 16 warps as with 24, and
// what 24 leave of the registers (80) spills (100 points of two detectors, N =
// 86164: 2.39 ms, 2.50 with three).
template <bool ADJ>
__global__ void __launch_bounds__(kThreads, 2) k_fu_sums(const double* __restrict__ xd, const double* __restrict__ pos,
                                                      const double* __restrict__ cmf, const double* __restrict__ smf,
                                                      const FuCand* __restrict__ cand, const double* __restrict__ coef,
                                                      FuDets dets, int n, int N, int nifo, int nch, double oms,
                                                      double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char fu_smem[];
  Sample* sh = reinterpret_cast<Sample*>(fu_smem);
  const int P = nifo * nch;
  const int p = blockIdx.x;
  const int d = p / nch;
  const int base = (p - d * nch) * kChunk;
  const int cnt = min(kChunk, N - base);
  for (int j = threadIdx.x; j < cnt; j += kThreads) {
    const int i = base + j;
    Sample v;
    v.x = xd[(size_t)d * N + i];
    v.cm = cmf[i];
    v.sm = smf[i];
    const double* r = pos + ((size_t)d * N + i) * 3;
    v.r0 = r[0];
    v.r1 = r[1];
    v.r2 = r[2];
    v.di = (double)i;
    sh[j] = v;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double is2 = dets.d[d].inv_sig2;
  const double k7 = dets.d[d].amod[7], k8 = dets.d[d].amod[8];
  for (int q = 0; q < kCandPerWarp; q++) {
    const int k = blockIdx.y * kCandPerCta + warp * kCandPerWarp + q;
    if (k >= n) break;
    const FuCand c = cand[k];
    if (!c.active) continue;
    const double* cf = coef + ((size_t)k * nifo + d) * kCoef;
    double Q[kCoef];
#pragma unroll
    for (int t = 0; t < kCoef; t++) Q[t] = cf[t];
    const double cosalfr = Q[0], sinalfr = Q[1];
    double acc[6] = {0., 0., 0., 0., 0., 0.};
    const double sd_ = c.nS[2];  // sin(delta), for E3 = -K7 sd, E4 = -K8 sd
    for (int j = lane; j < cnt; j += 32) {
      const Sample v = sh[j];
      const double cc = cosalfr * v.cm + sinalfr * v.sm;
      const double ss = sinalfr * v.cm - cosalfr * v.sm;
      const double c2 = cc * cc, cs = cc * ss;
      const double a = 2. * Q[2] * c2 + Q[3] * cs + Q[4] * cc + Q[5] * ss + Q[6];
      const double b = 2. * Q[7] * c2 + Q[8] * cs + Q[9] * cc + Q[10] * ss + Q[11];
      double sn, co;
      const double shft = c.nS[0] * v.r0 + c.nS[1] * v.r1 + c.nS[2] * v.r2;
      fu_phase(c, oms, v.di, shft, &sn, &co);
      if (!ADJ) {
        const double xa = v.x * a, xb = v.x * b;
        acc[0] += xa * co;
        acc[1] -= xa * sn;
        acc[2] += xb * co;
        acc[3] -= xb * sn;
        acc[4] += a * a;
        acc[5] += b * b;
      } else {
        // conj(X) E with E = co - i sn
        const double rea = c.xar * co - c.xai * sn, ima = -(c.xar * sn + c.xai * co);
        const double reb = c.xbr * co - c.xbi * sn, imb = -(c.xbr * sn + c.xbi * co);
        const double gph = v.x * (c.ka * a * ima + c.kb * b * imb);
        const double ga = v.x * c.ka * rea + 2. * c.qa * a;
        const double gb = v.x * c.kb * reb + 2. * c.qb * b;
        const double fi = v.di;
        const double sh_de = c.nD[0] * v.r0 + c.nD[1] * v.r1 + c.nD[2] * v.r2;
        const double sh_al = c.nA[0] * v.r0 + c.nA[1] * v.r1;
        const double om = c.om0 + c.s2 * fi;
        // d a / d alpha, d b / d alpha
        const double a_al = -ss * (4. * Q[2] * cc + Q[3] * ss + Q[4]) + cc * (Q[3] * cc + Q[5]);
        const double b_al = -ss * (4. * Q[7] * cc + Q[8] * ss + Q[9]) + cc * (Q[8] * cc + Q[10]);
        // d a / d delta, d b / d delta
        const double a_de = Q[12] * c2 + Q[13] * cs + Q[14] * cc + Q[15] * ss + Q[16];
        const double b_de = Q[17] * c2 + Q[18] * cs - k7 * sd_ * cc - k8 * sd_ * ss + Q[19];
        acc[0] += gph * (fi + shft);
        acc[1] += gph * (fi * fi + 2. * fi * shft);
        acc[2] += gph * om * sh_de + ga * a_de + gb * b_de;
        acc[3] += gph * om * sh_al + ga * a_al + gb * b_al;
      }
    }
    constexpr int NA = ADJ ? 4 : 6;
    double* out = part + ((size_t)k * P + p) * NA;
#pragma unroll
    for (int t = 0; t < NA; t++) {
      const double v = warp_sum(acc[t]);
      if (lane == 0) out[t] = v * is2;
    }
  }
}

// Sum of the partials of one point in a fixed order (lane stride, then a
// fixed shuffle tree).
__device__ __forceinline__ double fixed_sum(const double* __restrict__ p, int P, int stride, int lane) {
  double s = 0.;
  for (int j = lane; j < P; j += 32) s += p[(size_t)j * stride];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// F and fstat_out (followup.c:508-529) per point; res[k] = {Xa, Xb, A, B}
// kept for the adjoint.  One warp per point.
__global__ void k_fu_final(const double* __restrict__ part, const double* __restrict__ pts,
                           FuCand* __restrict__ cand, int n, int P, double* __restrict__ res,
                           double* __restrict__ Fo, double* __restrict__ out, const double* __restrict__ seed) {
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (k >= n) return;
  if (!cand[k].active) return;
  double v[6];
  for (int t = 0; t < 6; t++) v[t] = fixed_sum(part + (size_t)k * P * 6 + t, P, 6, lane);
  if (lane) return;
  const double xr = v[0], xi = v[1], yr = v[2], yi = v[3], A = v[4], B = v[5];
  const double F = ((xr * xr + xi * xi) / A) + ((yr * yr + yi * yi) / B);
  if (res)
    for (int t = 0; t < 6; t++) res[(size_t)k * 6 + t] = v[t];
  if (Fo) Fo[k] = F;
  if (out) {
    double* o = out + (size_t)k * 11;
    o[5] = -F;
    o[0] = 2 * xr / A;
    o[1] = 2 * yr / B;
    o[2] = -2 * xi / A;
    o[3] = -2 * yi / B;
    o[4] = sqrt(2 * (F - 2));
    for (int j = 0; j < 4; j++) o[6 + j] = pts[4 * k + j];
    o[10] = sqrt((2 * xr) * (2 * xr) + (2 * yr) * (2 * yr) + (2 * xi) * (2 * xi) + (2 * yi) * (2 * yi));
  }
  // seeds of the adjoint pass
  const double sd = seed ? seed[k] : 1.0;
  FuCand& c = cand[k];
  c.xar = xr;
  c.xai = xi;
  c.xbr = yr;
  c.xbi = yi;
  c.ka = (2. * sd / A);
  c.kb = (2. * sd / B);
  c.qa = (-sd * (xr * xr + xi * xi) / (A * A));
  c.qb = (-sd * (yr * yr + yi * yi) / (B * B));
}

__global__ void k_fu_final_adj(const double* __restrict__ part, const FuCand* __restrict__ cand, int n, int P,
                               double* __restrict__ grad) {
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (k >= n) return;
  if (!cand[k].active) return;
  double v[4];
  for (int t = 0; t < 4; t++) v[t] = fixed_sum(part + (size_t)k * P * 4 + t, P, 4, lane);
  if (lane) return;
  for (int t = 0; t < 4; t++) grad[(size_t)k * 4 + t] = v[t];
}

// ---------------------------------------------------------------------
// Gradient ascent state machine (one thread per point): BFGS on -F in
// scaled coordinates u = theta / scale (peak-width units), with a
// backtracking line search.
//   propose: trial u' = u + t p, p = H g_u (g_u = scale * grad; H the
//            inverse-Hessian estimate of -F, first H = (step0/|g_u|) I)
//   decide:  F(trial) >= F + 1e-4 t g_u.p -> accept (t = 1 next), need the
//            gradient there; otherwise t *= 0.5
//   take:    with s = u' - u, y = g_u(old) - g_u(new): when y.s > 0,
//            H <- (I - r s y^T) H (I - r y s^T) + r s s^T, r = 1/y.s
//   a point stops when its step |t p| falls below min_step, its gradient
//   vanishes, or the direction stops being an ascent direction.
// ---------------------------------------------------------------------
struct AscentState {
  double theta[4], grad[4], trial[4];
  double gold[4], sdir[4];   // g_u before the accepted step, the step s
  double H[16];              // inverse-Hessian estimate (row-major)
  double p[4];               // search direction
  double F, t;
  int active, iters;
};

__global__ void k_asc_propose(AscentState* __restrict__ st, int n, double s0, double s1, double s2, double s3,
                              double min_step, double* __restrict__ trial_pts, unsigned char* __restrict__ mask) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  AscentState& a = st[k];
  const double sc[4] = {s0, s1, s2, s3};
  if (a.active) {
    double gu[4], slope = 0., plen = 0.;
    for (int j = 0; j < 4; j++) gu[j] = sc[j] * a.grad[j];
    for (int i = 0; i < 4; i++) {
      double v = 0.;
      for (int j = 0; j < 4; j++) v += a.H[4 * i + j] * gu[j];
      a.p[i] = v;
      slope += v * gu[i];
      plen += v * v;
    }
    plen = sqrt(plen);
    if (!(slope > 0.) || !isfinite(slope) || a.t * plen < min_step) a.active = 0;
  }
  mask[k] = (unsigned char)a.active;
  for (int j = 0; j < 4; j++) {
    a.trial[j] = a.active ? a.theta[j] + sc[j] * a.t * a.p[j] : a.theta[j];
    trial_pts[4 * k + j] = a.trial[j];
  }
}

__global__ void k_asc_decide(AscentState* __restrict__ st, int n, double s0, double s1, double s2, double s3,
                             const double* __restrict__ Ftrial, unsigned char* __restrict__ need_grad,
                             int* __restrict__ nactive) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  AscentState& a = st[k];
  need_grad[k] = 0;
  if (!a.active) return;
  const double sc[4] = {s0, s1, s2, s3};
  double slope = 0.;
  for (int j = 0; j < 4; j++) slope += a.p[j] * sc[j] * a.grad[j];
  const double Ft = Ftrial[k];
  if (Ft >= a.F + 1e-4 * a.t * slope && Ft > a.F) {
    for (int j = 0; j < 4; j++) {
      a.gold[j] = sc[j] * a.grad[j];
      a.sdir[j] = a.t * a.p[j];
      a.theta[j] = a.trial[j];
    }
    a.F = Ft;
    a.t = 1.0;
    a.iters++;
    need_grad[k] = 1;
  } else {
    a.t *= 0.5;
  }
  atomicAdd(nactive, 1);
}

__global__ void k_asc_init(AscentState* __restrict__ st, int n, const double* __restrict__ pts,
                           const double* __restrict__ F, const double* __restrict__ grad, double s0, double s1,
                           double s2, double s3, double step0) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  AscentState& a = st[k];
  const double sc[4] = {s0, s1, s2, s3};
  double nrm = 0.;
  for (int j = 0; j < 4; j++) {
    a.theta[j] = pts[4 * k + j];
    a.grad[j] = grad[4 * k + j];
    a.trial[j] = a.theta[j];
    a.gold[j] = a.sdir[j] = a.p[j] = 0.;
    nrm += (sc[j] * a.grad[j]) * (sc[j] * a.grad[j]);
  }
  nrm = sqrt(nrm);
  const double h0 = nrm > 0. ? step0 / nrm : 0.;
  for (int j = 0; j < 16; j++) a.H[j] = (j % 5 == 0) ? h0 : 0.;
  a.F = F[k];
  a.t = 1.0;
  a.active = nrm > 0. && isfinite(nrm);
  a.iters = 0;
}

__global__ void k_asc_take_grad(AscentState* __restrict__ st, int n, double s0, double s1, double s2, double s3,
                                const unsigned char* __restrict__ need, const double* __restrict__ grad) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || !need[k]) return;
  AscentState& a = st[k];
  const double sc[4] = {s0, s1, s2, s3};
  double y[4], ys = 0.;
  for (int j = 0; j < 4; j++) {
    a.grad[j] = grad[4 * k + j];
    y[j] = a.gold[j] - sc[j] * a.grad[j];
    ys += y[j] * a.sdir[j];
  }
  if (!(ys > 0.) || !isfinite(ys)) return;  // keep H (curvature condition fails)
  const double r = 1. / ys;
  // H <- (I - r s y^T) H (I - r y s^T) + r s s^T
  double Hy[4], yHy = 0.;
  for (int i = 0; i < 4; i++) {
    double v = 0.;
    for (int j = 0; j < 4; j++) v += a.H[4 * i + j] * y[j];
    Hy[i] = v;
    yHy += y[i] * v;
  }
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++)
      a.H[4 * i + j] += -r * (a.sdir[i] * Hy[j] + Hy[i] * a.sdir[j]) + (r * r * yHy + r) * a.sdir[i] * a.sdir[j];
}

__global__ void k_asc_export(const AscentState* __restrict__ st, int n, double* __restrict__ pts,
                             int* __restrict__ iters) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  for (int j = 0; j < 4; j++) pts[4 * k + j] = st[k].theta[j];
  iters[k] = st[k].iters;
}

}  // namespace

// ---------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------
struct pa_followup {
  int dev = 0;
  bool fp64 = false;
  int N = 0, nifo = 0, nch = 0;
  double oms = 0.;
  FuDets dets;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  double* pos = nullptr;
  // FP64 form
  double* xd = nullptr;
  double* cm = nullptr;
  double* sm = nullptr;
  // mixed form: samples [nifo][nch][2][1024] float4 {x u_0 .. x u_3},
  // {x u_4, r}, integer rests [nifo][nch][3][1024], the chunks' motion
  float4* samp = nullptr;
  int* rough = nullptr;
  fu32::Chunk* chunk = nullptr;
  fu32::Gram gram;
  fu32::Centre centre;
  fu32::Bounds top;              // of all chunks
  // per-batch buffers (grown on demand)
  int cap = 0;
  double* pts = nullptr;
  FuCand* cand = nullptr;        // FP64 form
  fu32::Point* point = nullptr;  // mixed form
  double* coef = nullptr;
  void* part = nullptr;
  double* totals = nullptr;      // mixed form: U, W per point and detector
  float* seeds = nullptr;        // mixed form: adjoint factors per point and detector
  int* list = nullptr;           // mixed form: active points
  int* nlist = nullptr;
  double* res = nullptr;
  double* F = nullptr;
  double* out = nullptr;
  double* grad = nullptr;
  double* seed = nullptr;
  unsigned char* mask = nullptr;
  unsigned char* need = nullptr;
  AscentState* asc = nullptr;
  int* iters = nullptr;
  int* counter = nullptr;
  double* trial = nullptr;
  std::string err;
  long long launches = 0;
  double last_ms = 0.;
};

static int fu_fail(pa_followup* f, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (f) f->err = buf;
  else g_fu_create_error = buf;
  return code;
}

#define FCK(call, what)                                                                             \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess) return fu_fail(f, PA_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e_)); \
  } while (0)

static void fu_free_batch(pa_followup* f) {
  void* ps[] = {f->pts, f->cand, f->point, f->coef, f->part, f->totals, f->seeds, f->list, f->nlist, f->res, f->F,
                f->out, f->grad, f->seed, f->mask, f->need, f->asc, f->iters, f->counter, f->trial};
  for (void* p : ps)
    if (p) cudaFree(p);
  f->pts = nullptr;
  f->cand = nullptr;
  f->point = nullptr;
  f->coef = f->totals = nullptr;
  f->part = nullptr;
  f->seeds = nullptr;
  f->list = f->nlist = nullptr;
  f->res = f->F = f->out = f->grad = f->seed = f->trial = nullptr;
  f->mask = f->need = nullptr;
  f->asc = nullptr;
  f->iters = f->counter = nullptr;
  f->cap = 0;
}

static int fu_reserve(pa_followup* f, int n) {
  if (n <= f->cap) return PA_OK;
  fu_free_batch(f);
  const int c = std::max(n, 64);
  const size_t P = (size_t)f->nifo * f->nch;
#define FALLOC(ptr, bytes) FCK(cudaMalloc((void**)&(ptr), (bytes)), "cudaMalloc")
  FALLOC(f->pts, sizeof(double) * 4 * c);
  FALLOC(f->coef, sizeof(double) * kCoef * f->nifo * (size_t)c);
  if (f->fp64) {
    FALLOC(f->cand, sizeof(FuCand) * c);
    FALLOC(f->part, sizeof(double) * 6 * P * c);
    FALLOC(f->res, sizeof(double) * 6 * c);
  } else {
    FALLOC(f->point, sizeof(fu32::Point) * c);
    FALLOC(f->part, sizeof(float) * std::max(fu32::kPartF, fu32::kPartA + fu32::kPartA2) * P * c);
    FALLOC(f->totals, sizeof(double) * 2 * fu32::kU * f->nifo * (size_t)c);
    FALLOC(f->seeds, sizeof(float) * 2 * fu32::kU * f->nifo * (size_t)c);
    FALLOC(f->list, sizeof(int) * c);
    FALLOC(f->nlist, sizeof(int));
  }
  FALLOC(f->F, sizeof(double) * c);
  FALLOC(f->out, sizeof(double) * 11 * c);
  FALLOC(f->grad, sizeof(double) * 4 * c);
  FALLOC(f->seed, sizeof(double) * c);
  FALLOC(f->mask, c);
  FALLOC(f->need, c);
  FALLOC(f->asc, sizeof(AscentState) * c);
  FALLOC(f->iters, sizeof(int) * c);
  FALLOC(f->counter, sizeof(int));
  FALLOC(f->trial, sizeof(double) * 4 * c);
#undef FALLOC
  f->cap = c;
  return PA_OK;
}

constexpr size_t kFuSmem = sizeof(Sample) * kChunk;

// One launch of the FP64 form's sums.
template <bool ADJ>
static void fu_sums(pa_followup* f, int n, dim3 grid) {
  k_fu_sums<ADJ><<<grid, kThreads, kFuSmem, f->stream>>>(f->xd, f->pos, f->cm, f->sm, f->cand, f->coef, f->dets, n, f->N,
                                                         f->nifo, f->nch, f->oms, (double*)f->part);
}

// The mixed form's adjoint pass for n points, or those of the list; all_fast:
// none of them needs another form of the phase than the fast one.
static void fu32_adjoint(pa_followup* f, int n, const int* list, bool all_fast) {
  const int P = f->nifo * f->nch;
  auto sums = all_fast ? fu32::k_sums<true, true> : fu32::k_sums<true, false>;
  sums<<<fu32::sum_grid(true, n, P), fu32::kThreads, 0, f->stream>>>(
      f->samp, f->rough, f->chunk, f->pos, f->point, f->seeds, list, f->nlist, n, f->N, f->nifo, f->nch, f->centre,
      (float*)f->part);
  fu32::k_final_adj<<<(n + fu32::kAdjPts - 1) / fu32::kAdjPts, 32 * fu32::kAdjPts, 0, f->stream>>>(
      (const float*)f->part, f->point, f->coef, f->chunk, f->dets, list, f->nlist, n, f->N, f->nifo, f->nch, f->oms,
      f->totals, f->grad);
  f->launches += 2;
}

// Whether n points (host copies) are fast over every chunk, forward and adjoint.
static bool fu32_all_fast(const pa_followup* f, const double* pts, int n) {
  double fo = 0., st2 = 0.;
  for (int k = 0; k < n; k++) {
    const double a = fabs((pts[4 * (size_t)k] + f->oms) * kInv2Pi), b = fabs(2. * pts[4 * (size_t)k + 1] * kInv2Pi);
    if (a > fo || a != a) fo = a;  // (a NaN stays)
    if (b > st2 || b != b) st2 = b;
  }
  return fu32::form_of(fo, st2, f->top, f->N, true) == fu32::kFast;
}

// Forward (and optionally adjoint) evaluation of n points already in
// f->pts; mask (device, may be null) selects the active points; grad: an
// adjoint pass follows, here or later; host_pts: the same points in host memory,
// where the caller has them.
static int fu_eval(pa_followup* f, int n, const unsigned char* mask, bool want_out, bool adjoint,
                   const double* seed_dev, bool grad, const double* host_pts = nullptr) {
  const int P = f->nifo * f->nch;
  if (f->fp64) {
    double* part = (double*)f->part;
    k_fu_prep<<<(n + 127) / 128, 128, 0, f->stream>>>(f->pts, n, mask, f->cand, f->coef, f->dets, f->nifo, f->oms);
    dim3 grid(P, (n + kCandPerCta - 1) / kCandPerCta);
    fu_sums<false>(f, n, grid);
    k_fu_final<<<(n + 7) / 8, 256, 0, f->stream>>>(part, f->pts, f->cand, n, P, f->res, f->F, want_out ? f->out : nullptr,
                                                   seed_dev);
    f->launches += 3;
    if (adjoint) {
      fu_sums<true>(f, n, grid);
      k_fu_final_adj<<<(n + 7) / 8, 256, 0, f->stream>>>(part, f->cand, n, P, f->grad);
      f->launches += 2;
    }
  } else {
    int* list = mask ? f->list : nullptr;
    if (list) FCK(cudaMemsetAsync(f->nlist, 0, sizeof(int), f->stream), "memset");
    auto prep = grad ? fu32::k_prep<true> : fu32::k_prep<false>;
    prep<<<(n + 7) / 8, 64, 0, f->stream>>>(f->pts, n, mask, f->point, f->coef, f->dets, f->gram, f->nifo, f->oms,
                                            f->top, f->N, list, f->nlist);
    fu32::k_sums<false, false><<<fu32::sum_grid(false, n, P), fu32::kThreads, 0, f->stream>>>(
        f->samp, f->rough, f->chunk, f->pos, f->point, nullptr, list, f->nlist, n, f->N, f->nifo, f->nch, f->centre,
        (float*)f->part);
    fu32::k_final<<<(n + 7) / 8, 256, 0, f->stream>>>((const float*)f->part, f->pts, f->point, f->coef, f->dets, list,
                                                      f->nlist, n, f->nifo, f->nch, f->totals, f->F,
                                                      want_out ? f->out : nullptr, seed_dev, f->seeds);
    f->launches += 3;
    if (adjoint) fu32_adjoint(f, n, list, host_pts && fu32_all_fast(f, host_pts, n));
  }
  FCK(cudaGetLastError(), "followup launch");
  return PA_OK;
}

// Adjoint pass only, for the points selected by need[] (device), with the
// constants and seeds of their last forward pass.
static int fu_adjoint(pa_followup* f, int n, const unsigned char* need) {
  const int P = f->nifo * f->nch;
  if (f->fp64) {
    k_fu_select<<<(n + 255) / 256, 256, 0, f->stream>>>(f->cand, n, need);
    fu_sums<true>(f, n, dim3(P, (n + kCandPerCta - 1) / kCandPerCta));
    k_fu_final_adj<<<(n + 7) / 8, 256, 0, f->stream>>>((const double*)f->part, f->cand, n, P, f->grad);
    f->launches += 3;
  } else {
    FCK(cudaMemsetAsync(f->nlist, 0, sizeof(int), f->stream), "memset");
    fu32::k_list<<<(n + 255) / 256, 256, 0, f->stream>>>(need, n, f->list, f->nlist);
    f->launches++;
    fu32_adjoint(f, n, f->list, false);
  }
  FCK(cudaGetLastError(), "followup adjoint launch");
  return PA_OK;
}

static int fu_begin(pa_followup* f, int n) {
  FCK(cudaSetDevice(f->dev), "cudaSetDevice");
  int rc = fu_reserve(f, n);
  if (rc) return rc;
  FCK(cudaEventRecord(f->ev0, f->stream), "event");
  return PA_OK;
}

static int fu_end(pa_followup* f) {
  FCK(cudaEventRecord(f->ev1, f->stream), "event");
  FCK(cudaStreamSynchronize(f->stream), "followup");
  float ms = 0.f;
  FCK(cudaEventElapsedTime(&ms, f->ev0, f->ev1), "event time");
  f->last_ms += ms;
  return PA_OK;
}

// The mixed form's inputs: per chunk the parabola through the first, middle and
// last position, and per sample x u_k and the rest of the position, in FP32 and
// in integers; the matrix of the u_k; what the form of the phase is chosen by.
static void fu32_samples(pa_followup* f, const pa_detector* det, const std::vector<double>& cw,
                         const std::vector<double>& sw, std::vector<float4>* samp, std::vector<int>* rough,
                         std::vector<fu32::Chunk>* chunk) {
  const int N = f->N, L = fu32::kChunk;
  samp->assign((size_t)f->nifo * f->nch * 2 * L, make_float4(0.f, 0.f, 0.f, 0.f));
  rough->assign((size_t)f->nifo * f->nch * 3 * L, 0);
  chunk->resize((size_t)f->nifo * f->nch);
  memset(&f->gram, 0, sizeof(f->gram));
  for (int i = 0; i < N; i++) {
    const double c = cw[i], s = sw[i], u[fu32::kU] = {1., c, s, c * c - s * s, 2. * s * c};
    for (int k = 0; k < fu32::kU; k++)
      for (int l = 0; l <= k; l++) f->gram.g[k][l] += u[k] * u[l];
  }
  for (int k = 0; k < fu32::kU; k++)
    for (int l = 0; l < k; l++) f->gram.g[l][k] = f->gram.g[k][l];
  // the adjoint's centre: the middle sample, a position in the middle of the data
  f->centre.i = (double)(N / 2);
  for (int t = 0; t < 3; t++) f->centre.R[t] = det[0].DetSSB[3 * (size_t)(N / 2) + t];
  f->top = {0., 0., 1, 0};
  // the largest value so far; once it is NaN, no comparison is true and it stays
  auto raise = [](double& top, double v) {
    if (v > top || v != v) top = v;
  };
  for (int p = 0; p < f->nifo * f->nch; p++) {
    const int d = p / f->nch, base = (p - d * f->nch) * L, cnt = std::min(L, N - base);
    fu32::Chunk& h = (*chunk)[p];
    const double* R = det[d].DetSSB + 3 * (size_t)base;
    const int e = cnt - 1, m = e / 2;
    double curv = 0.;
    for (int t = 0; t < 3; t++) {
      // Newton's divided differences on samples 0, m, e
      const double y0 = R[t], ym = R[3 * (size_t)m + t], ye = R[3 * (size_t)e + t];
      double V = 0., A = 0.;
      if (m > 0) {
        const double d1 = (ym - y0) / m;
        A = ((ye - ym) / (e - m) - d1) / e;
        V = d1 - A * m;
      } else if (e > 0) {
        V = (ye - y0) / e;
      }
      h.R0[t] = y0;
      h.V[t] = V;
      h.A[t] = A;
      curv += A * A;
    }
    h.top = {0., sqrt(curv), 0, 0};
    const double b = (double)base, ic = f->centre.i;
    h.db = b - ic;
    h.db2 = b * b - ic * ic;
    for (int t = 0; t < 3; t++) {
      h.dR[t] = h.R0[t] - f->centre.R[t];
      h.dbR[t] = b * h.R0[t] - ic * f->centre.R[t];
    }
    float4* s0 = &(*samp)[(size_t)p * 2 * L];
    for (int j = 0; j < cnt; j++) {
      const int i = base + j;
      const double x = det[d].xDat[i], c = cw[i], s = sw[i];
      double r[3], rr = 0.;
      for (int t = 0; t < 3; t++) {
        r[t] = R[3 * (size_t)j + t] - ((h.A[t] * j + h.V[t]) * j + h.R0[t]);
        rr += r[t] * r[t];
      }
      raise(h.top.rest, sqrt(rr));
      s0[j] = make_float4((float)x, (float)(x * c), (float)(x * s), (float)(x * (c * c - s * s)));
      s0[L + j] = make_float4((float)(x * (2. * s * c)), (float)r[0], (float)r[1], (float)r[2]);
    }
    // sum g j r is left out of sum g i R: 2 x 1024 |r| against i^2 ~ N^2 / 12
    h.top.adj_fast = 2. * L * h.top.rest <= (double)N * N / 12. * 5.96e-8;
    raise(f->top.rest, h.top.rest);
    raise(f->top.curv, h.top.curv);
    f->top.adj_fast &= h.top.adj_fast;
    // integer rests: a unit that holds the largest in 30 bits
    h.unit = 1.;
    if (h.top.rest > 0. && h.top.rest < 1e300) {
      int ex;
      frexp(h.top.rest, &ex);
      h.unit = ldexp(1., ex - 30);
      int* ri = &(*rough)[(size_t)p * 3 * L];
      for (int j = 0; j < cnt; j++)
        for (int t = 0; t < 3; t++)
          ri[t * L + j] = (int)lrint((R[3 * (size_t)j + t] - ((h.A[t] * j + h.V[t]) * j + h.R0[t])) / h.unit);
    }
  }
}

extern "C" {

pa_followup* pa_followup_create(const pa_settings* sett, const pa_detector* det, int nifo, const pa_config* cfg,
                                int* status) {
  pa::TraceRange trace_("pa_followup_create");
  auto ret = [&](int st) {
    if (status) *status = st;
    return (pa_followup*)nullptr;
  };
  pa_followup* f = nullptr;
  if (!sett || !det || nifo < 1 || nifo > PA_MAX_DETECTORS || sett->N < 1)
    return fu_fail(f, PA_ERR_ARG, "pa_followup_create: invalid settings or detectors"), ret(PA_ERR_ARG);
  const pa_config dflt = {PA_PREC_MIXED, PA_PHASE_FIXED, 0, 0};
  const pa_config c = cfg ? *cfg : dflt;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1)
    return fu_fail(f, PA_ERR_NODEV, "pa_followup_create: no CUDA device"), ret(PA_ERR_NODEV);
  if (c.device < 0 || c.device >= ndev)
    return fu_fail(f, PA_ERR_ARG, "pa_followup_create: device %d out of range", c.device), ret(PA_ERR_ARG);
  f = new pa_followup();
  f->dev = c.device;
  f->fp64 = c.precision == PA_PREC_FP64;
  f->N = sett->N;
  f->nifo = nifo;
  f->nch = (sett->N + kChunk - 1) / kChunk;
  f->oms = sett->oms;
  memset(&f->dets, 0, sizeof(f->dets));
  for (int d = 0; d < nifo; d++) {
    memcpy(f->dets.d[d].amod, det[d].amod, sizeof(double) * 9);
    f->dets.d[d].cphir = det[d].cphir;
    f->dets.d[d].sphir = det[d].sphir;
    f->dets.d[d].inv_sig2 = 1. / det[d].sig2;
  }
  auto bail = [&](const char* what, cudaError_t e) {
    g_fu_create_error = std::string("pa_followup_create: ") + what + ": " + cudaGetErrorString(e);
    pa_followup_destroy(f);
    if (status) *status = PA_ERR_CUDA;
    return (pa_followup*)nullptr;
  };
  cudaError_t e;
  if ((e = cudaSetDevice(f->dev)) != cudaSuccess) return bail("cudaSetDevice", e);
  if ((e = cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking)) != cudaSuccess) return bail("stream", e);
  if ((e = cudaEventCreate(&f->ev0)) != cudaSuccess) return bail("event", e);
  if ((e = cudaEventCreate(&f->ev1)) != cudaSuccess) return bail("event", e);
  const int N = sett->N;
  if ((e = cudaMalloc((void**)&f->pos, sizeof(double) * 3 * nifo * (size_t)N)) != cudaSuccess)
    return bail("cudaMalloc", e);
  for (int d = 0; d < nifo; d++)
    if ((e = cudaMemcpy(f->pos + (size_t)d * 3 * N, det[d].DetSSB, sizeof(double) * 3 * N,
                        cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail("upload", e);
  // cos/sin(omr i) (followup init.c:470-475)
  std::vector<double> c64(N), s64(N);
  for (int i = 0; i < N; i++) {
    const double omrt = sett->omr * i;
    c64[i] = cos(omrt);
    s64[i] = sin(omrt);
  }
  if (f->fp64) {
    if ((e = cudaMalloc((void**)&f->xd, sizeof(double) * nifo * (size_t)N)) != cudaSuccess) return bail("cudaMalloc", e);
    if ((e = cudaMalloc((void**)&f->cm, sizeof(double) * N)) != cudaSuccess) return bail("cudaMalloc", e);
    if ((e = cudaMalloc((void**)&f->sm, sizeof(double) * N)) != cudaSuccess) return bail("cudaMalloc", e);
    for (int d = 0; d < nifo; d++)
      if ((e = cudaMemcpy(f->xd + (size_t)d * N, det[d].xDat, sizeof(double) * N, cudaMemcpyHostToDevice)) != cudaSuccess)
        return bail("upload", e);
    if ((e = cudaMemcpy(f->cm, c64.data(), sizeof(double) * N, cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail("upload", e);
    if ((e = cudaMemcpy(f->sm, s64.data(), sizeof(double) * N, cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail("upload", e);
    cudaFuncSetAttribute(k_fu_sums<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFuSmem);
    cudaFuncSetAttribute(k_fu_sums<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFuSmem);
  } else {
    std::vector<float4> samp;
    std::vector<int> rough;
    std::vector<fu32::Chunk> chunk;
    fu32_samples(f, det, c64, s64, &samp, &rough, &chunk);
    if ((e = cudaMalloc((void**)&f->rough, sizeof(int) * rough.size())) != cudaSuccess) return bail("cudaMalloc", e);
    if ((e = cudaMemcpy(f->rough, rough.data(), sizeof(int) * rough.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail("upload", e);
    if ((e = cudaMalloc((void**)&f->samp, sizeof(float4) * samp.size())) != cudaSuccess) return bail("cudaMalloc", e);
    if ((e = cudaMalloc((void**)&f->chunk, sizeof(fu32::Chunk) * chunk.size())) != cudaSuccess)
      return bail("cudaMalloc", e);
    if ((e = cudaMemcpy(f->samp, samp.data(), sizeof(float4) * samp.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail("upload", e);
    if ((e = cudaMemcpy(f->chunk, chunk.data(), sizeof(fu32::Chunk) * chunk.size(), cudaMemcpyHostToDevice)) !=
        cudaSuccess)
      return bail("upload", e);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return bail("set-up", e);
  if (status) *status = PA_OK;
  return f;
}

void pa_followup_destroy(pa_followup* f) {
  if (!f) return;
  cudaSetDevice(f->dev);
  if (f->stream) cudaStreamSynchronize(f->stream);
  fu_free_batch(f);
  void* ps[] = {f->xd, f->pos, f->cm, f->sm, f->samp, f->rough, f->chunk};
  for (void* p : ps)
    if (p) cudaFree(p);
  if (f->ev0) cudaEventDestroy(f->ev0);
  if (f->ev1) cudaEventDestroy(f->ev1);
  if (f->stream) cudaStreamDestroy(f->stream);
  delete f;
}

const char* pa_followup_last_error(const pa_followup* f) {
  return f ? f->err.c_str() : g_fu_create_error.c_str();
}

double pa_followup_last_call_ms(const pa_followup* f) { return f ? f->last_ms : 0.; }
long long pa_followup_kernel_launches(const pa_followup* f) { return f ? f->launches : 0; }

int pa_fstatnet(pa_followup* f, const double* sgnlo, int n, double* out) {
  pa::TraceRange trace_("pa_fstatnet");
  if (!f || !sgnlo || !out || n < 0) return fu_fail(f, PA_ERR_ARG, "pa_fstatnet: invalid arguments");
  if (n == 0) return PA_OK;
  f->last_ms = 0.;
  int rc = fu_begin(f, n);
  if (rc) return rc;
  FCK(cudaMemcpyAsync(f->pts, sgnlo, sizeof(double) * 4 * n, cudaMemcpyHostToDevice, f->stream), "copy");
  if ((rc = fu_eval(f, n, nullptr, true, false, nullptr, false, sgnlo))) return rc;
  FCK(cudaMemcpyAsync(out, f->out, sizeof(double) * 11 * n, cudaMemcpyDeviceToHost, f->stream), "copy");
  return fu_end(f);
}

int pa_fstatnet_grad(pa_followup* f, const double* sgnlo, int n, const double* seed, double* F, double* grad) {
  pa::TraceRange trace_("pa_fstatnet_grad");
  if (!f || !sgnlo || !F || !grad || n < 0) return fu_fail(f, PA_ERR_ARG, "pa_fstatnet_grad: invalid arguments");
  if (n == 0) return PA_OK;
  f->last_ms = 0.;
  int rc = fu_begin(f, n);
  if (rc) return rc;
  FCK(cudaMemcpyAsync(f->pts, sgnlo, sizeof(double) * 4 * n, cudaMemcpyHostToDevice, f->stream), "copy");
  if (seed)
    FCK(cudaMemcpyAsync(f->seed, seed, sizeof(double) * n, cudaMemcpyHostToDevice, f->stream), "copy");
  if ((rc = fu_eval(f, n, nullptr, false, true, seed ? f->seed : nullptr, true, sgnlo))) return rc;
  FCK(cudaMemcpyAsync(F, f->F, sizeof(double) * n, cudaMemcpyDeviceToHost, f->stream), "copy");
  FCK(cudaMemcpyAsync(grad, f->grad, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost, f->stream), "copy");
  return fu_end(f);
}

int pa_followup_ascent(pa_followup* f, double* sgnlo, int n, const pa_ascent_opts* opts, double* out, int* iters) {
  pa::TraceRange trace_("pa_followup_ascent");
  if (!f || !sgnlo || !out || !opts || n < 0) return fu_fail(f, PA_ERR_ARG, "pa_followup_ascent: invalid arguments");
  for (int j = 0; j < 4; j++)
    if (!(opts->scale[j] > 0.)) return fu_fail(f, PA_ERR_ARG, "pa_followup_ascent: scale[%d] must be > 0", j);
  if (n == 0) return PA_OK;
  const double step0 = opts->step0 > 0. ? opts->step0 : 0.25;
  const double min_step = opts->min_step > 0. ? opts->min_step : 1e-3;
  const int max_iter = opts->max_iter > 0 ? opts->max_iter : 100;
  f->last_ms = 0.;
  int rc = fu_begin(f, n);
  if (rc) return rc;
  const int nb = (n + 255) / 256;
  FCK(cudaMemcpyAsync(f->pts, sgnlo, sizeof(double) * 4 * n, cudaMemcpyHostToDevice, f->stream), "copy");
  if ((rc = fu_eval(f, n, nullptr, false, true, nullptr, true))) return rc;
  const double* sc = opts->scale;
  k_asc_init<<<nb, 256, 0, f->stream>>>(f->asc, n, f->pts, f->F, f->grad, sc[0], sc[1], sc[2], sc[3], step0);
  f->launches++;
  int* h_active = nullptr;
  FCK(cudaMallocHost((void**)&h_active, sizeof(int)), "cudaMallocHost");
  for (int it = 0; it < max_iter; it++) {
    // trial points -> f->pts (the evaluation reads them from there)
    k_asc_propose<<<nb, 256, 0, f->stream>>>(f->asc, n, sc[0], sc[1], sc[2], sc[3], min_step, f->pts, f->mask);
    f->launches++;
    if ((rc = fu_eval(f, n, f->mask, false, false, nullptr, true))) break;
    cudaMemsetAsync(f->counter, 0, sizeof(int), f->stream);
    k_asc_decide<<<nb, 256, 0, f->stream>>>(f->asc, n, sc[0], sc[1], sc[2], sc[3], f->F, f->need, f->counter);
    f->launches++;
    // gradient at the accepted points: the trial evaluation left their
    // constants and adjoint seeds in cand[]; only the adjoint pass runs
    if ((rc = fu_adjoint(f, n, f->need))) break;
    k_asc_take_grad<<<nb, 256, 0, f->stream>>>(f->asc, n, sc[0], sc[1], sc[2], sc[3], f->need, f->grad);
    f->launches++;
    if (cudaGetLastError() != cudaSuccess) {
      rc = fu_fail(f, PA_ERR_CUDA, "pa_followup_ascent: launch failed");
      break;
    }
    cudaMemcpyAsync(h_active, f->counter, sizeof(int), cudaMemcpyDeviceToHost, f->stream);
    if (cudaStreamSynchronize(f->stream) != cudaSuccess) {
      rc = fu_fail(f, PA_ERR_CUDA, "pa_followup_ascent: %s", cudaGetErrorString(cudaGetLastError()));
      break;
    }
    if (*h_active == 0) break;
  }
  cudaFreeHost(h_active);
  if (rc) return rc;
  // final points and their fstat_out
  k_asc_export<<<nb, 256, 0, f->stream>>>(f->asc, n, f->pts, f->iters);
  f->launches++;
  if ((rc = fu_eval(f, n, nullptr, true, false, nullptr, false))) return rc;
  FCK(cudaMemcpyAsync(sgnlo, f->pts, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost, f->stream), "copy");
  FCK(cudaMemcpyAsync(out, f->out, sizeof(double) * 11 * n, cudaMemcpyDeviceToHost, f->stream), "copy");
  if (iters) FCK(cudaMemcpyAsync(iters, f->iters, sizeof(int) * n, cudaMemcpyDeviceToHost, f->stream), "copy");
  return fu_end(f);
}

}  // extern "C"

// ---------------------------------------------------------------------
// The reference simplex as a resumable state machine per point, so that
// the evaluations of all points can be batched.  Mirrors amoeba()
// (followup.c:1126-1174) step for step: make_simplex (:971-984),
// evaluate_simplex (:986-1009), simplex_extremes (:1011-1040),
// simplex_bearings (:1042-1053), update_simplex (:1055-1087),
// contract_simplex (:1089-1118), check_tol (:1120-1124, ZEPS 1e-14).
// ---------------------------------------------------------------------
namespace {

enum SxState { SX_INIT, SX_REFLECT, SX_EXPAND, SX_CONTRACT, SX_SHRINK, SX_DONE };

struct Simplex {
  double sx[5][4];
  double fx[5][11];
  double mid[4], line[4], next[4];
  int ihi, ilo, inhi;
  int state;
  int nev;
};

void sx_extremes(Simplex& S) {
  int hi, lo, nhi;
  if (S.fx[0][5] > S.fx[1][5]) {
    hi = 0;
    lo = nhi = 1;
  } else {
    hi = 1;
    lo = nhi = 0;
  }
  for (int i = 2; i < 5; i++) {
    if (S.fx[i][5] <= S.fx[lo][5]) lo = i;
    else if (S.fx[i][5] > S.fx[hi][5]) {
      nhi = hi;
      hi = i;
    } else if (S.fx[i][5] > S.fx[nhi][5]) nhi = i;
  }
  S.ihi = hi;
  S.ilo = lo;
  S.inhi = nhi;
}

// Loop head of amoeba: extremes, bearings, tolerance; returns true when done.
bool sx_head(Simplex& S, double tol, int max_evals) {
  sx_extremes(S);
  for (int j = 0; j < 4; j++) S.mid[j] = 0.0;
  for (int i = 0; i < 5; i++)
    if (i != S.ihi)
      for (int j = 0; j < 4; j++) S.mid[j] += S.sx[i][j];
  for (int j = 0; j < 4; j++) {
    S.mid[j] /= 4;
    S.line[j] = S.sx[S.ihi][j] - S.mid[j];
  }
  const double fmax = S.fx[S.ihi][5], fmin = S.fx[S.ilo][5];
  if (fabs(fmax - fmin) < (fabs(fmax) + fabs(fmin)) * tol + 1e-14) return true;
  if (max_evals > 0 && S.nev >= max_evals) return true;
  return false;
}

void sx_propose(Simplex& S, double scale) {
  for (int j = 0; j < 4; j++) S.next[j] = S.mid[j] + scale * S.line[j];
}

}  // namespace

extern "C" int pa_followup_simplex(pa_followup* f, double* sgnlo, int n, const double* pc2, double tol,
                                   int max_evals, double* out, int* nevals) {
  pa::TraceRange trace_("pa_followup_simplex");
  if (!f || !sgnlo || !pc2 || !out || n < 0) return fu_fail(f, PA_ERR_ARG, "pa_followup_simplex: invalid arguments");
  if (n == 0) return PA_OK;
  std::vector<Simplex> S(n);
  for (int k = 0; k < n; k++) {
    Simplex& s = S[k];
    for (int i = 0; i < 5; i++)
      for (int j = 0; j < 4; j++) s.sx[i][j] = sgnlo[4 * k + j];
    for (int i = 0; i < 4; i++) s.sx[i][i] = s.sx[i][i] + pc2[i];
    s.state = SX_INIT;
    s.nev = 0;
  }
  std::vector<double> pts, res;
  std::vector<std::pair<int, int>> who;  // (point, vertex or -1 for next)
  double total_ms = 0.;
  int rc = PA_OK;
  for (;;) {
    pts.clear();
    who.clear();
    for (int k = 0; k < n; k++) {
      Simplex& s = S[k];
      if (s.state == SX_DONE) continue;
      if (s.state == SX_INIT) {
        for (int i = 0; i < 5; i++) {
          pts.insert(pts.end(), s.sx[i], s.sx[i] + 4);
          who.push_back({k, i});
        }
      } else if (s.state == SX_SHRINK) {
        for (int i = 0; i < 5; i++)
          if (i != s.ilo) {
            pts.insert(pts.end(), s.sx[i], s.sx[i] + 4);
            who.push_back({k, i});
          }
      } else {
        pts.insert(pts.end(), s.next, s.next + 4);
        who.push_back({k, -1});
      }
    }
    if (who.empty()) break;
    const int m = (int)who.size();
    res.resize((size_t)m * 11);
    if ((rc = pa_fstatnet(f, pts.data(), m, res.data()))) break;
    total_ms += f->last_ms;
    // feed the results back, in the order amoeba() would see them
    size_t r = 0;
    while (r < who.size()) {
      const int k = who[r].first;
      Simplex& s = S[k];
      if (s.state == SX_INIT || s.state == SX_SHRINK) {
        for (; r < who.size() && who[r].first == k; r++) {
          memcpy(s.fx[who[r].second], &res[r * 11], sizeof(double) * 11);
          s.nev++;
        }
        s.state = SX_REFLECT;  // to the loop head
        if (sx_head(s, tol, max_evals)) s.state = SX_DONE;
        else sx_propose(s, -1.0);
        continue;
      }
      const double* f2 = &res[r * 11];
      r++;
      s.nev++;
      const int st = s.state;
      // update_simplex: accept when better than the current worst
      const bool upd = f2[5] < s.fx[s.ihi][5];
      if (upd) {
        for (int j = 0; j < 4; j++) s.sx[s.ihi][j] = s.next[j];
        memcpy(s.fx[s.ihi], f2, sizeof(double) * 11);
      }
      bool head = false;
      if (st == SX_REFLECT) {
        if (s.fx[s.ihi][5] < s.fx[s.ilo][5]) {
          s.state = SX_EXPAND;
          sx_propose(s, -2.0);
        } else if (s.fx[s.ihi][5] > s.fx[s.inhi][5]) {
          s.state = SX_CONTRACT;
          sx_propose(s, 0.5);
        } else {
          head = true;
        }
      } else if (st == SX_EXPAND) {
        head = true;
      } else if (st == SX_CONTRACT) {
        if (upd) {
          head = true;
        } else {
          for (int i = 0; i < 5; i++)
            if (i != s.ilo)
              for (int j = 0; j < 4; j++) s.sx[i][j] = (s.sx[s.ilo][j] + s.sx[i][j]) * 0.5;
          s.state = SX_SHRINK;
        }
      }
      if (head) {
        s.state = SX_REFLECT;
        if (sx_head(s, tol, max_evals)) s.state = SX_DONE;
        else sx_propose(s, -1.0);
      }
    }
  }
  f->last_ms = total_ms;
  if (rc) return rc;
  for (int k = 0; k < n; k++) {
    const Simplex& s = S[k];
    for (int j = 0; j < 4; j++) sgnlo[4 * k + j] = s.sx[s.ilo][j];
    memcpy(out + (size_t)11 * k, s.fx[s.ilo], sizeof(double) * 11);
    if (nevals) nevals[k] = s.nev;
  }
  return PA_OK;
}
