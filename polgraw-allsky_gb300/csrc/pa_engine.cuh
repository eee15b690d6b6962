// pa_engine.cuh -- device kernels of the coherent-search hot path and the
// templated engine that enqueues them.  Included by the per-precision
// translation units only.
//
// Reference correspondence (search/network/src-cpu):
//   k_prelude_mod   modvir (settings.c:281-325), shft/shftf/_tmp1 and the
//                   prelude phase modulation (jobcore.c:277-313)
//   resample FFTs   jobcore.c:319-362 (pass A/B with PlainLoader; the
//                   interpolating inverse at half length: HalfShiftLoader,
//                   InterpStore)
//   k_resample      FP32 forms: spline() (auxi.c:56-81), splint/splintpad
//                   (auxi.c:83-122), 1/sig2 (jobcore.c:386-389), aa and bb
//                   (jobcore.c:375-393)
//   k_spline_fwd/bwd, k_splint   the same for the FP64 form (aa, bb: last CTA
//                   of k_prelude_mod)
//   SpinLoader      spindown phase modulation (jobcore.c:455-623)
//   FstatStore      F = |Xa|^2/aa + |Xb|^2/bb (jobcore.c:635-638)
//   k_normthresh    FStat() block means and normalisation (auxi.c:214-240),
//                   threshold, run clustering, argmax (jobcore.c:659-669)
#pragma once
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>

#include "pa_engine.h"
#include "pa_fft.cuh"
#include "pa_pair.cuh"
#include "pa_sincos.cuh"

namespace pa {

enum { PM_F64 = 0, PM_FIXED = 1, PM_FF = 2 };

constexpr double kInvTwoPi = 0.15915494309189535;
constexpr double kTurnsPerRad64 = 2.9358905032820014e18;  // 2^64 / (2 pi)
// 2 pi as the sum of three floats with 12, 24 and 24 significant bits; k*A
// is exact for |k| < 2^12
constexpr float kTwoPiF_A = 6.28125f;
constexpr float kTwoPiF_B = 1.9353071693331003e-3f;
constexpr float kTwoPiF_C = 1.0253131677018246e-11f;
constexpr float kInvTwoPiF = 0.15915494309189533577f;

// x mod 1 as a 64-bit fixed-point fraction (t / 2^64), computed exactly
// from the bits of x with integer operations only: x = m 2^(e-1075) with the
// 53-bit integer significand m, so x 2^64 mod 2^64 = m << (e - 1011) (or
// >> for negative shifts), negated for x < 0.
__device__ __forceinline__ uint64_t turns_fixed(double x) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((bits >> 52) & 0x7ff);
  if (e == 0) return 0ull;  // zero or subnormal: |x| < 2^-1022
  const unsigned long long m = (bits & 0xfffffffffffffull) | 0x10000000000000ull;
  const int sh = e - 1011;
  unsigned long long t;
  if (sh >= 64) t = 0ull;
  else if (sh >= 0) t = m << sh;
  else if (sh > -64) t = m >> (-sh);
  else t = 0ull;
  return (bits >> 63) ? (0ull - t) : t;
}

// ------------------------------------------------------------------
// prelude: modvir + time shift + prelude phase modulation

// Sum of two values over a 256-thread block in a fixed order (xor tree in
// each warp, then warps in index order); the result is valid in every thread.
__device__ __forceinline__ void block_sum2(double& a, double& b, double (*red)[8]) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, off);
    b += __shfl_xor_sync(0xffffffffu, b, off);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = a;
    red[1][w] = b;
  }
  __syncthreads();
  double sa = 0., sb = 0.;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
    sa += red[0][k];
    sb += red[1][k];
  }
  __syncthreads();
  a = sa;
  b = sb;
}

// aa = sum_n (sum_i a^2)/sig2_n in detector order (jobcore.c:375-393) and bb,
// from the partial sums of k_prelude_mod in a fixed order, by one block (FP64 form).
template <typename R>
__device__ void sum_parts(const double* part, int nblk, int nifo, const DetConst* dc, double* sums, R* sums_r,
                          double (*red)[8]) {
  double acc = 0.;  // thread 0: aa, thread 1: bb (of the first warp)
  for (int dd = 0; dd < nifo; ++dd) {
    double sa = 0., sb = 0.;
    for (int k = threadIdx.x; k < nblk; k += blockDim.x) {
      sa += __ldcg(&part[((size_t)dd * nblk + k) * 2 + 0]);
      sb += __ldcg(&part[((size_t)dd * nblk + k) * 2 + 1]);
    }
    __syncthreads();
    block_sum2(sa, sb, red);
    if (threadIdx.x < 32) acc += (threadIdx.x & 1 ? sb : sa) / dc[dd].sig2;
  }
  if (threadIdx.x < 2) {
    const double inv = 1.0 / acc;
    sums[threadIdx.x] = acc;
    sums[2 + threadIdx.x] = inv;
    sums_r[threadIdx.x] = (R)inv;
  }
}

// The same for the FP32 forms, by a block of 128 in k_resample: the warps share
// the detectors (four warps on one, two on each of two, else one a detector), so
// that the partial sums are loaded at once and the detectors' FP64 chains run side
// by side: the block starts after the wait and is waited for like the others.  One
// detector after the other, by the whole block: one short sky point 40.4 us on the
// device, 96 x 200 spindowns 22.26 ms; so 40.2 us and 22.22 ms, 24 x 100 of three
// detectors 3.91 -> 3.89 ms.
__device__ __forceinline__ void sum_parts_f32(const double* part, int nblk, int nifo, const DetConst* dc, double* sums,
                                              float* sums_r) {
  __shared__ double red[kMaxDet][4][2];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int share = nifo == 1 ? 4 : (nifo == 2 ? 2 : 1);  // warps of a detector
  const int slice = w % share;
  for (int dd = w / share; dd < nifo; dd += 4 / share) {
    const double2* p = reinterpret_cast<const double2*>(part) + (size_t)dd * nblk;
    double a = 0., b = 0.;
#pragma unroll 8
    for (int k = slice * 32 + lane; k < nblk; k += 32 * share) {
      const double2 v = __ldcg(p + k);
      a += v.x;
      b += v.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, off);
      b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    if (lane == 0) {
      red[dd][slice][0] = a;
      red[dd][slice][1] = b;
    }
  }
  __syncthreads();
  if (w) return;
  // lanes 2 dd (aa) and 2 dd + 1 (bb), then both sums in detector order
  double v = 0.;
  if (lane < 2 * nifo) {
    for (int q = 0; q < share; ++q) v += red[lane >> 1][q][lane & 1];
    v /= dc[lane >> 1].sig2;
  }
  double acc = 0.;
  for (int dd = 0; dd < nifo; ++dd) acc += __shfl_sync(0xffffffffu, v, 2 * dd + (lane & 1));
  if (lane < 2) {
    const double inv = 1.0 / acc;
    sums[lane] = acc;
    sums[2 + lane] = inv;
    sums_r[lane] = (float)inv;
  }
}

// The FP32 forms' time shift n . R of a sample at D, with fused multiply-adds
// (shft1_fma is the same expression at sample 0).
__device__ __forceinline__ double time_shift(const SkyArgs& sky, const double* D) {
  return fma(sky.nS[0], D[0], fma(sky.nS[1], D[1], __dmul_rn(sky.nS[2], D[2])));
}

// One sample a thread.  The FP32 forms take blocks of 128, so that the FP64
// operations (about 25 a sample, at 2 lanes per clock and SM) spread over the
// SMs also for the shortest segments; their aa and bb are summed in k_resample,
// off this kernel's path.
template <typename R> constexpr int mod_threads() { return sizeof(R) == 4 ? 128 : 256; }

template <typename R, int PM>
__global__ void __launch_bounds__(mod_threads<R>())
    k_prelude_mod(const double* __restrict__ xDat, const double* __restrict__ DetSSB,
                  const R* __restrict__ cosmodf, const R* __restrict__ sinmodf,
                  const DetConst* __restrict__ dc, const SkyArgs sky, int N, int NP,
                  typename CT<R>::T* __restrict__ xin, double* __restrict__ shftf, void* ph0,
                  double* __restrict__ part, double* __restrict__ sums, R* __restrict__ sums_r,
                  unsigned int* __restrict__ counter) {
  typedef typename CT<R>::T T;
  CtaTrace trace_(KK_PRELUDE_MOD);
  const int d = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  R a2r = 0, b2r = 0;
  pdl_wait();
  pdl_go();
  if (i < N) {
    const DetConst& k = dc[d];
    // modvir, settings.c:303-322
    // FP32 forms read the FP32 copies: no double-to-float conversion per
    // thread (conversions run on the FP64 pipe)
    const bool f32 = sizeof(R) == 4;
    const R cosalfr = f32 ? (R)sky.cosalfr_f[d] : (R)sky.cosalfr[d];
    const R sinalfr = f32 ? (R)sky.sinalfr_f[d] : (R)sky.sinalfr[d];
    const R cm = cosmodf[i], sm = sinmodf[i];
    const R c = cosalfr * cm + sinalfr * sm;
    const R s = sinalfr * cm - cosalfr * sm;
    const R cosdel = f32 ? (R)sky.cosdel_f : (R)sky.cosdel, sindel = f32 ? (R)sky.sindel_f : (R)sky.sindel;
    const R c2d = cosdel * cosdel, c2sd = sindel * cosdel;
    const R c2s = (R)2 * c * c, cs = c * s;
#define PA_AMOD(j) (f32 ? (R)k.amod_f[j] : (R)k.amod[j])
    const R k0 = PA_AMOD(0), k1 = PA_AMOD(1), k2 = PA_AMOD(2), k3 = PA_AMOD(3), k4 = PA_AMOD(4),
            k5 = PA_AMOD(5), k6 = PA_AMOD(6), k7 = PA_AMOD(7), k8 = PA_AMOD(8);
#undef PA_AMOD
    const R two_m = (R)2 - c2d;
    const R aa = k0 * two_m * c2s + k1 * two_m * (R)2 * cs + k2 * c2sd * c + k3 * c2sd * s -
                 k0 * two_m + k4 * c2d;
    const R bb = k5 * sindel * c2s + k6 * sindel * (R)2 * cs + k7 * cosdel * c + k8 * cosdel * s -
                 k5 * sindel;
    a2r = aa * aa;
    b2r = bb * bb;
    // shft, shftf, _tmp1 (jobcore.c:285-295)
    const double* D = DetSSB + 3 * ((size_t)d * N + i);
    const size_t o = (size_t)d * N + i, op = (size_t)d * NP + i;
    const double di = (double)i;
    R sp, cp;
    if (sizeof(R) == 8) {
      // FP64 form: the reference's rounding sequence (no FMA contraction):
      // shftf[0] must be exactly 0, as shft1 comes from the same expression
      // on the host; a contracted product would leave +-1 ulp there and push
      // the spline abscissa 2(i - shftf) below 0, where splint returns 0
      // (auxi.c:89).
      const double shft = __dadd_rn(__dadd_rn(__dmul_rn(sky.nS[0], D[0]), __dmul_rn(sky.nS[1], D[1])),
                                    __dmul_rn(sky.nS[2], D[2]));
      shftf[o] = shft - sky.shft1[d];
      const double tmp1 = __dadd_rn(__dmul_rn(di, di), __dmul_rn((double)(2 * i), shft));
      reinterpret_cast<double*>(ph0)[o] = tmp1;
      // prelude phase het0 i + oms shft (jobcore.c:299), FP64
      const double phase = __dadd_rn(__dmul_rn(sky.het0, di), __dmul_rn(sky.oms, shft));
      double sd, cd;
      sincos_fast(phase, &sd, &cd);
      sp = (R)sd;
      cp = (R)cd;
    } else {
      const double shft = time_shift(sky, D);
      // 2 i shft, the non-integer part of _tmp1 = i^2 + 2 i shft
      const double p2 = __dmul_rn(di + di, shft);
      const uint64_t ii2 = (uint64_t)i * (uint64_t)i;
      if (PM == PM_FIXED) {
        // spindown phase s1(ss) tmp1 = s1(ss_base) tmp1 + (ss - ss_base) (M5 tmp1)
        // as 64-bit fixed-point turns: the i^2 part exactly in integers from
        // the fixed-point coefficients, the 2 i shft part from its FP64 value
        const uint64_t A = sky.s1f * ii2 + turns_fixed(sky.s1_0 * p2);
        const uint64_t B = sky.m5f * ii2 + turns_fixed(sky.M5 * p2);
        reinterpret_cast<uint4*>(ph0)[op] = make_uint4((unsigned)A, (unsigned)(A >> 32), (unsigned)B, (unsigned)(B >> 32));
      } else {
        const double tmp1 = (double)ii2 + p2;
        if (PM == PM_FF) {
          const float hi = (float)tmp1;
          reinterpret_cast<float2*>(ph0)[op] = make_float2(hi, (float)(tmp1 - (double)hi));
        } else {
          reinterpret_cast<double*>(ph0)[op] = tmp1;
        }
      }
      // prelude phase het0 i + oms shft (jobcore.c:299) in fixed-point
      // turns: het0/2pi exactly in integers, oms shft/2pi from its FP64 value
      const uint64_t t = sky.h0f * (uint64_t)i + turns_fixed(sky.oms_t * shft);
      float sf, cf;
      sincospif((float)(int)(t >> 32) * 4.656612873077393e-10f, &sf, &cf);
      sp = (R)sf;
      cp = (R)cf;
    }
    const R x = (R)xDat[(size_t)d * N + i];
    const R xa = x * aa, xb = x * bb;
    // x a exp(-i phase)
    if constexpr (sizeof(R) == 4) {
      reinterpret_cast<float4*>(xin)[o] = make_float4(xa * cp, xb * cp, -xa * sp, -xb * sp);
    } else {
      xin[((size_t)d * 2 + 0) * N + i] = mk(xa * cp, -xa * sp);
      xin[((size_t)d * 2 + 1) * N + i] = mk(xb * cp, -xb * sp);
    }
  }
  // deterministic block reduction of a^2, b^2: xor tree of each warp in the
  // working precision, warps summed in FP64 in index order
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a2r += __shfl_xor_sync(0xffffffffu, a2r, off);
    b2r += __shfl_xor_sync(0xffffffffu, b2r, off);
  }
  __shared__ double red[2][8];
  __shared__ bool last;
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = (double)a2r;
    red[1][threadIdx.x >> 5] = (double)b2r;
  }
  __syncthreads();
  double a2 = 0., b2 = 0.;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      a2 += red[0][k];
      b2 += red[1][k];
    }
  if (threadIdx.x == 0) {
    part[((size_t)d * gridDim.x + blockIdx.x) * 2 + 0] = a2;
    part[((size_t)d * gridDim.x + blockIdx.x) * 2 + 1] = b2;
  }
  if (sizeof(R) == 4) return;
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned int done = atomicAdd(counter, 1u);
    last = done == gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (!last) return;
  // the last CTA to finish
  sum_parts(part, gridDim.x, gridDim.y, dc, sums, sums_r, red);
  if (threadIdx.x == 0) *counter = 0u;
}

// ------------------------------------------------------------------
// FFT loaders / storers

// The zero-padded input of a transform, FP64 form.
template <typename R> struct PlainLoader {
  typedef typename CT<R>::T T;
  static constexpr int kTraceKind = KK_FFT_FWD_A;
  const T* in;   // [batch][2][ld]
  int len, ld;
  __device__ __forceinline__ void load2(int batch, int n, T& a, T& b) const {
    if (n < len) {
      a = in[((size_t)batch * 2 + 0) * ld + n];
      b = in[((size_t)batch * 2 + 1) * ld + n];
    } else {
      a = b = mk((R)0, (R)0);
    }
  }
};

// FP32 forms: arrays of pairs, {a.re, b.re, a.im, b.im} per element, so that
// every pass reads and writes 16 bytes of one array.
struct PairLoader {
  static constexpr int kTraceKind = KK_FFT_FWD_A;
  const float4* in;  // [batch][len]
  int len;
  // the passes' interface (pa_pair.cuh)
  template <int NIN, int NCHK> struct Ahead {
    static constexpr int v = 8;
  };
  struct Ctx {
    const float4* p;
    int left;
  };
  typedef P2 Raw;
  __device__ __forceinline__ int count() const { return len; }
  __device__ __forceinline__ Ctx begin(int batch, int n0, int) const { return Ctx{after_wait(in) + (size_t)batch * len + n0, len - n0}; }
  __device__ __forceinline__ void next(Ctx&) const {}
  __device__ __forceinline__ Raw fetch(const Ctx& k, int off) const { return off < k.left ? pld(k.p + off) : pzero(); }
  __device__ __forceinline__ P2 value(const Ctx&, const Raw& r, int) const { return r; }
};
// The results of a transform as pairs, scaled.
template <int KIND> struct PairStore {
  static constexpr int kTraceKind = KIND;
  float4* out;  // [batch][ldo]
  int ldo;
  float scale;
  struct Ctx {};
  __device__ __forceinline__ Ctx begin() const { return Ctx{}; }
  __device__ __forceinline__ void put(const Ctx&, int batch, int k1, int k2, P2 v) const {
    const f2 s = dup(scale);
    pst(out + (size_t)batch * ldo + k1 + (k2 << 8), P2{mul2(v.re, s), mul2(v.im, s)});
  }
};

// The interpolating inverse transform of jobcore.c:338-362 at half length.
// The reference keeps bins [0, nyqst) of the length-nfft spectrum X, moves
// [nyqst, nfft) up by Ninterp - nfft = nfft and inverse-transforms at length
// Ninterp = 2 nfft with scale 2/Ninterp.  With that remap the output is
//   y[2m]   = x[m]                                  (the input itself)
//   y[2m+1] = (1/nfft) sum_j X[j] s_j e^{i pi j/nfft} e^{2 pi i j m/nfft}
// with s_j = +1 below nyqst and -1 from it (the moved bins pick up
// e^{i pi (2m+1)} = -1), i.e. an inverse FFT of length nfft of the
// phase-shifted spectrum: half the transform length, and no transform of the
// zero gap.  This loader feeds that transform; InterpStore interleaves (FP32
// forms: HalfShiftPair feeds it, and the spline reads x and the transform).
template <typename R> struct HalfShiftLoader {
  typedef typename CT<R>::T T;
  static constexpr int kTraceKind = KK_FFT_INV_A;
  const T* spec;    // [batch][2][nfft]
  const T* twlo;    // e^{+2 pi i m/Ninterp}, m < 1024
  const T* twhi;    // e^{+2 pi i 1024 m/Ninterp}
  int nfft, nyqst;
  __device__ __forceinline__ T phase(int j) const {
    const T w = cmul(__ldg(&twlo[j & 1023]), __ldg(&twhi[j >> 10]));
    return j < nyqst ? w : mk(-w.x, -w.y);
  }
  __device__ __forceinline__ void load2(int batch, int j, T& a, T& b) const {
    const T w = phase(j);
    a = cmul(spec[((size_t)batch * 2 + 0) * nfft + j], w);
    b = cmul(spec[((size_t)batch * 2 + 1) * nfft + j], w);
  }
};
struct HalfShiftPair {
  static constexpr int kTraceKind = KK_FFT_INV_A;
  const float4* spec;   // [batch][nfft]
  const float2* twlo;   // as HalfShiftLoader
  const float2* twhi;
  int nfft, nyqst;
  template <int NIN, int NCHK> struct Ahead {
    static constexpr int v = 4;
  };
  struct Ctx {
    const float4* p;
    int n0;
  };
  struct Raw {
    P2 v;
    float2 wl, wh;
  };
  __device__ __forceinline__ int count() const { return nfft; }
  __device__ __forceinline__ Ctx begin(int batch, int n0, int) const { return Ctx{after_wait(spec) + (size_t)batch * nfft + n0, n0}; }
  __device__ __forceinline__ void next(Ctx&) const {}
  __device__ __forceinline__ Raw fetch(const Ctx& k, int off) const {
    const int j = k.n0 + off;
    return Raw{pld(k.p + off), __ldg(&twlo[j & 1023]), __ldg(&twhi[j >> 10])};
  }
  __device__ __forceinline__ P2 value(const Ctx& k, const Raw& r, int off) const {
    const float2 w = cmul(r.wl, r.wh);
    return k.n0 + off < nyqst ? pmul(r.v, w) : pmul(r.v, -w.x, -w.y);
  }
};

// Most spindowns in one launch of the spindown passes (the buffers are sized
// for at most 128).
constexpr int kSpinBatchMax = 128;

// het1 = fmod(ss M4, M0), wrapped into [0, M0) (jobcore.c:466-467), as
// 64-bit fixed-point turns: round-to-nearest-even of het1 2^64 / (2 pi),
// saturated as __double2ull_rn does.  fmod is exact and the two products
// are single roundings, so the host and the device give the same bits.
inline uint64_t het1_turns_fixed(int ss, double M4, double M0) {
  double het1 = fmod(ss * M4, M0);
  if (het1 < 0) het1 += M0;
  const double x = het1 * kTurnsPerRad64;
  if (!(x > 0.)) return 0;
  if (x >= 18446744073709551616.0) return ~0ull;
  // round half to even without depending on the host's rounding mode: below
  // 2^53, x - floor(x) is exact; from 2^53 on, x is an integer
  uint64_t r = (uint64_t)x;
  if (x < 9007199254740992.0) {
    const double fr = x - (double)r;
    if (fr > 0.5 || (fr == 0.5 && (r & 1))) ++r;
  }
  return r;
}

// Per-launch spindown constants of each batch item, formed on the host and
// passed by value with the loader, so that no CTA of pass A waits on a chain
// of FP64 operations before its first phase.  het1 = fmod(ss M4, M0) wrapped
// (jobcore.c:466-467), s1 = ss M5 + s1_0 (one rounding).
struct SpinHet64 {  // FP64 form
  double het1[kSpinBatchMax], s1[kSpinBatchMax];
};
template <int PM> struct SpinHet {  // PM_FIXED
  unsigned long long H[kSpinBatchMax];  // het1 as 64-bit fixed-point turns
};
template <> struct SpinHet<PM_F64> {
  unsigned long long H[kSpinBatchMax];
  double s1t[kSpinBatchMax];  // s1 / 2 pi
};
template <> struct SpinHet<PM_FF> {
  float4 c[kSpinBatchMax];  // s1 and het1 as two floats each
};

inline void spin_het_fill(SpinHet<PM_FIXED>& h, int k, int ss, const SkyArgs& sky, int) {
  h.H[k] = het1_turns_fixed(ss, sky.M4, sky.M0);
}
inline void spin_het1_s1(int ss, const SkyArgs& sky, int s0_flag, double* het1, double* s1) {
  *het1 = fmod(ss * sky.M4, sky.M0);
  if (*het1 < 0) *het1 += sky.M0;
  *s1 = s0_flag ? 0. : fma((double)ss, sky.M5, sky.s1_0);
}
inline void spin_het_fill(SpinHet64& h, int k, int ss, const SkyArgs& sky, int s0_flag) {
  spin_het1_s1(ss, sky, s0_flag, &h.het1[k], &h.s1[k]);
}
inline void spin_het_fill(SpinHet<PM_F64>& h, int k, int ss, const SkyArgs& sky, int s0_flag) {
  double het1, s1;
  spin_het1_s1(ss, sky, s0_flag, &het1, &s1);
  h.H[k] = het1_turns_fixed(ss, sky.M4, sky.M0);
  h.s1t[k] = s1 * kInvTwoPi;
}
inline void spin_het_fill(SpinHet<PM_FF>& h, int k, int ss, const SkyArgs& sky, int s0_flag) {
  double het1, s1;
  spin_het1_s1(ss, sky, s0_flag, &het1, &s1);
  const float s1h = (float)s1, h1h = (float)het1;
  h.c[k] = make_float4(s1h, (float)(s1 - (double)s1h), h1h, (float)(het1 - (double)h1h));
}

// (a * b) mod 2^64 for a 64-bit a and a 32-bit b
__device__ __forceinline__ uint64_t mul64x32(uint64_t a, unsigned b) {
  return (uint64_t)(unsigned)a * b + ((uint64_t)((unsigned)(a >> 32) * b) << 32);
}

// High word of a t mod 1, for products of any size (a call: the compiler would
// issue a rare branch's FP64 operations for every sample).
static __device__ __noinline__ unsigned far_turns(double a, double t) { return (unsigned)(turns_fixed(a * t) >> 32); }

// Phase-modulated detector sum of the spindown loop (jobcore.c:455-623):
//   x_{a,b}[n] = sum_d xm_{a,b,d}[n] exp(-i (het1 n + s1 tmp1_d[n]))  (n < N)
// FP64 form:
struct SpinLoader64 {
  static constexpr int kTraceKind = KK_SPIN_A;
  const double2* xm;   // [nifo][2][N]
  const double* tmp1;  // [nifo][N]
  int N, nifo;
  SpinHet64 het;

  __device__ __forceinline__ void load2(int batch, int n, double2& va, double2& vb) const {
    va = vb = mk(0., 0.);
    if (n >= N) return;
    const double het1 = het.het1[batch], s1 = het.s1[batch];
    for (int d = 0; d < nifo; ++d) {
      const double2 xa = xm[((size_t)d * 2 + 0) * N + n], xb = xm[((size_t)d * 2 + 1) * N + n];
      // het1*i + s1*_tmp1 with the reference's rounding (jobcore.c:606)
      const double ph = __dadd_rn(__dmul_rn(het1, (double)n), __dmul_rn(s1, tmp1[(size_t)d * N + n]));
      double sn, cs;
      sincos_fast(ph, &sn, &cs);
      // x * (cos - i sin)
      va.x += xa.x * cs + xa.y * sn;
      va.y += xa.y * cs - xa.x * sn;
      vb.x += xb.x * cs + xb.y * sn;
      vb.y += xb.y * cs - xb.x * sn;
    }
  }
};

// FP32 forms (pa_pair.cuh).  The data xm and the phase terms lie in two
// arrays of 16 (or 8) bytes per detector and sample, so that each load of a
// warp reads whole 128-byte lines; a thread takes all detectors of its
// position, one sine and cosine each for both arrays.  The arrays have zeros
// behind the N samples (stride NP), so that the lanes of a warp that reaches
// the last row need no condition of their own.  NIFO: the number of
// detectors (0: any, without loads ahead).
template <int PM> struct SpinTerm {
  typedef uint2 T;  // FP64 phase: tmp1; two-float phase: float2
};
template <> struct SpinTerm<PM_FIXED> {
  typedef uint4 T;  // A, B
};
template <int PM, int NIFO> struct SpinLoader {
  static constexpr int kTraceKind = KK_SPIN_A;
  typedef typename SpinTerm<PM>::T Term;
  static constexpr int ND = NIFO ? NIFO : 1;
  static constexpr bool kQuarters = NIFO > 0;
  // positions loaded ahead: of the numbers that the 128 registers of a thread
  // hold beside the NIN values, or nearly (8 to 48 bytes are spilled in instances
  // of two and three detectors), the fastest
  template <int NIN, int NCHK> struct Ahead {
    static constexpr int v =
        NIFO == 0 ? 0 : (NIFO == 1 ? 4 : (NIFO == 2 ? (NIN < 16 ? 3 : 1) : (NIN < 16 || NCHK > 0 ? 1 : 0)));
  };
  const float4* xm;  // [nifo][NP] {a.re, b.re, a.im, b.im}
  const Term* ph;    // [nifo][NP]
  int N, NP, nifo, ss_rel, s0_flag;  // ss_rel: first spindown of the launch less ss_base
  SpinHet<PM> het;

  struct Ctx {
    const float4* x[ND];
    const Term* p[ND];
    unsigned long long hn, hstep;  // fixed point: H n, and H times the step of n
    unsigned ssr;                  // spindown less ss_base
    int n0;
    double s1t;
    float4 c;
  };
  struct Raw {
    float4 x[ND];
    Term p[ND];
  };

  __device__ __forceinline__ int count() const { return N; }
  __device__ __forceinline__ Ctx begin(int batch, int n0, int step) const {
    Ctx k;
    k.n0 = n0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      k.x[d] = after_wait(xm) + (size_t)d * NP + n0;
      k.p[d] = after_wait(ph) + (size_t)d * NP + n0;
    }
    if constexpr (PM == PM_FIXED) {
      const unsigned long long H = het.H[batch];
      k.hn = mul64x32(H, (unsigned)n0);
      k.hstep = mul64x32(H, (unsigned)step);
      k.ssr = s0_flag ? 0u : (unsigned)(ss_rel + batch);
    } else if constexpr (PM == PM_F64) {
      const unsigned long long H = het.H[batch];
      k.hn = mul64x32(H, (unsigned)n0);
      k.hstep = mul64x32(H, (unsigned)step);
      k.s1t = het.s1t[batch];
    } else {
      k.c = het.c[batch];
    }
    return k;
  }
  __device__ __forceinline__ void next(Ctx& k) const {
    if constexpr (PM != PM_FF) k.hn += k.hstep;
  }
  __device__ __forceinline__ Raw fetch(const Ctx& k, int off) const {
    Raw r{};
    if constexpr (NIFO > 0) {
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        r.x[d] = __ldg(k.x[d] + off);
        r.p[d] = __ldg(k.p[d] + off);
      }
    }
    return r;
  }
  // sine and cosine of the phase of one detector
  __device__ __forceinline__ void phasor(const Ctx& k, const Term& p, int n, float* sn, float* cs) const {
    if constexpr (PM == PM_FIXED) {
      // The phase in turns, A + B ssr + H n, is formed from the high words of
      // its three terms (H n is carried from position to position).  The
      // carries of the low words that this drops lower it by at most 2 units
      // of 2^-32 turns (3e-9 rad), far below the FP32 rounding of the angle
      // that follows (up to 2^-25 of a half turn, 9e-8 rad).  The angle, in
      // [-pi, pi), goes to the hardware sine and cosine (__sincosf: absolute
      // error at most 2^-21.41 = 3.6e-7 in that range).
      const unsigned th = p.y + (__umulhi(p.z, k.ssr) + p.w * k.ssr) + (unsigned)(k.hn >> 32);
      __sincosf((float)(int)th * 1.4629180792671596e-9f, sn, cs);  // pi 2^-31
    } else if constexpr (PM == PM_F64) {
      // s1 tmp1 in turns, one FP64 operation per detector and sample (FP64
      // runs at 1/64 of the FP32 rate, and nine of them bounded pass A): the
      // fma onto 1.5 2^20 rounds the product to 2^-32 turns (1.5e-9 rad, far
      // below the FP32 rounding of the angle) and leaves it mod 1 in the low
      // word, as long as it is below 2^19 turns.  H n is exact.  Day of two
      // detectors, FP64 phases (N = 43082, 12 x 75 spindowns): 2.17 -> 1.46 ms.
      const double t1 = __hiloint2double((int)p.y, (int)p.x);
      const double q = fma(k.s1t, t1, 1572864.0);
      unsigned th = (unsigned)__double2loint(q);
      if (((unsigned)__double2hiint(q) >> 20) != 0x413u) th = far_turns(k.s1t, t1);
      th += (unsigned)(k.hn >> 32);
      sincospif((float)(int)th * 4.656612873077393e-10f, sn, cs);
    } else {
      // compensated float-float phase
      const float2 tt = make_float2(__uint_as_float(p.x), __uint_as_float(p.y));
      float p1 = k.c.x * tt.x;
      float e1 = fmaf(k.c.x, tt.x, -p1);
      e1 = fmaf(k.c.x, tt.y, e1);
      e1 = fmaf(k.c.y, tt.x, e1);
      const float nf = (float)n;
      float p2 = k.c.z * nf;
      float e2 = fmaf(k.c.z, nf, -p2);
      e2 = fmaf(k.c.w, nf, e2);
      const float s = p1 + p2;
      const float bb = s - p1;
      const float err = (p1 - (s - bb)) + (p2 - bb);
      const float e = err + e1 + e2;
      const float kk = rintf(s * kInvTwoPiF);
      float r = fmaf(-kk, kTwoPiF_A, s);
      r = fmaf(-kk, kTwoPiF_B, r);
      r = fmaf(-kk, kTwoPiF_C, r);
      r += e;
      sincosf(r, sn, cs);
    }
  }
  __device__ __forceinline__ P2 value(const Ctx& k, const Raw& r, int off) const {
    P2 v;
    const int n = k.n0 + off;
    if constexpr (NIFO > 0) {
#pragma unroll
      for (int d = 0; d < ND; ++d) add_det(k, r.x[d], r.p[d], n, d == 0, v);
    } else {
      v = pzero();
      for (int d = 0; d < nifo; ++d)
        add_det(k, __ldg(k.x[0] + (size_t)d * NP + off), __ldg(k.p[0] + (size_t)d * NP + off), n, false, v);
    }
    return v;
  }
  // v (+)= x (cos - i sin)
  __device__ __forceinline__ void add_det(const Ctx& k, const float4& x, const Term& p, int n, bool first, P2& v) const {
    float sn, cs;
    phasor(k, p, n, &sn, &cs);
    const f2 re = pk(x.x, x.y), im = pk(x.z, x.w);
    const f2 c2 = dup(cs), s2 = dup(sn), m2 = dup(-sn);
    if (first) {
      v.re = fma2(im, s2, mul2(re, c2));
      v.im = fma2(re, m2, mul2(im, c2));
    } else {
      v.re = fma2(im, s2, fma2(re, c2, v.re));
      v.im = fma2(re, m2, fma2(im, c2, v.im));
    }
  }
};

// Complex output with a scale factor (resampling FFTs).
template <typename R> struct CStore {
  typedef typename CT<R>::T T;
  static constexpr int kTraceKind = KK_FFT_FWD_B;
  T* out;   // [batch][2][ldo]
  int ldo;
  R scale;
  struct Ctx {};
  __device__ __forceinline__ Ctx begin() const { return Ctx{}; }
  __device__ __forceinline__ void put(const Ctx&, int batch, int k1, int k2, T a, T b, int logL1) const {
    const size_t k = (size_t)k1 + ((size_t)k2 << logL1);
    out[((size_t)batch * 2 + 0) * ldo + k] = mk(a.x * scale, a.y * scale);
    out[((size_t)batch * 2 + 1) * ldo + k] = mk(b.x * scale, b.y * scale);
  }
};

// F-statistic epilogue: F[k] = |Xa[k]|^2 / aa + |Xb[k]|^2 / bb, k in [nmin, nmax)
template <typename R> struct FstatStore {
  typedef typename CT<R>::T T;
  static constexpr int kTraceKind = KK_SPIN_B;
  R* F;             // [batch][bins]
  const R* inv;     // 1/aa, 1/bb in the working precision
  int nmin, nmax, bins;
  // 1/aa and 1/bb, loaded when the CTA starts (beside the first loads of
  // the intermediate) rather than where the epilogue needs them
  struct Ctx {
    R ia, ib;
  };
  __device__ __forceinline__ Ctx begin() const {
    const R* p = after_wait(inv);
    return Ctx{__ldg(&p[0]), __ldg(&p[1])};
  }
  __device__ __forceinline__ void put(const Ctx& c, int batch, int k1, int k2, T a, T b, int logL1) const {
    const int k = k1 + (k2 << logL1);
    if (k >= nmin && k < nmax)
      F[(size_t)batch * bins + (k - nmin)] = (a.x * a.x + a.y * a.y) * c.ia + (b.x * b.x + b.y * b.y) * c.ib;
  }
  __device__ __forceinline__ void put(const Ctx& c, int batch, int k1, int k2, P2 v) const {
    const int k = k1 + (k2 << 8);
    float a, b;
    upk(fma2(v.im, v.im, mul2(v.re, v.re)), a, b);
    if ((unsigned)(k - nmin) < (unsigned)bins) F[(size_t)batch * bins + (k - nmin)] = fmaf(a, (float)c.ia, b * (float)c.ib);
  }
};

// Output of the half-length interpolating transform: y[2m] = x[m] (zero
// past the N input samples), y[2m+1] = transform[m] / nfft, written as one
// 16-byte pair per (array, m) into yint [batch][2][Ninterp].
template <typename R> struct InterpStore {
  typedef typename CT<R>::T T;
  static constexpr int kTraceKind = KK_FFT_INV_B;
  T* yint;
  const T* xin;     // [batch][2][N]
  int N, Ninterp;
  R scale;          // 1/nfft
  struct Ctx {};
  __device__ __forceinline__ Ctx begin() const { return Ctx{}; }
  __device__ __forceinline__ void put(const Ctx&, int batch, int k1, int k2, T a, T b, int logL1) const {
    const int m = k1 + (k2 << logL1);
    const size_t qa = (size_t)batch * 2, qb = qa + 1;
    const T xa = m < N ? xin[qa * N + m] : mk((R)0, (R)0);
    const T xb = m < N ? xin[qb * N + m] : mk((R)0, (R)0);
    Pair<T>::st(yint + qa * Ninterp + 2 * (size_t)m, xa, mk(a.x * scale, a.y * scale));
    Pair<T>::st(yint + qb * Ninterp + 2 * (size_t)m, xb, mk(b.x * scale, b.y * scale));
  }
};

// ------------------------------------------------------------------
// Compensated two-float (float-float) arithmetic for the spline of the FP32
// forms, two values at once: a value is hi + lo with |lo| <= ulp(hi)/2 (about 48
// significant bits).  Products use fmaf for their exact error terms (Dekker), sums
// the two-sum of Knuth.
struct FF2 {
  f2 hi, lo;
};

// acc + c t, c a float-float constant (nch = -c.hi), t a float
__device__ __forceinline__ FF2 ff2_add_prod(FF2 acc, f2 ch, f2 nch, f2 cl, f2 t) {
  const f2 p = mul2(ch, t);
  const f2 ne = fma2(nch, t, p);  // minus the product's error
  const f2 s = add2(acc.hi, p);
  const f2 bb = sub2(s, acc.hi);
  const f2 e = add2(sub2(acc.hi, sub2(s, bb)), sub2(p, bb));
  return FF2{s, add2(acc.lo, fma2(cl, t, sub2(e, ne)))};
}

// ------------------------------------------------------------------
// FP32 forms: the natural spline (auxi.c:56-81) and its evaluation at x =
// interpftpad (i - shftf_i) (splint, auxi.c:83-122), then / sig2, in one
// kernel.
//
// The second derivatives solve y2_{k-1} + 4 y2_k + y2_{k+1} = 6 d_k with
// d_k = y_{k-1} - 2 y_k + y_{k+1} and y2 = 0 at both ends.  The inverse of that
// matrix on the whole line is z^|j| / (2 sqrt(3)), z = sqrt(3) - 2 = -0.268, and
// the ends are met by continuing d as an odd function about them, so
//   y2_k = sqrt(3) sum_j z^|j| d_{k+j},
// 16 terms to each side: the rest is below 0.268^17 = 2e-10 of the largest d,
// far below FP32 rounding.  The sum is compensated (coefficients and sum as two
// floats) from |j| = kSplineFull on inwards; the terms outside are below 1e-4 of
// the sum, so that their plain sum errs by 6e-12 of it.  The two sweeps of the
// elimination have 48 dependent steps of 9 dependent operations, which took
// most of this kernel's time; here every point is its own sum.
//
// A block takes kSiSamples output samples; the points that they lie between
// start at the smallest of them (base), and kSiPoints points from there hold
// them all when the shift changes slowly (it changes by 1e-4 a sample); samples
// beyond them are taken in another turn with a later base, whatever the shifts
// are.  Both arrays go through packed FP32 arithmetic.  The even points of the
// resampled series are the input itself (x), the odd ones the interpolating
// transform's results.  The shifts are formed here as k_prelude_mod forms them,
// from the ephemeris and before the wait for that kernel's results.
// What bounds it: for a short segment the latency of three dependent rounds of
// loads, for a long one instruction issue.  Three
// kernels with sweeps through global memory took 23 us on one sky point of two
// detectors (N = 10771) and 25 us of one (N = 86164), one kernel with sweeps in
// shared memory 12 and 14 us, this one 7.5 and 12 us with the shifts from an
// array, and alone 9.5 and 14 us with the shifts formed here; in the chain that
// part runs while the kernel before ends (calls of 76 and 140 us either way, 76
// and 144 with the array read after the wait).  FP64 operations are kept few there
// (one conversion for the floor, its rest for both weights): 96 x 200 spindowns
// 22.30 -> 22.25 ms.
constexpr int kSiThreads = 128, kSiSamples = 112, kSplineFull = 6;
constexpr int kSiPoints = 2 * kSiSamples + 16;           // points with y2
constexpr int kSiD = kSiPoints + 2 * kSplineTaps;        // points with d, from base - kSplineTaps on
static_assert(kSiPoints <= 2 * kSiThreads, "two points a thread");

static __global__ void __launch_bounds__(kSiThreads)
    k_resample(const float4* __restrict__ xin, const float4* __restrict__ odd, int nodd,
               const double* __restrict__ DetSSB, const __grid_constant__ SkyArgs sky,
               const DetConst* __restrict__ dc, int N, int NP, float4* __restrict__ xm,
               const __grid_constant__ SplineTab tab, const double* __restrict__ part,
               int npart, double* __restrict__ sums, float* __restrict__ sums_r) {
  CtaTrace trace_(KK_SPLINT);
  __shared__ float4 ds[kSiD], zs[kSiPoints];
  __shared__ int s_min[kSiThreads / 32];
  const int d = blockIdx.y;
  const int n = 2 * N;
  const int t = threadIdx.x;
  const int i = ((int)blockIdx.x - 1) * kSiSamples + t;
  constexpr int kNone = 0x7fffffff;
  int klo = kNone;
  bool outside = false;
  float a = 0.f, b = 0.f;
  // (the extra block has i < 0 and no samples of its own)
  if (blockIdx.x > 0 && t < kSiSamples && i < N) {
    const double shftf = time_shift(sky, DetSSB + 3 * ((size_t)d * N + i)) - sky.shft1_fma[d];
    const double x = __dmul_rn(2.0, __dsub_rn((double)i, shftf));
    // floor(x): the least int for a NaN, the nearest int for what no int holds;
    // x - floor(x) and 1 less that are exact
    const int fl = __double2int_rd(x);
    const double fr = x - (double)fl;
    outside = fl < 0 || fl > n - 1 || (fl == n - 1 && fr > 0.);
    if (!outside) {
      klo = fl;
      a = (float)(1. - fr);
      b = (float)fr;
    }
  }
  const float is2 = dc[d].inv_sig2_f;
  pdl_wait();
  pdl_go();
  if (blockIdx.x == 0) {  // an extra block, the first: aa and bb
    if (d == 0) sum_parts_f32(after_wait(part), npart, gridDim.y, dc, sums, sums_r);
    return;
  }
  if (outside) xm[(size_t)d * NP + i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4* xq = after_wait(xin) + (size_t)d * N;
  const float4* oq = after_wait(odd) + (size_t)d * nodd;
  auto point = [&](int k) { return pld((k & 1 ? oq : xq) + (k >> 1)); };
  for (;;) {
    // the first point of the samples that are left
    const int wm = __reduce_min_sync(0xffffffffu, klo);
    if ((t & 31) == 0) s_min[t >> 5] = wm;
    __syncthreads();
    int base = s_min[0];
#pragma unroll
    for (int k = 1; k < kSiThreads / 32; ++k) base = min(base, s_min[k]);
    if (base == kNone) break;
#pragma unroll
    for (int r = 0; r < (kSiD + kSiThreads - 1) / kSiThreads; ++r) {
      const int m = r * kSiThreads + t;
      const int k0 = base - kSplineTaps + m;
      // odd about both ends (more than once only for series shorter than the taps)
      int k = k0;
      bool neg = false;
      while (k < 0 || k > n - 1) {
        k = k < 0 ? -k : 2 * (n - 1) - k;
        neg = !neg;
      }
      P2 v = pzero();
      if (m < kSiD && k > 0 && k < n - 1) {
        const P2 p = point(k - 1), c = point(k), q = point(k + 1);
        // formed in FP32: its rounding is below the data's own
        const f2 m2 = dup(-2.f);
        v.re = add2(fma2(m2, c.re, p.re), q.re);
        v.im = add2(fma2(m2, c.im, p.im), q.im);
        if (neg) v = P2{sub2(0ull, v.re), sub2(0ull, v.im)};
      }
      if (m < kSiD) pst(ds + m, v);
    }
    __syncthreads();
    {
      // points t and t + kSiThreads (threads without a second one repeat it)
      const float4* d0 = ds + kSplineTaps + t;
      const float4* d1 = ds + kSplineTaps + min(t + kSiThreads, kSiPoints - 1);
      // (compact loops: the kernel runs once per sky point, and its
      // instructions come from L2 then)
      P2 f0 = pzero(), f1 = pzero();
#pragma unroll 2
      for (int j = kSplineTaps; j > kSplineFull; --j) {
        const P2 v = padd(pld(d0 + j), pld(d0 - j)), w = padd(pld(d1 + j), pld(d1 - j));
        const f2 c = dup(tab.ch[j]);
        f0 = P2{fma2(c, v.re, f0.re), fma2(c, v.im, f0.im)};
        f1 = P2{fma2(c, w.re, f1.re), fma2(c, w.im, f1.im)};
      }
      FF2 z[4] = {{f0.re, 0ull}, {f0.im, 0ull}, {f1.re, 0ull}, {f1.im, 0ull}};
#pragma unroll 1
      for (int j = kSplineFull; j >= 0; --j) {
        P2 v = pld(d0 + j), w = pld(d1 + j);
        if (j) {
          v = padd(v, pld(d0 - j));
          w = padd(w, pld(d1 - j));
        }
        const f2 ch = dup(tab.ch[j]), nch = dup(-tab.ch[j]), cl = dup(tab.cl[j]);
        z[0] = ff2_add_prod(z[0], ch, nch, cl, v.re);
        z[1] = ff2_add_prod(z[1], ch, nch, cl, v.im);
        z[2] = ff2_add_prod(z[2], ch, nch, cl, w.re);
        z[3] = ff2_add_prod(z[3], ch, nch, cl, w.im);
      }
      pst(zs + t, P2{add2(z[0].hi, z[0].lo), add2(z[1].hi, z[1].lo)});
      if (t + kSiThreads < kSiPoints)
        pst(zs + t + kSiThreads, P2{add2(z[2].hi, z[2].lo), add2(z[3].hi, z[3].lo)});
    }
    __syncthreads();
    if (klo <= base + kSiPoints - 2) {
      const int h = min(klo + 1, n - 1);
      const P2 zl = pld(zs + (klo - base)), zh = pld(zs + (h - base)), yl = point(klo), yh = point(h);
      const f2 ca = dup((a * a * a - a) / 6.f), cb = dup((b * b * b - b) / 6.f), fa = dup(a), fb = dup(b), s2 = dup(is2);
      const f2 re = add2(fma2(fa, yl.re, mul2(fb, yh.re)), fma2(ca, zl.re, mul2(cb, zh.re)));
      const f2 im = add2(fma2(fa, yl.im, mul2(fb, yh.im)), fma2(ca, zl.im, mul2(cb, zh.im)));
      pst(xm + (size_t)d * NP + i, P2{mul2(re, s2), mul2(im, s2)});
      klo = kNone;
    }
    __syncthreads();
  }
}

// FP64 form: spline() as chunked recurrences.  The forward sweep u_i =
// (-u_{i-1}/2 + 3 d_i) invp_i has |dU_i/dU_{i-1}| -> 2 - sqrt(3) = 0.268 and the
// back substitution y2_k = p_k y2_{k+1} + u_k likewise, so a chunk can start
// kSplineWarm steps early from zero: the start error shrinks by 0.268^32 =
// 5e-19.  Chunks whose warm start reaches the array ends start from the exact
// boundary values u_0 = 0, y2_{n-1} = 0.
constexpr int kSplineChunk = 64, kSplineWarm = 32;
constexpr int kSplineThreads = 256;                        // threads for staging loads/stores
constexpr int kSplineSeg = 4096;                           // elements per CTA

// Asynchronous global-to-shared copies (cp.async): every copy of a staging
// loop is in flight at once, with no registers held; an invalid element is
// zero-filled (source size 0, the source address is not read).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Shared-memory slot of staged element k: one padding element per chunk, so
// that the recurrence threads (chunk starts one chunk apart) hit different
// banks.
__host__ __device__ constexpr int spad(int k) { return k + k / kSplineChunk; }
__host__ __device__ constexpr int spad_len(int n) { return n + n / kSplineChunk + 1; }

// Forward sweep.  A CTA owns one segment of kSplineSeg elements of one
// array; it stages y[seg - warm - 1, seg_end + 1) in shared memory with
// coalesced loads, every thread runs its chunk's recurrence from shared
// memory, and the u values leave through shared memory again so the global
// stores are coalesced.
static __global__ void __launch_bounds__(kSplineThreads)
    k_spline_fwd(const double2* __restrict__ y, int ldy, double2* __restrict__ u, int n, int nseg,
                 const double* __restrict__ invp) {
  CtaTrace trace_(KK_SPLINE_FWD);
  extern __shared__ __align__(16) unsigned char sm_raw[];
  double2* us = reinterpret_cast<double2*>(sm_raw);  // spad_len(kSplineSeg)
  double2* ys = us + spad_len(kSplineSeg);           // spad_len(kSplineSeg + kSplineWarm + 2)
  const int q = blockIdx.x / nseg, sg = blockIdx.x - q * nseg;
  const double2* yq = y + (size_t)q * ldy;
  double2* uq = u + (size_t)q * n;
  const int seg0 = sg * kSplineSeg;
  const int y0 = seg0 - kSplineWarm - 1;             // first staged index
  const int ny = kSplineSeg + kSplineWarm + 2;
  // the coefficients of the first 64 steps of the array, in shared memory
  // (the first chunks' recurrences read one per step)
  __shared__ double tab[64];
  if (threadIdx.x < 64) tab[threadIdx.x] = invp[threadIdx.x];
  for (int k = threadIdx.x; k < ny; k += kSplineThreads) {
    const int i = y0 + k;
    const bool ok = i >= 0 && i < n;
    cp_async16(&ys[spad(k)], ok ? (const void*)(yq + i) : (const void*)yq, ok);
  }
  cp_async_wait_all();
  __syncthreads();
  if (threadIdx.x < (kSplineSeg / kSplineChunk)) {
    const int lo = seg0 + threadIdx.x * kSplineChunk;
    const int hi = min(lo + kSplineChunk, n - 1);
    // u_i = (-u_{i-1}/2 + 3 d_i) invp_i = al_i u_{i-1} + be_i d_i
    int i = max(1, lo - kSplineWarm);
    double2 p = ys[spad(i - 1 - y0)], cc = ys[spad(i - y0)];
    double ux = 0., uy = 0.;
    for (; i < hi; ++i) {
      const double2 nn = ys[spad(i + 1 - y0)];
      const double dx = p.x - 2. * cc.x + nn.x, dy = p.y - 2. * cc.y + nn.y;
      const int ti = i < 64 ? i : 63;
      const double al = -.5 * tab[ti], be = 3. * tab[ti];
      ux = fma(al, ux, be * dx);
      uy = fma(al, uy, be * dy);
      if (i >= lo) us[spad(i - seg0)] = make_double2(ux, uy);
      p = cc;
      cc = nn;
    }
    if (lo == 0) us[spad(0)] = make_double2(0., 0.);
  }
  __syncthreads();
  const int cnt = min(kSplineSeg, n - 1 - seg0);
  for (int k = threadIdx.x; k < cnt; k += kSplineThreads) uq[seg0 + k] = us[spad(k)];
}

// Back substitution, same staging: u[seg0, seg_end + warm) in shared memory,
// y2 of the segment written back through shared memory.
static __global__ void __launch_bounds__(kSplineThreads)
    k_spline_bwd(const double2* __restrict__ u, double2* __restrict__ y2, int n, int nseg,
                 const double* __restrict__ ptab) {
  CtaTrace trace_(KK_SPLINE_BWD);
  extern __shared__ __align__(16) unsigned char sm_raw[];
  double2* us = reinterpret_cast<double2*>(sm_raw);       // spad_len(kSplineSeg + kSplineWarm)
  double2* ys = us + spad_len(kSplineSeg + kSplineWarm);  // spad_len(kSplineSeg)
  const int q = blockIdx.x / nseg, sg = blockIdx.x - q * nseg;
  const double2* uq = u + (size_t)q * n;
  double2* yq = y2 + (size_t)q * n;
  const int seg0 = sg * kSplineSeg;
  const int nu = min(kSplineSeg + kSplineWarm, n - 1 - seg0);  // u defined on [0, n-2]
  __shared__ double tab[64];
  if (threadIdx.x < 64) tab[threadIdx.x] = ptab[threadIdx.x];
  for (int k = threadIdx.x; k < nu; k += kSplineThreads) cp_async16(&us[spad(k)], uq + seg0 + k, true);
  cp_async_wait_all();
  __syncthreads();
  const int lo = seg0 + threadIdx.x * kSplineChunk;
  const int hi = min(lo + kSplineChunk, n);
  if (threadIdx.x < (kSplineSeg / kSplineChunk) && lo < n) {
    const int kst = min(n - 2, hi - 1 + kSplineWarm);
    double vx = 0., vy = 0.;
    for (int k = kst; k >= lo; --k) {
      const double p = tab[k < 64 ? k : 63];
      const double2 uk = us[spad(k - seg0)];
      vx = p * vx + uk.x;
      vy = p * vy + uk.y;
      if (k < hi) ys[spad(k - seg0)] = make_double2(vx, vy);
    }
    if (hi == n) ys[spad(n - 1 - seg0)] = make_double2(0., 0.);
  }
  __syncthreads();
  const int cnt = min(kSplineSeg, n - seg0);
  for (int k = threadIdx.x; k < cnt; k += kSplineThreads) yq[seg0 + k] = ys[spad(k)];
}

// splint at x = interpftpad (i - shftf_i) (auxi.c:83-122), then / sig2
static __global__ void __launch_bounds__(256)
    k_splint(const double2* __restrict__ y, int ldy, const double2* __restrict__ y2,
             const double* __restrict__ shftf, const DetConst* __restrict__ dc, int N, double2* __restrict__ xm) {
  CtaTrace trace_(KK_SPLINT);
  const int d = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int n = 2 * N;
  const double x = __dmul_rn(2.0, __dsub_rn((double)i, shftf[(size_t)d * N + i]));
  const double is2 = dc[d].inv_sig2;
  for (int arr = 0; arr < 2; ++arr) {
    const size_t q = (size_t)d * 2 + arr;
    double2 v = make_double2(0., 0.);
    if (x >= 0 && x <= n - 1) {  // (false for a NaN, which as an int would be no index)
      const int klo = (int)floor(x);
      const int khi = klo + 1;
      const int kh = khi < n ? khi : n - 1;
      const double a = khi - x, b = x - klo;
      const double2 ylo = y[q * ldy + klo], yhi = y[q * ldy + kh];
      const double2 zlo = y2[q * n + klo], zhi = y2[q * n + kh];
      const double ca = (a * a * a - a), cb = (b * b * b - b);
      v.x = a * ylo.x + b * yhi.x + (ca * zlo.x + cb * zhi.x) / 6.;
      v.y = a * ylo.y + b * yhi.y + (ca * zlo.y + cb * zhi.y) / 6.;
    }
    xm[q * N + i] = make_double2(v.x * is2, v.y * is2);
  }
}

// ------------------------------------------------------------------
// FStat normalisation and thresholding

// FStat normalisation (auxi.c:214-240) and thresholding (jobcore.c:659-669)
// in one kernel.  One CTA per two 4096-bin chunks of one spindown: it loads
// the chunks, forms each block mean mu = sum/(2*4096) with a fixed reduction
// order (16 loads per thread at stride 256, xor tree per warp, warps in
// order), so a chunk's mu is bit-identical whichever CTA computes it; chunks
// beyond the last full block stay unnormalised.  When a bin is above trl,
// the normalised values go to shared memory, where runs of bins above trl
// are found; a run produces one candidate at its maximum, ties to the later
// bin.  The neighbour chunks' means are formed on demand (run starting at
// the chunk's first bin, or reaching its end), with all threads taking part.
__device__ __forceinline__ void emit_cand(DevCand* cand, int* ncand, int cap, int task, int ss, int ii,
                                          double F) {
  const int slot = atomicAdd(ncand, 1);
  if (slot < cap) {
    DevCand d;
    d.task = task;
    d.ss = ss;
    d.ii = ii;
    d.pad = 0;
    d.F = F;
    cand[slot] = d;
  }
}

template <typename R> __device__ __forceinline__ R chunk_sum(const R* f, int base, int cnt, R (*red)) {
  R v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = k * 256 + threadIdx.x;
    v[k] = i < cnt ? f[base + i] : (R)0;
  }
  R acc = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) acc += v[k];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  R sum = 0;
  for (int k = 0; k < 8; ++k) sum += red[k];
  return sum;
}

// One chunk's normalised values v (this thread's 16, at k * 256 + tid),
// loaded as in load_chunk and scaled by its 1/mu: its runs above trl, their
// candidates, and a run reaching the chunk end followed into the next
// chunks.  Called by all threads of the CTA (it has barriers).
template <typename R>
__device__ __forceinline__ void chunk_runs(const R* f, R (&v)[16], unsigned above, int c, int bins, int nblk,
                                           int white, R trl, int nmin, int ss, int task, DevCand* cand,
                                           int* ncand, int cap, R* sv, R* red) {
  const int nchunk = (bins + 4095) >> 12;
  const int base = c * 4096;
  const int cnt = min(4096, bins - base);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = k * 256 + threadIdx.x;
    if (i < cnt) sv[i + 1] = v[k];
  }
  __syncthreads();
  // value of the bin before the chunk, needed only when the chunk's first
  // bin is above the threshold
  if (c > 0 && sv[1] > trl) {
    const bool pn = !white && c - 1 < nblk;
    const R s = chunk_sum(f, base - 4096, 4096, red);
    if (threadIdx.x == 0) sv[0] = pn ? f[base - 1] * ((R)(2 * 4096) / s) : f[base - 1];
    __syncthreads();
  }
  int ii = -1;
  R Fc = 0;
  bool pend = false;  // this thread's run reaches the chunk end
  while (above) {
    const int k = __ffs(above) - 1;
    above &= above - 1;
    const int i = k * 256 + threadIdx.x;
    if (base + i != 0 && sv[i] > trl) continue;  // not the start of a run
    int iib = base + i;
    R Fcb = sv[i + 1];
    int jj = i + 1;
    for (; jj < cnt; ++jj) {
      const R w = sv[jj + 1];
      if (!(w > trl)) break;
      if (w >= Fcb) {
        iib = base + jj;
        Fcb = w;
      }
    }
    if (jj == cnt && c + 1 < nchunk) {
      ii = iib;  // continued below
      Fc = Fcb;
      pend = true;
    } else {
      emit_cand(cand, ncand, cap, task, ss, iib + nmin, Fcb);
    }
  }
  // follow a run across chunk ends; uniform loop, at most one thread active
  bool cont = pend;
  int cur = c;
  while (__syncthreads_or(cont)) {
    ++cur;
    if (cur >= nchunk) break;
    const int b2 = cur * 4096, n2 = min(4096, bins - b2);
    const bool pn = !white && cur < nblk;
    const R s = chunk_sum(f, b2, n2, red);
    if (cont) {
      const R im2 = pn ? (R)(2 * 4096) / s : (R)1;
      int j = 0;
      for (; j < n2; ++j) {
        const R w = f[b2 + j] * im2;
        if (!(w > trl)) break;
        if (w >= Fc) {
          ii = b2 + j;
          Fc = w;
        }
      }
      cont = (j == n2);
    }
  }
  if (pend) emit_cand(cand, ncand, cap, task, ss, ii + nmin, Fc);
  __syncthreads();  // sv is reused by the next chunk
}

// Two 4096-bin chunks per CTA (blockIdx.x: chunks 2x and 2x + 1 of the
// spindown blockIdx.y): both chunks' loads in flight together.
template <typename R>
__global__ void __launch_bounds__(256)
    k_normthresh(const R* __restrict__ F, int bins, int nblk, int white, R trl, int nmin, int ss0, int task,
                 DevCand* __restrict__ cand, int* __restrict__ ncand, int cap, R* __restrict__ Fdbg) {
  __shared__ R sv[4096 + 1];
  __shared__ R red[16];
  CtaTrace trace_(KK_THRESHOLD);
  const int sidx = blockIdx.y;
  const int nchunk = (bins + 4095) >> 12;
  pdl_wait();
  pdl_go();
  const R* f = after_wait(F) + (size_t)sidx * bins;
  const int cA = 2 * blockIdx.x, cB = cA + 1;
  R va[16], vb[16];
  auto load = [&](int c, R (&v)[16]) {
    const int base = c * 4096, cnt = c < nchunk ? min(4096, bins - base) : 0;
    if (cnt == 4096) {
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = f[base + k * 256 + threadIdx.x];
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const int i = k * 256 + threadIdx.x;
        v[k] = i < cnt ? f[base + i] : (R)0;
      }
    }
  };
  load(cA, va);
  load(cB, vb);
  // normalised value = F * (1/mu), mu = block sum / (2*4096); within one
  // ulp of F/mu.  The two chunks' sums in the same fixed order as one.
  R accA = 0, accB = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    accA += va[k];
    accB += vb[k];
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    accA += __shfl_xor_sync(0xffffffffu, accA, off);
    accB += __shfl_xor_sync(0xffffffffu, accB, off);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = accA;
    red[8 + (threadIdx.x >> 5)] = accB;
  }
  __syncthreads();
  R sumA = 0, sumB = 0;
  for (int k = 0; k < 8; ++k) {
    sumA += red[k];
    sumB += red[8 + k];
  }
  const R imA = (!white && cA < nblk) ? (R)(2 * 4096) / sumA : (R)1;
  const R imB = (!white && cB < nblk) ? (R)(2 * 4096) / sumB : (R)1;
  unsigned abA = 0, abB = 0;  // bit k: element k*256 + tid is above the threshold
  const int cntA = min(4096, bins - cA * 4096), cntB = cB < nchunk ? min(4096, bins - cB * 4096) : 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = k * 256 + threadIdx.x;
    va[k] *= imA;
    vb[k] *= imB;
    abA |= (i < cntA && va[k] > trl) ? (1u << k) : 0u;
    abB |= (i < cntB && vb[k] > trl) ? (1u << k) : 0u;
  }
  if (Fdbg) {
    for (int k = 0; k < 16; ++k) {
      const int i = k * 256 + threadIdx.x;
      if (i < cntA) Fdbg[(size_t)sidx * bins + cA * 4096 + i] = va[k];
      if (i < cntB) Fdbg[(size_t)sidx * bins + cB * 4096 + i] = vb[k];
    }
  }
  // no bin of either chunk above the threshold (the usual case): no run
  // starts here (a run from the previous chunk is followed by that chunk's
  // CTA)
  if (!__syncthreads_or((abA | abB) != 0u)) return;
  chunk_runs(f, va, abA, cA, bins, nblk, white, trl, nmin, ss0 + sidx, task, cand, ncand, cap, sv, red);
  if (cB < nchunk)
    chunk_runs(f, vb, abB, cB, bins, nblk, white, trl, nmin, ss0 + sidx, task, cand, ncand, cap, sv, red);
}

// ------------------------------------------------------------------
// engine

inline Geom make_geom(int L) {
  Geom g;
  int m = 0;
  while ((1 << m) < L) ++m;
  g.L = L;
  g.logL = m;
  return g;
}

template <typename R, int PM> class EngineT : public Engine {
  typedef typename CT<R>::T T;
  Buffers b_;
  Geom gf_, gm_;
  long long launches_ = 0;
  int split_ = 0;
  int dev_ = 0;  // device the engine was made on (current at construction)

  // CUDA events around a launch when profiling is on
  void pre(int kind, int items, cudaStream_t st) {
    if (!prof || !prof->on) return;
    if (prof->n == prof->cap) return;  // pool exhausted: stop recording
    Prof::Rec& r = prof->recs[prof->n];
    r.kind = kind;
    r.items = items;
    cudaEventRecord(r.a, st);
  }
  void post(cudaStream_t st) {
    if (!prof || !prof->on) return;
    if (prof->n == prof->cap) return;
    cudaEventRecord(prof->recs[prof->n].b, st);
    prof->n++;
  }

  // opt-in above 48 KB of dynamic shared memory, once per kernel instance and
  // device (the attribute is set on the current device: the engine's own,
  // made current by every entry point); `done` holds one bit per device
  template <class K> void smem_attr(K kernel, int bytes, std::atomic<unsigned long long>& done) const {
    const unsigned long long bit = 1ull << (dev_ & 63);
    if (!(done.load(std::memory_order_acquire) & bit)) {
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      done.fetch_or(bit, std::memory_order_release);
    }
  }

  // Launches a kernel that waits for the one before it in the stream by itself
  // (pdl_wait): its blocks come to the SMs while that one runs out.  Per call,
  // without and with: one short sky point 91 and 77 us, one of 2^17 163 and 144
  // us, 96 x 200 spindowns of two detectors on two lanes 25.3 and 23.9 ms, 24 x
  // 100 of three 4.45 and 4.10 ms, 6 x 400 of 2^19 14.5 and 13.8 ms.
  template <class K, class... Args>
  void launch(K kernel, dim3 grid, int threads, int smem, cudaStream_t st, const Args&... args) const {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
  }

  // FP64 form: tw: W_L1 and W_L2 tables of the default split (L1 =
  // 2^ceil(m/2)), then the two halves of the inter-pass twiddle; SPLIT 1 swaps
  // the factors and so the first two tables.
  template <int SIGN, int LOGL, int SPLIT, class Loader, class Storer>
  cudaError_t fft_l(const void* const* tw, const Loader& ld, const Storer& st, int batch, cudaStream_t stream,
                    int kind_a, int kind_b, void* ybuf) {
    typedef FftShape<R, LOGL, SPLIT> G;
    constexpr int NT = TileCfg<R>::NT;
    const T* t1 = (const T*)tw[SPLIT ? 1 : 0];
    const T* t2 = (const T*)tw[SPLIT ? 0 : 1];
    T* yb = (T*)ybuf;
    auto ka = k_pass_a<R, SIGN, LOGL, Loader, SPLIT>;
    auto kb = k_pass_b<R, SIGN, LOGL, Storer, SPLIT>;
    static std::atomic<unsigned long long> doneA{0}, doneB{0};
    smem_attr(ka, G::smem_a, doneA);
    smem_attr(kb, G::smem_b, doneB);
    dim3 ga(G::L2 >> G::LOGC, batch), gb(G::L1 >> G::LOGRR, batch);
    pre(kind_a, batch, stream);
    ka<<<ga, NT, G::smem_a, stream>>>(ld, t1, (const T*)tw[2], (const T*)tw[3], yb);
    post(stream);
    pre(kind_b, batch, stream);
    kb<<<gb, NT, G::smem_b, stream>>>(st, t2, yb);
    post(stream);
    launches_ += 2;
    return cudaGetLastError();
  }

  // FP32 forms: which = 0: length nfft, 1: nfftf; HALF: only the outputs below
  // half the length are wanted; NIN, NCHK: k_pair_a.
  template <int SIGN, int LOGL, int LTA, int LOGS, int LTB, bool HALF, int NIN, int NCHK, class Loader, class Storer>
  cudaError_t pair_l(int which, const Loader& ld, const Storer& st, int batch, cudaStream_t stream, int kind_a,
                     int kind_b, void* ybuf) {
    typedef PairShape<LOGL, LTA, LOGS> A;
    typedef PairShape<LOGL, LTB> B;
    auto ka = k_pair_a<SIGN, LOGL, LTA, LOGS, NIN, NCHK, Loader>;
    auto kb = k_pair_b<SIGN, LOGL, LTB, Storer, HALF>;
    static std::atomic<unsigned long long> doneA{0}, doneB{0};
    smem_attr(ka, A::smem_a, doneA);
    smem_attr(kb, B::smem_b, doneB);
    dim3 ga(A::L2 >> A::LOGC, (batch + (1 << LOGS) - 1) >> LOGS), gb(256 >> B::LOGRR, batch);
    pre(kind_a, batch, stream);
    launch(ka, ga, A::NT, A::smem_a, stream, ld, (const float2*)b_.pair_tw1, (const float2*)b_.pair_pass[which],
           (float4*)ybuf, batch);
    post(stream);
    pre(kind_b, batch, stream);
    launch(kb, gb, B::NB, B::smem_b, stream, st, (const float2*)b_.pair_row[which], (const float4*)ybuf);
    post(stream);
    launches_ += 2;
    return cudaGetLastError();
  }

  // Dispatch on the transform length (2^12 .. 2^20) to the compile-time
  // geometry of the passes; FP64 form: with SPLITS, odd lengths may take the
  // swapped split (split = 1).
  template <int SIGN, bool SPLITS = false, class Loader, class Storer>
  cudaError_t fft(const Geom& g, const void* const* tw, const Loader& ld, const Storer& st, int batch,
                  cudaStream_t stream, int kind_a, int kind_b, void* ybuf, int split = 0) {
    switch (g.logL) {
#define PA_FFT_CASE(M)                                                                              \
  case M:                                                                                           \
    if (SPLITS && (M & 1) && split)                                                                 \
      return fft_l<SIGN, M, SPLITS && (M & 1)>(tw, ld, st, batch, stream, kind_a, kind_b, ybuf);    \
    return fft_l<SIGN, M, 0>(tw, ld, st, batch, stream, kind_a, kind_b, ybuf);
      PA_FFT_CASE(12) PA_FFT_CASE(13) PA_FFT_CASE(14) PA_FFT_CASE(15) PA_FFT_CASE(16)
      PA_FFT_CASE(17) PA_FFT_CASE(18) PA_FFT_CASE(19) PA_FFT_CASE(20)
#undef PA_FFT_CASE
      default: return cudaErrorInvalidValue;
    }
  }

  // The resampling transforms (length nfft, at most 2^19) take half-size
  // tiles: one or a few detectors give few CTAs, and they are waited for.
  template <int SIGN, int NCHK, class Loader, class Storer>
  cudaError_t pair_pre(const Loader& ld, const Storer& st, int batch, cudaStream_t stream, int kind_a, int kind_b) {
    switch (gf_.logL) {
#define PA_FFT_CASE(M) \
  case M: return pair_l<SIGN, M, 11, 0, 11, false, 16, NCHK>(0, ld, st, batch, stream, kind_a, kind_b, b_.ybuf_pre);
      PA_FFT_CASE(12) PA_FFT_CASE(13) PA_FFT_CASE(14) PA_FFT_CASE(15) PA_FFT_CASE(16)
      PA_FFT_CASE(17) PA_FFT_CASE(18) PA_FFT_CASE(19)
#undef PA_FFT_CASE
      default: return cudaErrorInvalidValue;
    }
  }

  // The spindown transform.  F is wanted on [nmin, nmax): below half the
  // length in every search set up as the reference's (settings.c:50-55).
  // The data fill more than half of the transform with fftpad = 1, and a
  // quarter to a half of it with 2: pass A takes the 16 rows (of 16 x 16) in
  // quarters, the last one of them with a condition, the empty ones left out.
  // That is compiled for the fixed-point form of one to three detectors from
  // 2^16 on; the others test every row.
  template <int M, class Loader>
  cudaError_t pair_main_l(const Loader& ld, const FstatStore<R>& st, int batch, cudaStream_t stream, void* yb) {
    constexpr int A = KK_SPIN_A, B = KK_SPIN_B;
    constexpr int LTA = 11, kLogS = 1, LTB = M >= 18 ? 12 : 11;
    if (b_.nmax > b_.nfftf / 2) return pair_l<-1, M, LTA, kLogS, LTB, false, 16, 0>(1, ld, st, batch, stream, A, B, yb);
    if constexpr (PM == PM_FIXED && M >= 16 && Loader::kQuarters) {
      const int q = b_.nfftf / 4;
      if (b_.N > 3 * q) return pair_l<-1, M, LTA, kLogS, LTB, true, 16, 12>(1, ld, st, batch, stream, A, B, yb);
      if (b_.N > 2 * q) return pair_l<-1, M, LTA, kLogS, LTB, true, 12, 8>(1, ld, st, batch, stream, A, B, yb);
      if (b_.N > q) return pair_l<-1, M, LTA, kLogS, LTB, true, 8, 4>(1, ld, st, batch, stream, A, B, yb);
    }
    return pair_l<-1, M, LTA, kLogS, LTB, true, 16, 0>(1, ld, st, batch, stream, A, B, yb);
  }
  template <class Loader>
  cudaError_t pair_main(const Loader& ld, const FstatStore<R>& st, int batch, cudaStream_t stream, void* ybuf) {
    switch (gm_.logL) {
#define PA_FFT_CASE(M) \
  case M: return pair_main_l<M>(ld, st, batch, stream, ybuf);
      PA_FFT_CASE(12) PA_FFT_CASE(13) PA_FFT_CASE(14) PA_FFT_CASE(15) PA_FFT_CASE(16)
      PA_FFT_CASE(17) PA_FFT_CASE(18) PA_FFT_CASE(19) PA_FFT_CASE(20)
#undef PA_FFT_CASE
      default: return cudaErrorInvalidValue;
    }
  }
  template <int NIFO>
  cudaError_t spin_main(const SkyArgs& sky, int slot, int ss0, int nb, int s0_flag, const FstatStore<R>& fs,
                        cudaStream_t st, void* yb) {
    SpinLoader<PM, NIFO> sl;
    sl.xm = (const float4*)b_.xm[slot];
    sl.ph = (const typename SpinTerm<PM>::T*)((const float4*)b_.xm[slot] + (size_t)b_.nifo * b_.NP);
    sl.N = b_.N;
    sl.NP = b_.NP;
    sl.nifo = b_.nifo;
    sl.ss_rel = ss0 - sky.ss_base;
    sl.s0_flag = s0_flag;
    for (int k = 0; k < nb; ++k) spin_het_fill(sl.het, k, ss0 + k, sky, s0_flag);
    return pair_main(sl, fs, nb, st, yb);
  }

 public:
  explicit EngineT(const Buffers& b) : b_(b) {
    cudaGetDevice(&dev_);
    gf_ = make_geom(b.nfft);
    gm_ = make_geom(b.nfftf);
  }

  long long launches() const override { return launches_; }
  size_t real_size() const override { return sizeof(R); }
  void set_split(int split) override { split_ = (gm_.logL & 1) ? split : 0; }
#ifdef PA_CTA_TRACE
  cudaError_t set_trace(void* buf, unsigned int cap) override {
    CtaTraceRec* p = static_cast<CtaTraceRec*>(buf);
    const unsigned int zero = 0, c = buf ? cap : 0u;
    cudaError_t e = cudaMemcpyToSymbol(c_trace_buf, &p, sizeof(p));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_trace_cap, &c, sizeof(c));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_trace_n, &zero, sizeof(zero));
    return e;
  }
  cudaError_t trace_count(unsigned int* n) override { return cudaMemcpyFromSymbol(n, g_trace_n, sizeof(*n)); }
#else
  cudaError_t set_trace(void*, unsigned int) override { return cudaErrorNotSupported; }
  cudaError_t trace_count(unsigned int*) override { return cudaErrorNotSupported; }
#endif
  int split() const override { return split_; }

  cudaError_t prelude(const SkyArgs& sky, int slot, cudaStream_t st) override {
    const int N = b_.N, nifo = b_.nifo;
    constexpr int NT = mod_threads<R>();
    const int nbx = (N + NT - 1) / NT;
    pre(KK_PRELUDE_MOD, nifo, st);
    launch(k_prelude_mod<R, PM>, dim3(nbx, nifo), NT, 0, st,
        b_.xDat, b_.DetSSB, (const R*)b_.cosmodf, (const R*)b_.sinmodf, b_.dc, sky, N, b_.NP, (T*)b_.xin,
        b_.shftf, sizeof(R) == 8 ? b_.ph0[slot] : (void*)((float4*)b_.xm[slot] + (size_t)nifo * b_.NP), b_.part, b_.sums[slot],
        (R*)b_.sums_r[slot], b_.counter);
    post(st);
    launches_ += 1;
    // forward FFT of the zero-padded series (length nfft), then spectrum remap
    // + backward FFT of length Ninterp, scale interpftpad/Ninterp
    // (jobcore.c:338-362), as a half-length transform (HalfShiftLoader), and the
    // spline through the first 2N points of each resampled array
    cudaError_t e;
    if constexpr (sizeof(R) == 4) {
      const PairLoader pl{(const float4*)b_.xin, N};
      const PairStore<KK_FFT_FWD_B> sp{(float4*)b_.spec, b_.nfft, 1.f};
      e = pair_pre<-1, 0>(pl, sp, nifo, st, KK_FFT_FWD_A, KK_FFT_FWD_B);
      if (e != cudaSuccess) return e;
      const HalfShiftPair hl{(const float4*)b_.spec, (const float2*)b_.tw_inv[2], (const float2*)b_.tw_inv[3], b_.nfft,
                             b_.nfft / 2 + 1};
      const PairStore<KK_FFT_INV_B> is{(float4*)b_.yint, b_.nfft, (float)(1.0 / b_.nfft)};
      e = pair_pre<+1, 16>(hl, is, nifo, st, KK_FFT_INV_A, KK_FFT_INV_B);
      if (e != cudaSuccess) return e;
      pre(KK_SPLINT, nifo, st);
      launch(k_resample, dim3((N + kSiSamples - 1) / kSiSamples + 1, nifo), kSiThreads, 0, st,
          (const float4*)b_.xin, (const float4*)b_.yint, b_.nfft, b_.DetSSB, sky, b_.dc, N, b_.NP,
          (float4*)b_.xm[slot], b_.spl, b_.part, nbx, b_.sums[slot], (float*)b_.sums_r[slot]);
      post(st);
      launches_ += 1;
    } else {
      PlainLoader<R> pl{(const T*)b_.xin, N, N};
      CStore<R> cs1{(T*)b_.spec, b_.nfft, (R)1};
      e = fft<-1>(gf_, b_.tw_fwd, pl, cs1, nifo, st, KK_FFT_FWD_A, KK_FFT_FWD_B, b_.ybuf_pre);
      if (e != cudaSuccess) return e;
      HalfShiftLoader<R> hl{(const T*)b_.spec, (const T*)b_.tw_inv[2], (const T*)b_.tw_inv[3], b_.nfft,
                            b_.nfft / 2 + 1};
      InterpStore<R> is{(T*)b_.yint, (const T*)b_.xin, N, b_.Ninterp, (R)(1.0 / b_.nfft)};
      e = fft<+1>(gf_, b_.tw_invh, hl, is, nifo, st, KK_FFT_INV_A, KK_FFT_INV_B, b_.ybuf_pre);
      if (e != cudaSuccess) return e;
      const int n = 2 * N;
      const int nseg = (n + kSplineSeg - 1) / kSplineSeg;
      constexpr int smf = (spad_len(kSplineSeg) + spad_len(kSplineSeg + kSplineWarm + 2)) * (int)sizeof(double2);
      constexpr int smb = (spad_len(kSplineSeg) + spad_len(kSplineSeg + kSplineWarm)) * (int)sizeof(double2);
      static std::atomic<unsigned long long> donef{0}, doneb{0};
      smem_attr(k_spline_fwd, smf, donef);
      smem_attr(k_spline_bwd, smb, doneb);
      pre(KK_SPLINE_FWD, nifo, st);
      k_spline_fwd<<<nseg * 2 * nifo, kSplineThreads, smf, st>>>((const double2*)b_.yint, b_.Ninterp,
                                                                 (double2*)b_.u, n, nseg, b_.spline_invp);
      post(st);
      pre(KK_SPLINE_BWD, nifo, st);
      k_spline_bwd<<<nseg * 2 * nifo, kSplineThreads, smb, st>>>((const double2*)b_.u, (double2*)b_.y2, n, nseg,
                                                                 b_.spline_p);
      post(st);
      pre(KK_SPLINT, nifo, st);
      k_splint<<<dim3((N + 255) / 256, nifo), 256, 0, st>>>((const double2*)b_.yint, b_.Ninterp,
                                                            (const double2*)b_.y2, b_.shftf, b_.dc, N,
                                                            (double2*)b_.xm[slot]);
      post(st);
      launches_ += 3;
    }
    return cudaGetLastError();
  }

  cudaError_t spindowns(const SkyArgs& sky, int slot, int lane, int ss0, int nb, double trl, int white,
                        int s0_flag, cudaStream_t st, void* Fdbg) override {
    const size_t lo = (size_t)lane * b_.lane_sb;  // first spindown of the lane in ybuf and F
    T* const yb = (T*)b_.ybuf + lo * 2 * b_.nfftf;
    R* const Fl = (R*)b_.F + lo * b_.bins;
    if (nb > kSpinBatchMax) return cudaErrorInvalidValue;
    FstatStore<R> fs{Fl, (const R*)b_.sums_r[slot], b_.nmin, b_.nmax, b_.bins};
    cudaError_t e;
    if constexpr (sizeof(R) == 4) {
      switch (b_.nifo) {
        case 1: e = spin_main<1>(sky, slot, ss0, nb, s0_flag, fs, st, yb); break;
        case 2: e = spin_main<2>(sky, slot, ss0, nb, s0_flag, fs, st, yb); break;
        case 3: e = spin_main<3>(sky, slot, ss0, nb, s0_flag, fs, st, yb); break;
        default: e = spin_main<0>(sky, slot, ss0, nb, s0_flag, fs, st, yb);
      }
    } else {
      SpinLoader64 sl;
      sl.xm = (const double2*)b_.xm[slot];
      sl.tmp1 = (const double*)b_.ph0[slot];
      sl.N = b_.N;
      sl.nifo = b_.nifo;
      for (int k = 0; k < nb; ++k) spin_het_fill(sl.het, k, ss0 + k, sky, s0_flag);
      e = fft<-1, true>(gm_, b_.tw_main, sl, fs, nb, st, KK_SPIN_A, KK_SPIN_B, yb, split_);
    }
    if (e != cudaSuccess) return e;
    const int nchunk = (b_.bins + 4095) / 4096;
    pre(KK_THRESHOLD, nb, st);
    launch(k_normthresh<R>, dim3((nchunk + 1) / 2, nb), 256, 0, st, Fl, b_.bins, b_.nblk, white, (R)trl,
           b_.nmin, ss0, sky.task, b_.cand, b_.ncand, b_.cand_cap, (R*)Fdbg);
    post(st);
    launches_ += 1;
    return cudaGetLastError();
  }
};

}  // namespace pa
