// pa_pair.cuh -- the FFT passes of the FP32 forms, for sm_103a.
//
// Every transform of this code runs on a pair of arrays (a, b) that share
// the loader's phase and all twiddles.  The passes hold one complex element
// of both arrays as two packed registers, re = (a.re, b.re) and im = (a.im,
// b.im), and compute with the packed FP32 instructions (add, mul, fma
// .f32x2): one issue slot for the same operation on a and b.  They run at
// half the rate of the scalar ones, so the FP32 pipe does the same work per
// element, but the passes were held by instruction issue and L1, not by that
// pipe; broadcast, negation and swap of a packed operand cost nothing.  Each
// half rounds as the scalar operation does.
//
// A length-L transform (L = 256 L2, 2^12 <= L <= 2^20) is two passes of the
// four-step scheme, n = L2 n1 + n2, k = k1 + 256 k2:
//   pass A: per column n2, Y[k1, n2] = W_L^{n2 k1} sum_n1 x[L2 n1 + n2] W_256^{n1 k1}
//   pass B: per row k1,    X[k1 + 256 k2] = sum_n2 Y[k1, n2] W_L2^{n2 k2}
// A CTA transforms a tile of T = 2^LOGT pairs with T/16 threads, 16 pairs a
// thread (64 registers of data at 128 a thread; pass B at 2^17 32 pairs a thread):
//   pass A: T/256 columns as 16 x 16, one exchange through shared memory;
//   pass B: T/L2 rows in two or three stages of radix 8, 16 or 32.
// 128 registers at half the warps hold the same data as 64 registers did at
// twice the warps, and leave room for the loads of the next positions.
//
// What bounds the spindown transform (2^17, two detectors, GB300): pass A reads
// 6.4 MB from L2 and writes 2 MB to it per spindown (0.32 us at the 20 TB/s and
// 0.24 us at the 8.5 TB/s that L2 was measured to give), pass B reads 2 MB and
// writes 0.25 MB, and neither overlaps these with its arithmetic completely.
// Launches of 32 spindowns, us per spindown: pass A 0.96 with tiles of 4096
// pairs, 0.84 with 2048 (four CTAs of 128 threads per SM: their phases
// interleave finer), 0.755 with two spindowns in a CTA (0.775 with four), which
// halves the record reads; pass B 0.64 with tiles of 4096, 0.58 with 2048 (at
// 2^18 and above a row of the smaller tile's F has too few bins side by side,
// and 4096 is the better one).  Against passes of 16-byte record halves and
// scalar arithmetic: 2^17 with two detectors 30.3 -> 25.4 ms for 96 x 200
// spindowns, three detectors 5.69 -> 4.79 ms (24 x 100), 2^19 19.2 -> 14.8 ms
// (6 x 400).
//
// The intermediate is stored in blocks of 2^lr rows, Y[k1 >> lr][n2][k1 mod
// 2^lr] (pair_row_block: as many rows as a pass-B tile has, at most 8), so
// that a warp of pass A stores 256 or 512 contiguous bytes and a pass-B tile
// is a few contiguous blocks, whatever the length.  The table of the
// inter-pass twiddles has the same order.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pa_engine.h"
#include "pa_f32x2.cuh"
#include "pa_fft.cuh"

namespace pa {

// Programmatic dependent launch: the blocks of a kernel may come to the SMs
// when all blocks of the one before it in the stream have called pdl_go, and
// wait in pdl_wait until it has finished and its results are visible.  Every
// block calls both, go after wait, so that whatever came before the kernel
// before has finished too.  Before the wait a kernel reads only what no kernel
// writes (tables and inputs) and writes nothing.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A pointer whose loads stay behind the wait, also those of read-only data
// that the compiler may otherwise move freely.
template <class T> __device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p));
  return p;
}

// One complex element of the arrays a and b.
struct P2 {
  f2 re, im;
};
__device__ __forceinline__ P2 pzero() { return P2{0ull, 0ull}; }
__device__ __forceinline__ P2 padd(P2 a, P2 b) { return P2{add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ P2 psub(P2 a, P2 b) { return P2{sub2(a.re, b.re), sub2(a.im, b.im)}; }
// x * (wr + i wi), the same factor for both arrays
__device__ __forceinline__ P2 pmul(P2 x, float wr, float wi) {
  return P2{fma2(x.im, dup(-wi), mul2(x.re, dup(wr))), fma2(x.im, dup(wr), mul2(x.re, dup(wi)))};
}
__device__ __forceinline__ P2 pmul(P2 x, float2 w) { return pmul(x, w.x, w.y); }
__device__ __forceinline__ P2 pld(const float4* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return P2{v.x, v.y};
}
__device__ __forceinline__ void pst(float4* p, P2 v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.re, v.im);
}
// the last read of global data: evict-first
__device__ __forceinline__ P2 pldlast(const float4* p) {
  const float4 v = __ldcs(p);
  return P2{pk(v.x, v.y), pk(v.z, v.w)};
}

// a, b, c, d <- the 4-point DFT in natural order
template <int SIGN> __device__ __forceinline__ void pdft4(P2& a, P2& b, P2& c, P2& d) {
  const P2 s = padd(a, c), t = psub(a, c), u = padd(b, d), w = psub(b, d);
  a = padd(s, u);
  c = psub(s, u);
  const P2 p = {sub2(t.re, w.im), add2(t.im, w.re)};  // t + i w
  const P2 m = {add2(t.re, w.im), sub2(t.im, w.re)};  // t - i w
  b = SIGN > 0 ? p : m;
  d = SIGN > 0 ? m : p;
}

// x * exp(SIGN 2 pi i e / 16), e = 1, 3 or 9
template <int SIGN, int e> __device__ __forceinline__ P2 pw16(P2 x) {
  constexpr float c = e == 1 ? 0.92387953251128675613f : (e == 3 ? 0.38268343236508977173f : -0.92387953251128675613f);
  constexpr float s = e == 1 ? 0.38268343236508977173f : (e == 3 ? 0.92387953251128675613f : -0.38268343236508977173f);
  return pmul(x, c, SIGN * s);
}
constexpr float kSqrtHalf = 0.70710678118654752440f;
// sqrt(2) x exp(SIGN 2 pi i / 8): the factor sqrt(1/2) goes into the fma that
// uses the value
template <int SIGN> __device__ __forceinline__ P2 pw8(P2 x) {
  return SIGN > 0 ? P2{sub2(x.re, x.im), add2(x.re, x.im)} : P2{add2(x.re, x.im), sub2(x.im, x.re)};
}
// a + h x and a - h x, h = sqrt(1/2)
__device__ __forceinline__ P2 phadd(P2 a, P2 x) {
  return P2{fma2(x.re, dup(kSqrtHalf), a.re), fma2(x.im, dup(kSqrtHalf), a.im)};
}
__device__ __forceinline__ P2 phsub(P2 a, P2 x) {
  return P2{fma2(x.re, dup(-kSqrtHalf), a.re), fma2(x.im, dup(-kSqrtHalf), a.im)};
}

// 8-point DFT in natural order: X[q] = E[q mod 4] +- W8^q O[q mod 4]
template <int SIGN> __device__ __forceinline__ void pdft8(P2* v) {
  P2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  pdft4<SIGN>(e0, e1, e2, e3);
  pdft4<SIGN>(o0, o1, o2, o3);
  v[0] = padd(e0, o0);
  v[4] = psub(e0, o0);
  const P2 t1 = pw8<SIGN>(o1);
  v[1] = phadd(e1, t1);
  v[5] = phsub(e1, t1);
  const P2 p = {sub2(e2.re, o2.im), add2(e2.im, o2.re)}, m = {add2(e2.re, o2.im), sub2(e2.im, o2.re)};
  v[2] = SIGN > 0 ? p : m;
  v[6] = SIGN > 0 ? m : p;
  // (SIGN i - 1)/sqrt2 o3, with the signs folded into the sums
  const f2 s = add2(o3.re, o3.im), d = sub2(o3.re, o3.im);
  const f2 h = dup(kSqrtHalf), nh = dup(-kSqrtHalf);
  if (SIGN > 0) {  // (-s, d)
    v[3] = P2{fma2(s, nh, e3.re), fma2(d, h, e3.im)};
    v[7] = P2{fma2(s, h, e3.re), fma2(d, nh, e3.im)};
  } else {  // (-d, -s)
    v[3] = P2{fma2(d, nh, e3.re), fma2(s, nh, e3.im)};
    v[7] = P2{fma2(d, h, e3.re), fma2(s, h, e3.im)};
  }
}

// second layer of the 16-point DFT: v[n2 + 4 k1] holds the inner transform
// (n2, k1); X[k1 + 4 k2] = sum_n2 W4^{n2 k2} W16^{n2 k1} v
template <int SIGN> __device__ __forceinline__ void pdft16_tail(P2* v) {
  P2 o[16];
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    P2 a = v[4 * k1], b = v[4 * k1 + 1], c = v[4 * k1 + 2], d = v[4 * k1 + 3];
    if (k1 == 1) {
      b = pw16<SIGN, 1>(b);
      const P2 t = pw8<SIGN>(c);
      d = pw16<SIGN, 3>(d);
      const P2 s = phadd(a, t), m = phsub(a, t), u = padd(b, d), w = psub(b, d);
      a = padd(s, u);
      c = psub(s, u);
      const P2 p = {sub2(m.re, w.im), add2(m.im, w.re)}, q = {add2(m.re, w.im), sub2(m.im, w.re)};
      b = SIGN > 0 ? p : q;
      d = SIGN > 0 ? q : p;
    } else if (k1 == 2) {
      // c W16^4 = SIGN i c; b W16^2 and d W16^6 share the factor sqrt(1/2)
      const P2 p = {sub2(a.re, c.im), add2(a.im, c.re)}, q = {add2(a.re, c.im), sub2(a.im, c.re)};
      const P2 s = SIGN > 0 ? p : q, m = SIGN > 0 ? q : p;
      const P2 bt = pw8<SIGN>(b);
      const f2 ds = add2(d.re, d.im), dd = sub2(d.re, d.im);
      // dt = sqrt(2) d W8^3: (-ds, dd) or (-dd, -ds)
      P2 u, w;
      if (SIGN > 0) {
        u = P2{sub2(bt.re, ds), add2(bt.im, dd)};
        w = P2{add2(bt.re, ds), sub2(bt.im, dd)};
      } else {
        u = P2{sub2(bt.re, dd), sub2(bt.im, ds)};
        w = P2{add2(bt.re, dd), add2(bt.im, ds)};
      }
      const f2 h = dup(kSqrtHalf), nh = dup(-kSqrtHalf);
      a = phadd(s, u);
      c = phsub(s, u);
      const P2 x = {fma2(w.im, nh, m.re), fma2(w.re, h, m.im)}, y = {fma2(w.im, h, m.re), fma2(w.re, nh, m.im)};
      b = SIGN > 0 ? x : y;
      d = SIGN > 0 ? y : x;
    } else if (k1 == 3) {
      b = pw16<SIGN, 3>(b);
      const f2 cs = add2(c.re, c.im), cd = sub2(c.re, c.im);
      d = pw16<SIGN, 9>(d);
      const f2 h = dup(kSqrtHalf), nh = dup(-kSqrtHalf);
      P2 s, m;  // a +- c W16^6
      if (SIGN > 0) {
        s = P2{fma2(cs, nh, a.re), fma2(cd, h, a.im)};
        m = P2{fma2(cs, h, a.re), fma2(cd, nh, a.im)};
      } else {
        s = P2{fma2(cd, nh, a.re), fma2(cs, nh, a.im)};
        m = P2{fma2(cd, h, a.re), fma2(cs, h, a.im)};
      }
      const P2 u = padd(b, d), w = psub(b, d);
      a = padd(s, u);
      c = psub(s, u);
      const P2 p = {sub2(m.re, w.im), add2(m.im, w.re)}, q = {add2(m.re, w.im), sub2(m.im, w.re)};
      b = SIGN > 0 ? p : q;
      d = SIGN > 0 ? q : p;
    } else {
      pdft4<SIGN>(a, b, c, d);
    }
    o[k1] = a;
    o[k1 + 4] = b;
    o[k1 + 8] = c;
    o[k1 + 12] = d;
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = o[k];
}

// 16-point DFT in natural order of v[0 .. NIN), zeros from there on (NIN: 8,
// 12 or 16)
template <int SIGN, int NIN = 16> __device__ __forceinline__ void pdft16(P2* v) {
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    if (NIN == 16) {
      pdft4<SIGN>(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    } else {
      const P2 a = v[n2], b = v[4 + n2];
      P2 s = a, t = a;
      if (NIN == 12) {
        s = padd(a, v[8 + n2]);
        t = psub(a, v[8 + n2]);
      }
      v[n2] = padd(s, b);
      v[8 + n2] = psub(s, b);
      const P2 p = {sub2(t.re, b.im), add2(t.im, b.re)}, m = {add2(t.re, b.im), sub2(t.im, b.re)};
      v[4 + n2] = SIGN > 0 ? p : m;
      v[12 + n2] = SIGN > 0 ? m : p;
    }
  }
  pdft16_tail<SIGN>(v);
}

// 32-point DFT in natural order, the first 16 results only with HALF: X[k] =
// E[k] + W32^k O[k], X[k + 16] = E[k] - W32^k O[k]
template <int SIGN, bool HALF> __device__ __forceinline__ void pdft32(P2* v) {
  constexpr float c[9] = {1.f, 0.98078528040323044913f, 0.92387953251128675613f, 0.83146961230254523708f,
                          kSqrtHalf, 0.55557023301960222474f, 0.38268343236508977173f, 0.19509032201612826785f, 0.f};
  P2 e[16], o[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  }
  pdft16<SIGN>(e);
  pdft16<SIGN>(o);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (k == 0) {
      v[0] = padd(e[0], o[0]);
      if (!HALF) v[16] = psub(e[0], o[0]);
    } else if (k == 8) {
      const P2 p = {sub2(e[8].re, o[8].im), add2(e[8].im, o[8].re)}, m = {add2(e[8].re, o[8].im), sub2(e[8].im, o[8].re)};
      v[8] = SIGN > 0 ? p : m;
      if (!HALF) v[24] = SIGN > 0 ? m : p;
    } else {
      const float wr = k < 8 ? c[k] : -c[16 - k], wi = SIGN * (k < 8 ? c[8 - k] : c[k - 8]);
      v[k] = P2{fma2(o[k].im, dup(-wi), fma2(o[k].re, dup(wr), e[k].re)),
                fma2(o[k].im, dup(wr), fma2(o[k].re, dup(wi), e[k].im))};
      if (!HALF)
        v[k + 16] = P2{fma2(o[k].im, dup(wi), fma2(o[k].re, dup(-wr), e[k].re)),
                       fma2(o[k].im, dup(-wr), fma2(o[k].re, dup(-wi), e[k].im))};
    }
  }
}

template <int SIGN, int R, bool HALF = false> __device__ __forceinline__ void pdft(P2* v) {
  static_assert(R == 1 || R == 4 || R == 8 || R == 16 || R == 32, "radix");
  if constexpr (R == 32) pdft32<SIGN, HALF>(v);
  if (R == 4) pdft4<SIGN>(v[0], v[1], v[2], v[3]);
  if (R == 8) pdft8<SIGN>(v);
  if (R == 16) pdft16<SIGN>(v);
}

// Geometry of the two passes of a length 2^LOGL transform with tiles of
// 2^LOGT pairs.
template <int LOGL, int LOGT, int LOGS = 0> struct PairShape {
  static constexpr int LOGL2 = LOGL - 8, L2 = 1 << LOGL2;
  static constexpr int T = 1 << LOGT, NT = T / 16;
  static constexpr int LOGQ = LOGT - 8, Q = 1 << LOGQ;            // pass A: column transforms of a tile,
  static constexpr int LOGC = LOGQ - LOGS, C = 1 << LOGC;         // C columns of 2^LOGS batch items
  static constexpr int LOGRR = LOGT > LOGL2 ? LOGT - LOGL2 : 0, RR = 1 << LOGRR;  // pass B: rows of a tile
  static constexpr int LR = pair_row_block(LOGL);                 // rows of a block of the intermediate
  // pass A tile: element (c, b, q) at c * ZC + b * Q + q, q = item * C +
  // column.  A quarter of a warp of stage 2 reads 2^LR values of c at 8 / 2^LR
  // values of q; the pad puts them into eight different 16-byte bank groups.
  static constexpr int ZC = 16 * Q + (LR == 0 ? 0 : (8 >> LR));
  static constexpr int smem_a = 16 * ZC * 16 + 272 * 8;
  // pass B: radices of the stages (first, middle, last); R2 = 1: two stages
  static constexpr int R1 = pair_radix(LOGL, 0), R2 = pair_radix(LOGL, 1), R3 = pair_radix(LOGL, 2);
  // pass B tile: element e of row rr at e * RR + (e / R1) * PAD + rr.  The
  // first stage stores R1 elements apart from lane to lane; with fewer than
  // 8 rows the pad after every R1 elements keeps that conflict-free.
  // threads of pass B: 16 pairs each, 32 with a radix-32 stage.  512-element
  // rows (2^17) as 16 x 32 exchange through shared memory once, as 8 x 8 x 8
  // twice, and shared memory is what pass B uses most: 48 x 200 spindowns of
  // two detectors 11.97 -> 11.25 ms, 64 of one 146 -> 138 us.  Five CTAs of 64
  // threads per SM, at 168 registers (six, with the pad given up for a swizzle:
  // 12.1 ms).  1024-element rows as 32 x 32 gained nothing.
  static constexpr int EB = R3 == 32 ? 32 : 16, NB = T / EB;
  static constexpr int LOGR1 = R1 == 16 ? 4 : (R1 == 8 ? 3 : (R1 == 4 ? 2 : 1));
  static constexpr int PAD = RR < 8 ? RR : 0;
  static constexpr int TW = pair_row_table(LOGL);                 // entries of the row twiddle table
  // CTAs of pass B per SM (three of 256 threads, at 80 registers, spill)
  static constexpr int MINB = EB == 32 ? 320 / NB : 512 / NB;
  static constexpr int smem_b = (L2 * RR + (L2 / R1) * PAD) * 16 + TW * 8;
  static_assert(LOGL >= 12 && LOGL <= 20 && LOGT >= 11 && LOGT <= 12, "no such tile");
  static_assert(LOGC >= 0 && C <= L2 && RR <= 256, "transform too short for the tile");
};

// a load that stays where it is written (before a barrier, say)
__device__ __forceinline__ float2 ldg_here(const float2* p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// Pass A.  The 16 x 16 column transforms: thread (b, col) of stage 1 loads the
// rows n1 = 16 a + b of column col, transforms over a and stores (c, b, col);
// thread (c, col) of stage 2 multiplies by W_256^{b c}, transforms over b,
// multiplies by the inter-pass twiddle and stores Y[k1 = c + 16 d].
// Loader: count() positions hold data; fetch(ctx, off) starts the loads of
// position n0 + off, value(ctx, raw, off) forms its value, next(ctx) goes on
// by one step; the loads run kAhead positions ahead, under a condition for
// the whole warp (rows past the data cost nothing).  NIN: rows a >= NIN hold
// no data; the condition is left out for a < NCHK, which do.
// A CTA takes the same columns of 2^LOGS batch items: their threads lie in one
// warp, so that each load of the loader's data serves all of them.
template <int SIGN, int LOGL, int LOGT, int LOGS, int NIN, int NCHK, class Loader>
__global__ void __launch_bounds__(PairShape<LOGL, LOGT, LOGS>::NT, 512 / PairShape<LOGL, LOGT, LOGS>::NT)
    k_pair_a(const __grid_constant__ Loader ld, const float2* __restrict__ tw1, const float2* __restrict__ twp,
             float4* __restrict__ ybuf, int nbatch) {
  typedef PairShape<LOGL, LOGT, LOGS> G;
  CtaTrace trace_(Loader::kTraceKind);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* z = reinterpret_cast<float4*>(smem_raw);
  float2* tws = reinterpret_cast<float2*>(z + 16 * G::ZC);  // W_256^{b c} at c * 17 + b
  const int t = threadIdx.x;
  const int batch0 = blockIdx.y << LOGS, c0 = blockIdx.x << G::LOGC;
  constexpr int RB = 1 << G::LR;
  // stage 2's transform and c, and the place of (k1 = c + 16 d, n2) in the
  // intermediate and in the twiddle table, for d = 0
  const int q2 = (t >> G::LR) & (G::Q - 1);
  const int c2 = (t & (RB - 1)) + ((t >> (G::LR + G::LOGQ)) << G::LR);
  const unsigned o2 =
      ((unsigned)((c2 >> G::LR) << G::LOGL2) + c0 + (q2 & (G::C - 1))) * RB + (c2 & (RB - 1));
  constexpr unsigned dstep = 16u << G::LOGL2;  // 16 rows on
  {
    const int q = t & (G::Q - 1), b = t >> G::LOGQ;
    const int n0 = (b << G::LOGL2) + c0 + (q & (G::C - 1));
    // the smallest position of the warp at a = 0
    const int nw = ((t >> 5 << 5 >> G::LOGQ) << G::LOGL2) + c0;
    constexpr int step = 16 << G::LOGL2;
    constexpr int PF = Loader::template Ahead<NIN, NCHK>::v;
    pdl_wait();
    pdl_go();
    // (items past the last one repeat it; they are not stored)
    typename Loader::Ctx ctx = ld.begin(min(batch0 + (q >> G::LOGC), nbatch - 1), n0, step);
    const int left = ld.count() - nw;
    typename Loader::Raw raw[PF + 1];
#pragma unroll
    for (int a = 0; a < PF; ++a)
      if (a < NCHK || a * step < left) raw[a] = ld.fetch(ctx, a * step);
    P2 v[16];
#pragma unroll
    for (int a = 0; a < NIN; ++a) {
      if (a + PF < NIN && (a + PF < NCHK || (a + PF) * step < left))
        raw[(a + PF) % (PF + 1)] = ld.fetch(ctx, (a + PF) * step);
      if (a < NCHK || a * step < left) v[a] = ld.value(ctx, raw[a % (PF + 1)], a * step);
      else v[a] = pzero();
      ld.next(ctx);
    }
    pdft16<SIGN, NIN>(v);
#pragma unroll
    for (int c = 0; c < 16; ++c) pst(z + c * G::ZC + b * G::Q + q, v[c]);
  }
  // the inter-pass twiddles exp(-2 pi i n2 k1 / L): in flight over the barrier
  // and stage 2's transform, when the registers of stage 1 are free
  float2 w[16];
#pragma unroll
  for (int d = 0; d < 16; ++d) w[d] = ldg_here(twp + (o2 + d * dstep));
#pragma unroll
  for (int k = 0; k <= 272 / G::NT; ++k) {
    const int q = t + k * G::NT;
    if (q < 272) {
      float2 e = __ldg(&tw1[(q / 17) * (q % 17) & 255]);
      if (SIGN > 0) e.y = -e.y;  // the tables hold exp(-2 pi i ...)
      tws[q] = e;
    }
  }
  __syncthreads();
  P2 v[16];
#pragma unroll
  for (int b = 0; b < 16; ++b) {
    v[b] = pld(z + c2 * G::ZC + b * G::Q + q2);
    if (b > 0) v[b] = pmul(v[b], tws[c2 * 17 + b]);
  }
  pdft16<SIGN>(v);
  const int batch = batch0 + (q2 >> G::LOGC);
  if (LOGS > 0 && batch >= nbatch) return;
  float4* yb = ybuf + ((size_t)batch << LOGL) + o2;
#pragma unroll
  for (int d = 0; d < 16; ++d) pst(yb + d * dstep, pmul(v[d], w[d].x, SIGN > 0 ? -w[d].y : w[d].y));
}

// One stage of the row transforms: R-point butterflies with the results of
// Ns-point ones (Stockham); thread t takes the butterflies (j, rr) = t, t + NT,
// ...  In: from `src(e, rr)`; out: `dst(e, rr, value)`.  FIRST: no twiddles.
template <int SIGN, int R, int LOGNS, class G, bool HALF = false, class Src>
__device__ __forceinline__ void pair_stage_load(const Src& src, const float2* tw, int q, int& j, int& rr, P2 (&v)[R]) {
  constexpr int J = G::L2 / R;  // butterflies of a row
  rr = q & (G::RR - 1);
  j = q >> G::LOGRR;
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = src(j + r * J, rr);
  if (LOGNS > 0) {
    constexpr int Ns = 1 << LOGNS;
    const int k = j & (Ns - 1);
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const float2 w = tw[r * Ns + k];
      v[r] = pmul(v[r], w.x, SIGN > 0 ? -w.y : w.y);
    }
  }
  pdft<SIGN, R, HALF>(v);
}

// Pass B.  Storer: Ctx begin() and put(ctx, batch, k1, k2, value); HALF: only
// the outputs below L/2 are wanted, so the last stage forms half of its
// outputs.
template <int SIGN, int LOGL, int LOGT, class Storer, bool HALF>
__global__ void __launch_bounds__(PairShape<LOGL, LOGT>::NB, PairShape<LOGL, LOGT>::MINB)
    k_pair_b(const Storer st, const float2* __restrict__ tw2, const float4* __restrict__ ybuf) {
  typedef PairShape<LOGL, LOGT> G;
  static_assert(LOGT >= G::LOGL2, "a row is longer than the tile");
  CtaTrace trace_(Storer::kTraceKind);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* s = reinterpret_cast<float4*>(smem_raw);
  float2* tws = reinterpret_cast<float2*>(s + G::L2 * G::RR + (G::L2 / G::R1) * G::PAD);
  const int t = threadIdx.x;
  // batches in reverse launch order: pass A wrote the last batch items last,
  // so their intermediate is the likeliest to be still in L2
  const int batch = gridDim.y - 1 - blockIdx.y;
  const int k10 = blockIdx.x << G::LOGRR;
  // the row twiddles, in flight over the wait; stored after the first stage
  constexpr int NTW = G::R2 == 1 && G::R3 == 1 ? 1 : (G::TW + G::NB - 1) / G::NB;
  float2 twv[NTW];
#pragma unroll
  for (int k = 0; k < NTW; ++k)
    if (t + k * G::NB < G::TW) twv[k] = ldg_here(&tw2[t + k * G::NB]);
  pdl_wait();
  pdl_go();
  const typename Storer::Ctx sctx = st.begin();
  const float4* yb = after_wait(ybuf) + ((size_t)batch << LOGL);
  auto at = [](int e, int rr) { return e * G::RR + (e >> G::LOGR1) * G::PAD + rr; };
  auto from_smem = [&](int e, int rr) { return pld(s + at(e, rr)); };
  // the intermediate is read once, here: evict-first
  auto from_y = [&](int n2, int rr) {
    const int k1 = k10 + rr;
    return pldlast(yb + (((((k1 >> G::LR) << G::LOGL2) + n2) << G::LR) + (k1 & ((1 << G::LR) - 1))));
  };
  constexpr int L1r = G::LOGR1;
  if constexpr (G::R2 == 1 && G::R3 == 1) {
    // rows of 16: a single stage
    P2 v[16];
    int j, rr;
    pair_stage_load<SIGN, 16, 0, G>(from_y, tws, t, j, rr, v);
#pragma unroll
    for (int r = 0; r < (HALF ? 8 : 16); ++r) st.put(sctx, batch, k10 + rr, j + r * (G::L2 / 16), v[r]);
  } else {
    // first stage
    constexpr int R = G::R1, PT = G::EB / R;
    P2 v[PT][R];
    int j[PT], rr[PT];
#pragma unroll
    for (int p = 0; p < PT; ++p) pair_stage_load<SIGN, R, 0, G>(from_y, tws, t + p * G::NB, j[p], rr[p], v[p]);
#pragma unroll
    for (int p = 0; p < PT; ++p)
#pragma unroll
      for (int r = 0; r < R; ++r) pst(s + at(j[p] * R + r, rr[p]), v[p][r]);
#pragma unroll
    for (int k = 0; k < NTW; ++k)
      if (t + k * G::NB < G::TW) tws[t + k * G::NB] = twv[k];
    __syncthreads();
  }
  if constexpr (G::R2 > 1) {
    constexpr int R = G::R2, PT = G::EB / R, Ns = 1 << L1r;
    P2 v[PT][R];
    int j[PT], rr[PT];
#pragma unroll
    for (int p = 0; p < PT; ++p) pair_stage_load<SIGN, R, L1r, G>(from_smem, tws, t + p * G::NB, j[p], rr[p], v[p]);
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PT; ++p) {
      const int d = ((j[p] >> L1r) * R << L1r) + (j[p] & (Ns - 1));
#pragma unroll
      for (int r = 0; r < R; ++r) pst(s + at(d + r * Ns, rr[p]), v[p][r]);
    }
    __syncthreads();
  }
  if constexpr (G::R3 > 1) {
    constexpr int R = G::R3, PT = G::EB / R;
    constexpr int LOGNS = G::LOGL2 - (R == 32 ? 5 : (R == 16 ? 4 : (R == 8 ? 3 : (R == 4 ? 2 : 1)))), Ns = 1 << LOGNS;
    const float2* tw = tws + (G::R2 > 1 ? G::R1 * G::R2 : 0);
#pragma unroll
    for (int p = 0; p < PT; ++p) {
      P2 v[R];
      int j, rr;
      pair_stage_load<SIGN, R, LOGNS, G, HALF>(from_smem, tw, t + p * G::NB, j, rr, v);
#pragma unroll
      for (int r = 0; r < (HALF ? R / 2 : R); ++r) st.put(sctx, batch, k10 + rr, j + r * Ns, v[r]);
    }
  }
}

}  // namespace pa
