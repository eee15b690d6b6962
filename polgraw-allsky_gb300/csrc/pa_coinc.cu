// pa_coinc.cu -- coincidences among the trigger files of several frames on
// the device: read_trigger_files() of coincidences/src/coincidences.c:117-600
// (cells, per-frame duplicate removal, coincidence count, records), plus the
// host-side transformation matrix of manage_grid_matrix (init.c:1142-1210).
//
// Data flow (one stream; arrays in HBM):
//   records [raw][5] f64 (uploaded per frame)
//   k_cells      band/frame-shift/SNR cuts and the 4 integer cells of each
//                record (those of the FP64 evaluation without contraction, in
//                the reference's expression order), per-block counts,
//                per-column min/max
//   scan + k_inband   ordered compaction of the kept records (read order,
//                frame by frame), with a cell key: the 4 cells as unsigned
//                offsets from the column maxima (descending cells sort
//                ascending), packed to the bits their range needs
//   radix sort   LSD, 8-bit digits, stable: the order of the reference's two
//                qsort()s at once (cells descending; equal cells keep frame
//                then read order, which is what qsort's merge sort leaves)
//   frame ranks  per-tile frame histograms + scan locate, for every frame,
//                its last sorted record and the record of an earlier frame
//                that the reference compares it with (the row left over at
//                that position of its candidate table)
//   k_dedup      runs of equal (cells, frame): the reference's highest-SNR
//                state machine per run (coincidences.c:317-413)
//   compaction   survivors in (cells desc, frame) order = the reference's
//                sorted allcandi
//   k_groups     runs of equal cells among survivors: multiplicity, stored
//                or not (coincidences.c:449-486)
//   radix pass   coincidences by multiplicity, descending, stable
//   k_means      FP64 means in the reference's member order (last to first)
//
// No kernel waits on another kernel or on a flag; every index is bounds
// checked against the sizes passed in.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <string>
#include <vector>

#include "../../include/polgraw_gb300.h"
#include "pa_trace.h"

namespace {

constexpr int kMaxFrames = 255;
constexpr int kT = 256;                 // threads per block everywhere
constexpr int kIt = 8;                  // items per thread (tiles of 2048)
constexpr int kTile = kT * kIt;
constexpr int kRTile = 4096;            // radix tile (items per block)

// The frames of one run.  The kernels take it by value (4 KB of parameters), so
// that every launch keeps the table of its own handle and run: handles run on
// streams of their own, and a table in a device symbol would be one for all.
struct FrameTab {
  int nframes;
  int frame_no[kMaxFrames];
  unsigned raw_start[kMaxFrames + 1];    // first raw record of each frame (below 2^31 in all)
  int blk_start[kMaxFrames + 1];         // first k_cells block of each frame
  unsigned in_start[kMaxFrames + 1];     // first in-band record of each frame
};

struct CellArgs {
  long long lo_k, hi_k;    // narrowdown band (pi/2 -+ narrowdown) and SNR cut as
  long long cut_k;         // order keys (order_key)
  double N, sqrN, omsN;    // coincidences.c:187-188
  double N2;               // 2 N
  double se, ce;           // sin/cos(C_EPSMA)
  double v[4][4];          // vedva / scale (coincidences.c:182-184)
  double half_shift[4];    // 0.5 shift[j]
  int refr;
  // sky terms in FP32: the columns' factors of be0 and be1 and, per column, the
  // bound on |cell value (FP64) - cell value (FP32 sky terms)|
  float se_f, ce_f, s2_f[4], s3_f[4], margin[4];
  // float-float (hi + lo) factors of the frequency and the spindown
  float f_h[4], f_l[4], d_h[4], d_l[4], hs_f[4];
  int fast;                // N < 2^24: the FP32/float-float path is on
};

// a number as the sum of two floats (about 48 significant bits)
struct FF {
  float h, l;
};
// d = h + l with h = (float)d and l = (float)(d - h), both by integer
// arithmetic on d's bits: a conversion or an FP64 subtraction takes the FP64
// pipe, which has 1/64 of the FP32 rate.  Numbers whose parts are not all
// normal floats (2^-74 <= |d| < 2^127 is enough) take the conversions.
// (a call, so that the conversions are not issued for every number)
__device__ __noinline__ FF ff_convert(double d) {
  const float h = (float)d;
  return {h, (float)(d - (double)h)};
}
constexpr long long kMag = 0x7fffffffffffffffll;
__device__ __forceinline__ FF ff_of(double d) {
  const long long b = __double_as_longlong(d), m = b & kMag;
  const int e = (int)(m >> 52);
  if (e < 949 || e > 1149) {
    if (m == 0) return {0.f, 0.f};  // (no spindown: common)
    return ff_convert(d);
  }
  // h: to nearest even at bit 29, then the exponent's new bias (mod 2^32)
  const long long r = (m + 0x0fffffff + ((m >> 29) & 1)) >> 29;
  const unsigned sign = (unsigned)((unsigned long long)b >> 32) & 0x80000000u;
  // the rest, an integer below 2^29 in units of the last place
  const int rest = (int)(m - (r << 29));
  const float l = (float)rest * __int_as_float((e - 1075 + 127) << 23);
  return {__uint_as_float(((unsigned)r - (896u << 23)) | sign), __uint_as_float(__float_as_uint(l) ^ sign)};
}
// Order key of a double: x < y <=> key(x) < key(y) for numbers that are not
// NaN, with -0 just below +0; positive NaNs lie above +inf, negative ones
// below -inf.  (An FP64 comparison takes the FP64 pipe too.)
__host__ __device__ __forceinline__ long long order_key(long long bits) { return bits ^ ((bits >> 63) & kMag); }
constexpr long long kInfBits = 0x7ff0000000000000ll;
constexpr long long kPiBits = 0x400921fb54442d18ll;  // M_PI

struct KeyLayout {
  int maxc[4];             // column maxima
  int shift[4];            // bit position of each column's field
  int bits;                // total key bits
};

__device__ __forceinline__ int frame_of_block(const FrameTab& ft, int b) {
  int lo = 0, hi = ft.nframes;  // blk_start[lo] <= b < blk_start[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (ft.blk_start[mid] <= b) lo = mid; else hi = mid;
  }
  return lo;
}

// frame of in-band record v: the last frame whose first in-band record is
// <= v (empty frames share their successor's start); s_in = in_start in
// shared memory
__device__ __forceinline__ int frame_of_in(unsigned v, const unsigned* s_in, int nf) {
  int lo = 0, hi = nf;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s_in[mid] <= v) lo = mid; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void load_in_start(const FrameTab& ft, unsigned* s_in) {
  for (int k = threadIdx.x; k <= ft.nframes; k += blockDim.x) s_in[k] = ft.in_start[k];
  __syncthreads();
}

// coincidences.c:229-270 for one record in FP64, the reference's expression
// order without contraction; the cells of the kept record in *cl
__device__ __noinline__ void cells_f64(double c0s, double c1, double c2, double c3, const CellArgs& a, int4* cl) {
  double t[4];
  t[0] = __dmul_rn(c0s, a.N);
  t[1] = __dmul_rn(c1, a.sqrN);
  double sa, ca, sd, cd;
  sincos(c3, &sa, &ca);
  sincos(c2, &sd, &cd);
  const double be0 = __dadd_rn(__dmul_rn(__dmul_rn(a.ce, sa), cd), __dmul_rn(a.se, sd));
  const double be1 = __dmul_rn(ca, cd);
  t[2] = __dmul_rn(a.omsN, be0);
  t[3] = __dmul_rn(a.omsN, be1);
  int c[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    double s = __dmul_rn(t[0], a.v[0][j]);
    s = __dadd_rn(s, __dmul_rn(t[1], a.v[1][j]));
    s = __dadd_rn(s, __dmul_rn(t[2], a.v[2][j]));
    s = __dadd_rn(s, __dmul_rn(t[3], a.v[3][j]));
    s = __dadd_rn(s, a.half_shift[j]);
    c[j] = (int)round(s);
  }
  *cl = make_int4(c[0], c[1], c[2], c[3]);
}

// Returns 0 when the record is not kept, 1 with its cells, 2 when it is kept
// and its cells have to be formed in FP64.
// GB300 runs FP64 at 1/64 of the FP32
// rate, so only the three operations of the frequency shift run in FP64 (2 c1 N
// = c1 (2 N): the doubling is exact); the band and SNR tests compare order
// keys, and the cell values are first formed with the frequency and spindown
// terms from float-float products (error-free by fmaf; each product and the sky
// term give their nearest integer away at once, so that the fractions add up in
// plain FP32) and the sky terms (two sincos, be0/be1 of ast2lin,
// auxi.c:34-35) in FP32.  Each column's value then lies within a.margin[j] +
// 1e-11 of the products' magnitude of the FP64 value.  (Products: what the two
// floats of each factor leave, 2 x 2^-48, the product of the low parts, 2^-48,
// and the roundings of the correction, 2^-46: below 2^-45 = 2.8e-14, as are the
// FP64 evaluation's own roundings.  FP32 sincosf: 2 units in the last place,
// 1.2e-7; the argument's rest in float is added by the derivative.  be0: 2.32 x
// 1.2e-7 + 2e-7 for its roundings, and 3e-7 relative for its FP32 factors:
// 0.8e-6; the margin allows 2e-6.)  When every column's
// fractional part is farther than that from 1/2, both round to the same
// integer; otherwise (or for terms >= 2^22, or |delta|, |alpha| > 8) the record
// is formed in FP64.  The cells are therefore those of the FP64 evaluation.
__device__ __forceinline__ int cell_of(double c0, double c1, double c2, double c3, double c4, double fshift,
                                       const CellArgs& a, int4* cl) {
  const long long k0 = order_key(__double_as_longlong(c0)), k4 = order_key(__double_as_longlong(c4));
  if (!(k0 > a.lo_k && k0 < a.hi_k && k4 > a.cut_k && k4 <= kInfBits)) return 0;
  const double c0s = __dadd_rn(c0, __dmul_rn(__dmul_rn(c1, a.N2), fshift));
  const long long ks = __double_as_longlong(c0s);
  if (!(ks > 0 && ks < kPiBits)) return 0;
  const FF x3 = ff_of(c3), x2 = ff_of(c2);
  if (!a.fast || !(fabsf(x3.h) <= 8.f && fabsf(x2.h) <= 8.f)) return 2;
  const FF u = ff_of(c0s), d = ff_of(c1);
  float sa, ca, sd, cd;
  sincosf(x3.h, &sa, &ca);
  sincosf(x2.h, &sd, &cd);
  const float sa1 = fmaf(ca, x3.l, sa), ca1 = fmaf(-sa, x3.l, ca);
  const float sd1 = fmaf(cd, x2.l, sd), cd1 = fmaf(-sd, x2.l, cd);
  const float be0 = fmaf(a.ce_f * sa1, cd1, a.se_f * sd1);
  const float be1 = ca1 * cd1;
  // x - (nearest integer), |x| < 2^22, by adding and subtracting 1.5 x 2^23
  auto nearest = [](float x) { return (x + 12582912.f) - 12582912.f; };
  bool ok = true;
  int c[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float p = u.h * a.f_h[j], q = d.h * a.d_h[j];
    const float pe = fmaf(u.h, a.f_l[j], fmaf(u.l, a.f_h[j], fmaf(u.h, a.f_h[j], -p)));
    const float qe = fmaf(d.h, a.d_l[j], fmaf(d.l, a.d_h[j], fmaf(d.h, a.d_h[j], -q)));
    const float w = fmaf(be0, a.s2_f[j], be1 * a.s3_f[j]);
    const float pi = nearest(p), qi = nearest(q), wi = nearest(w);
    const float fr = (((p - pi) + (q - qi)) + (w - wi)) + ((pe + qe) + a.hs_f[j]);
    const float ri = nearest(fr);
    const float terms = fabsf(p) + fabsf(q);
    // (false for a NaN, too)
    ok = ok && terms + fabsf(w) < 4194304.f && 0.5f - fabsf(fr - ri) > fmaf(terms, 1e-11f, a.margin[j]);
    c[j] = (int)((pi + qi) + (wi + ri));
  }
  *cl = make_int4(c[0], c[1], c[2], c[3]);
  return ok ? 1 : 2;
}

__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  unsigned t = 0;
  for (int k = 0; k < kT / 32; k++) t += sh[k];
  return t;
}

// In-tile positions of the set flags among flag[t0 .. min(t0 + kTile, end)), in
// order, into list[]; returns their number (also to threads that write none).
// One pass over the tile and two barriers: warp w takes the 256 flags from
// 256 w on, 32 at a time.
__device__ __forceinline__ unsigned tile_list(const uint8_t* __restrict__ flag, long long t0, long long end,
                                              unsigned short* list, unsigned* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int first = w * (kTile / (kT / 32));
  constexpr int kRows = kTile / kT;
  uint8_t fl[kRows];
#pragma unroll
  for (int k = 0; k < kRows; k++) {
    const long long i = t0 + first + 32 * k + lane;
    fl[k] = i < end ? flag[i] : (uint8_t)0;
  }
  unsigned bal[kRows], n = 0;
#pragma unroll
  for (int k = 0; k < kRows; k++) {
    bal[k] = __ballot_sync(0xffffffffu, fl[k]);
    n += __popc(bal[k]);
  }
  if (lane == 0) sh[w] = n;
  __syncthreads();
  unsigned before = 0, tot = 0;
#pragma unroll
  for (int k = 0; k < kT / 32; k++) {
    const unsigned c = sh[k];
    if (k < w) before += c;
    tot += c;
  }
#pragma unroll
  for (int k = 0; k < kRows; k++) {
    if (fl[k]) list[before + __popc(bal[k] & ((1u << lane) - 1u))] = (unsigned short)(first + 32 * k + lane);
    before += __popc(bal[k]);
  }
  __syncthreads();
  return tot;
}

// ---- cells of every raw record ------------------------------------------

// A record that needs the FP64 cells would hold its whole warp for the FP64
// sincos; a block puts them on a list instead and forms them at the end, full
// warps at a time.  24 x 2^18 records: 424 us with FP64 comparisons and
// conversions and the FP64 cells in place (the FP64 pipe 80 % busy), 119 us now
// (252 MB in and 107 MB out: 53 us at the copy rate; the rest is instruction
// issue, two sincosf a record).
__global__ void __launch_bounds__(kT) k_cells(const __grid_constant__ FrameTab ft, const double* __restrict__ rec,
                                              const __grid_constant__ CellArgs a,
                                              int4* __restrict__ cells_raw, uint8_t* __restrict__ flag,
                                              unsigned* __restrict__ blk_cnt, int* __restrict__ minmax,
                                              unsigned* __restrict__ nexact, double* __restrict__ snr_raw) {
  __shared__ unsigned sh[kT / 32];
  __shared__ int smm[8];
  __shared__ unsigned short list[kTile];
  __shared__ unsigned nlist;
  const int b = blockIdx.x;
  const int f = frame_of_block(ft, b);
  const long long fend = ft.raw_start[f + 1];
  const long long tile0 = (long long)ft.raw_start[f] + (long long)(b - ft.blk_start[f]) * kTile;
  const double fshift = (double)(a.refr - ft.frame_no[f]);
  if (threadIdx.x == 0) nlist = 0;
  if (threadIdx.x < 4) smm[threadIdx.x] = INT_MAX;
  else if (threadIdx.x < 8) smm[threadIdx.x] = INT_MIN;
  __syncthreads();
  unsigned cnt = 0;
  int mn[4] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX}, mx[4] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN};
  auto extend = [&](int4 cl) {
    mn[0] = min(mn[0], cl.x); mx[0] = max(mx[0], cl.x);
    mn[1] = min(mn[1], cl.y); mx[1] = max(mx[1], cl.y);
    mn[2] = min(mn[2], cl.z); mx[2] = max(mx[2], cl.z);
    mn[3] = min(mn[3], cl.w); mx[3] = max(mx[3], cl.w);
  };
  // the record of the next round is loaded before this round's arithmetic
  double nx[5] = {0, 0, 0, 0, 0};
  auto load = [&](long long r) {
    if (r < fend)
#pragma unroll
      for (int k = 0; k < 5; k++) nx[k] = __ldg(rec + 5 * r + k);
  };
  load(tile0 + threadIdx.x);
#pragma unroll 1
  for (int it = 0; it < kIt; it++) {
    const long long r = tile0 + (long long)it * kT + threadIdx.x;
    if (r >= fend) break;
    const double c0 = nx[0], c1 = nx[1], c2 = nx[2], c3 = nx[3], c4 = nx[4];
    if (it + 1 < kIt) load(r + kT);
    int4 cl = make_int4(0, 0, 0, 0);
    const int ok = cell_of(c0, c1, c2, c3, c4, fshift, a, &cl);
    flag[r] = ok != 0;
    snr_raw[r] = c4;
    cnt += ok != 0;
    if (ok == 2) {
      list[atomicAdd(&nlist, 1u)] = (unsigned short)(it * kT + threadIdx.x);
    } else {
      cells_raw[r] = cl;
      if (ok) extend(cl);
    }
  }
  __syncthreads();
  const unsigned nl = nlist;
  for (unsigned q = threadIdx.x; q < nl; q += kT) {
    const long long r = tile0 + list[q];
    const double c0 = rec[5 * r], c1 = rec[5 * r + 1];
    int4 cl;
    cells_f64(__dadd_rn(c0, __dmul_rn(__dmul_rn(c1, a.N2), fshift)), c1, rec[5 * r + 2], rec[5 * r + 3], a, &cl);
    cells_raw[r] = cl;
    extend(cl);
  }
  if (threadIdx.x == 0 && nl) atomicAdd(nexact, nl);
  const unsigned tot = block_sum(cnt, sh);
  if (threadIdx.x == 0) blk_cnt[b] = tot;
  if (mx[0] >= mn[0]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      atomicMin(&smm[j], mn[j]);
      atomicMax(&smm[4 + j], mx[j]);
    }
  }
  __syncthreads();
  if (tot && threadIdx.x < 4) {
    atomicMin(&minmax[threadIdx.x], smm[threadIdx.x]);
    atomicMax(&minmax[4 + threadIdx.x], smm[4 + threadIdx.x]);
  }
}

template <typename K>
__device__ __forceinline__ K make_key(int4 c, const KeyLayout& L);

template <>
__device__ __forceinline__ unsigned long long make_key<unsigned long long>(int4 c, const KeyLayout& L) {
  const int cc[4] = {c.x, c.y, c.z, c.w};
  unsigned long long k = 0;
#pragma unroll
  for (int j = 0; j < 4; j++)
    k |= (unsigned long long)(unsigned)(L.maxc[j] - cc[j]) << L.shift[j];
  return k;
}

struct U128 {
  unsigned long long lo, hi;
};
__device__ __forceinline__ bool operator==(const U128& a, const U128& b) { return a.lo == b.lo && a.hi == b.hi; }

template <>
__device__ __forceinline__ U128 make_key<U128>(int4 c, const KeyLayout& L) {
  // one 32-bit field per column: (maxc - c) < 2^32 always
  U128 k;
  k.hi = ((unsigned long long)(unsigned)(L.maxc[0] - c.x) << 32) | (unsigned)(L.maxc[1] - c.y);
  k.lo = ((unsigned long long)(unsigned)(L.maxc[2] - c.z) << 32) | (unsigned)(L.maxc[3] - c.w);
  return k;
}

__device__ __forceinline__ unsigned digit_of(unsigned long long k, int shift) { return (unsigned)(k >> shift) & 255u; }
__device__ __forceinline__ unsigned digit_of(const U128& k, int shift) {
  return shift < 64 ? (unsigned)(k.lo >> shift) & 255u : (unsigned)(k.hi >> (shift - 64)) & 255u;
}
__device__ __forceinline__ bool key_is(unsigned long long k, unsigned long long lo, unsigned long long hi) {
  return k == lo && hi == 0;
}
__device__ __forceinline__ bool key_is(const U128& k, unsigned long long lo, unsigned long long hi) {
  return k.lo == lo && k.hi == hi;
}
__device__ __forceinline__ void key_split(unsigned long long k, unsigned long long* lo, unsigned long long* hi) {
  *lo = k;
  *hi = 0;
}
__device__ __forceinline__ void key_split(const U128& k, unsigned long long* lo, unsigned long long* hi) {
  *lo = k.lo;
  *hi = k.hi;
}

// ordered compaction of the kept records, with their keys
template <typename K>
__global__ void __launch_bounds__(kT) k_inband(const __grid_constant__ FrameTab ft, const uint8_t* __restrict__ flag,
                                               const int4* __restrict__ cells_raw,
                                               const unsigned* __restrict__ blk_off, KeyLayout L,
                                               unsigned* __restrict__ rawidx, int4* __restrict__ cells_in,
                                               K* __restrict__ key, unsigned* __restrict__ val,
                                               const double* __restrict__ snr_raw, double* __restrict__ snr_in) {
  __shared__ unsigned sh[kT / 32];
  __shared__ unsigned short list[kTile];
  const int b = blockIdx.x;
  const int f = frame_of_block(ft, b);
  const long long tile0 = (long long)ft.raw_start[f] + (long long)(b - ft.blk_start[f]) * kTile;
  const unsigned base = blk_off[b];
  const unsigned tot = tile_list(flag, tile0, ft.raw_start[f + 1], list, sh);
  for (unsigned q = threadIdx.x; q < tot; q += kT) {
    const long long r = tile0 + list[q];
    const unsigned o = base + q;
    const int4 cl = cells_raw[r];
    rawidx[o] = (unsigned)r;
    cells_in[o] = cl;
    key[o] = make_key<K>(cl, L);
    val[o] = o;
    snr_in[o] = snr_raw[r];
  }
}

// ---- scan (exclusive, in place) ------------------------------------------

// One block scans up to kScanOne elements: the tile counts of a few million
// records are a few thousand, where three launches took 12 us and one takes 4
// (a round of 8192 elements takes about 2.5 us, so four rounds at most).
constexpr int kST = 1024;
constexpr long long kScanOne = 4 * kST * kIt;
__global__ void __launch_bounds__(kST) k_scan_one(unsigned* __restrict__ d, int n) {
  __shared__ unsigned sh[kST / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned carry = 0;
  for (int r = 0; r < n; r += kST * kIt) {
    const int t0 = r + threadIdx.x * kIt;
    unsigned v[kIt], s = 0;
#pragma unroll
    for (int k = 0; k < kIt; k++) {
      v[k] = (t0 + k < n) ? d[t0 + k] : 0u;
      s += v[k];
    }
    unsigned x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    unsigned z = sh[lane];  // inclusive scan of the warp sums, in every warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, z, o);
      if (lane >= o) z += y;
    }
    const unsigned before = w ? __shfl_sync(0xffffffffu, z, w ? w - 1 : 0) : 0u;
    const unsigned all = __shfl_sync(0xffffffffu, z, 31);
    unsigned run = carry + before + x - s;
#pragma unroll
    for (int k = 0; k < kIt; k++) {
      if (t0 + k < n) d[t0 + k] = run;
      run += v[k];
    }
    carry += all;
    __syncthreads();
  }
}

// Exclusive scan of every row d[r * n .. r * n + n) in place, one block per
// row; the row's sum to total[r].
__global__ void __launch_bounds__(kT) k_scan_rows(unsigned* __restrict__ d, int n, unsigned* __restrict__ total) {
  __shared__ unsigned sh[kT / 32];
  unsigned* row = d + (long long)blockIdx.x * n;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned carry = 0;
  for (long long r = 0; r < n; r += kTile) {
    const long long t0 = r + threadIdx.x * kIt;
    unsigned v[kIt], s = 0;
#pragma unroll
    for (int k = 0; k < kIt; k++) {
      v[k] = (t0 + k < n) ? row[t0 + k] : 0u;
      s += v[k];
    }
    unsigned x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kT / 32; k++) {
      const unsigned c = sh[k];
      if (k < w) before += c;
      all += c;
    }
    unsigned run = carry + before + x - s;
#pragma unroll
    for (int k = 0; k < kIt; k++) {
      if (t0 + k < n) row[t0 + k] = run;
      run += v[k];
    }
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(kT) k_scan_tiles(unsigned* __restrict__ d, long long n, unsigned* __restrict__ sums) {
  __shared__ unsigned sh[kT];
  const long long t0 = (long long)blockIdx.x * kTile + (long long)threadIdx.x * kIt;
  unsigned v[kIt], s = 0;
#pragma unroll
  for (int k = 0; k < kIt; k++) {
    v[k] = (t0 + k < n) ? d[t0 + k] : 0u;
    s += v[k];
  }
  // block exclusive scan of the thread sums
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned acc = 0;
    for (int k = 0; k < kT / 32; k++) {
      const unsigned c = sh[k];
      sh[k] = acc;
      acc += c;
    }
    sh[kT / 32] = acc;
  }
  __syncthreads();
  unsigned run = sh[w] + x - s;
  if (threadIdx.x == kT - 1 && sums) sums[blockIdx.x] = sh[kT / 32];
#pragma unroll
  for (int k = 0; k < kIt; k++) {
    if (t0 + k < n) d[t0 + k] = run;
    run += v[k];
  }
}

__global__ void __launch_bounds__(kT) k_scan_add(unsigned* __restrict__ d, long long n, const unsigned* __restrict__ sums) {
  const unsigned add = sums[blockIdx.x];
  const long long t0 = (long long)blockIdx.x * kTile;
  for (int k = threadIdx.x; k < kTile; k += kT)
    if (t0 + k < n) d[t0 + k] += add;
}

// ---- radix sort (LSD, 8-bit digits, stable) ------------------------------

constexpr int kRItems = kRTile / kT;

template <typename K>
__global__ void __launch_bounds__(kT) k_radix_hist(const K* __restrict__ key, long long n, int shift, int nblk,
                                                   unsigned* __restrict__ hist) {
  __shared__ unsigned h[256];
  const long long t0 = (long long)blockIdx.x * kRTile + threadIdx.x;
  // only the 32-bit word that holds the digit; all of a thread's loads together
  const unsigned* word = reinterpret_cast<const unsigned*>(key) + (shift >> 5);
  unsigned d[kRItems];
#pragma unroll
  for (int k = 0; k < kRItems; k++) {
    const long long i = t0 + k * kT;
    d[k] = i < n ? (word[i * (int)(sizeof(K) / 4)] >> (shift & 31)) & 255u : 256u;
  }
  h[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kRItems; k++)
    if (d[k] < 256u) atomicAdd(&h[d[k]], 1u);
  __syncthreads();
  hist[(long long)threadIdx.x * nblk + blockIdx.x] = h[threadIdx.x];
}

// digit = frame of the element (for the per-frame ranks of the sorted order)
__global__ void __launch_bounds__(kT) k_frame_hist(const __grid_constant__ FrameTab ft, const unsigned* __restrict__ val, long long n, int nblk,
                                                   unsigned* __restrict__ hist) {
  __shared__ unsigned h[256];
  __shared__ unsigned s_in[kMaxFrames + 1];
  const long long t0 = (long long)blockIdx.x * kRTile + threadIdx.x;
  unsigned v[kRItems];
#pragma unroll
  for (int k = 0; k < kRItems; k++) v[k] = t0 + k * kT < n ? val[t0 + k * kT] : 0u;
  h[threadIdx.x] = 0;
  load_in_start(ft, s_in);
  const int nf = ft.nframes;
#pragma unroll
  for (int k = 0; k < kRItems; k++)
    if (t0 + k * kT < n) atomicAdd(&h[frame_of_in(v[k], s_in, nf)], 1u);
  __syncthreads();
  if (threadIdx.x < nf) hist[(long long)threadIdx.x * nblk + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one 8-bit digit.  A block takes a tile of kRTile items,
// every warp kWItems consecutive ones in rows of 32.  A row's items of one
// digit find each other by eight ballots (one per bit); the lowest of them
// adds their number to the warp's own counter of the digit, so that the rows
// need no barrier.  One barrier, a prefix of the counters over warps and
// digits, and every item is staged in shared memory at its digit's place in
// the tile; the tile is then written out digit run by digit run, so that
// consecutive threads store to consecutive addresses.  Places past the end
// count as digit 255: they come after every item of the tile.
// What bounds it: instruction issue and shared memory in the ranking, then 24
// bytes an item through L2 and HBM (38 MB of keys and 19 MB of indices each way
// do not stay in L2 together).  4.7 million items: 52 us a pass with counters
// shared by the block (a barrier after every 512 items), 32 us now; the digit
// counts 10 us, their scan by rows 4 us (14 us as one scan of 256 x tiles).
constexpr int kSThreads = 512;
constexpr int kSWarps = kSThreads / 32;
constexpr int kWItems = kRTile / kSWarps;
constexpr int kSRows = kWItems / 32;

template <typename K>
constexpr size_t scatter_smem() {
  return (size_t)kRTile * (sizeof(K) + sizeof(unsigned)) + sizeof(unsigned short) * 256 * kSWarps;
}

template <typename K>
__global__ void __launch_bounds__(kSThreads, 2)
    k_radix_scatter(const K* __restrict__ kin, const unsigned* __restrict__ vin, K* __restrict__ kout,
                    unsigned* __restrict__ vout, long long n, int shift, int nblk, const unsigned* __restrict__ off,
                    const unsigned* __restrict__ total) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned goff[256];
  __shared__ unsigned long long scr[8];
  K* st_k = (K*)smem;
  unsigned* st_v = (unsigned*)(st_k + kRTile);
  unsigned short* cnt = (unsigned short*)(st_v + kRTile);  // [kSWarps][256]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long t0 = (long long)blockIdx.x * kRTile;
  const int tn = (int)(n - t0 < kRTile ? n - t0 : kRTile);
  K kk[kSRows] = {};
  unsigned vv[kSRows] = {};
#pragma unroll
  for (int k = 0; k < kSRows; k++) {
    const int li = w * kWItems + 32 * k + lane;
    if (li < tn) {
      kk[k] = kin[t0 + li];
      vv[k] = vin[t0 + li];
    }
  }
  unsigned o = 0, all = 0;
  if (threadIdx.x < 256) {
    o = off[(long long)threadIdx.x * nblk + blockIdx.x];
    all = total[threadIdx.x];
  }
  unsigned short* cw = cnt + w * 256;
#pragma unroll
  for (int k = 0; k < 4; k++) reinterpret_cast<unsigned*>(cw)[32 * k + lane] = 0;
  __syncwarp();
  unsigned short rank[kSRows];
#pragma unroll
  for (int k = 0; k < kSRows; k++) {
    const unsigned d = w * kWItems + 32 * k + lane < tn ? digit_of(kk[k], shift) : 255u;
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int bit = 0; bit < 8; bit++) {
      const bool one = (d >> bit) & 1u;
      const unsigned bal = __ballot_sync(0xffffffffu, one);
      peers &= one ? bal : ~bal;
    }
    const int lead = __ffs(peers) - 1;
    unsigned before = 0;
    if (lane == lead) {
      before = cw[d];
      cw[d] = (unsigned short)(before + __popc(peers));
    }
    __syncwarp();
    rank[k] = (unsigned short)(__shfl_sync(0xffffffffu, before, lead) + __popc(peers & ((1u << lane) - 1u)));
  }
  __syncthreads();
  // the digit's items in the warps before, in the tile's digits before, and
  // in all digits before: one scan over the digits carries the last two
  unsigned long long x = 0, own = 0;
  if (threadIdx.x < 256) {
    unsigned p = 0;
#pragma unroll
    for (int k = 0; k < kSWarps; k++) {
      const unsigned c = cnt[k * 256 + threadIdx.x];
      cnt[k * 256 + threadIdx.x] = (unsigned short)p;
      p += c;
    }
    own = x = ((unsigned long long)all << 32) | p;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x, q);
      if (lane >= q) x += y;
    }
    if (lane == 31) scr[w] = x;
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    unsigned long long before = x - own;
    for (int k = 0; k < w; k++) before += scr[k];
    const unsigned tile0 = (unsigned)before;
#pragma unroll
    for (int k = 0; k < kSWarps; k++) cnt[k * 256 + threadIdx.x] += (unsigned short)tile0;
    goff[threadIdx.x] = (unsigned)(before >> 32) + o - tile0;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kSRows; k++) {
    const unsigned d = w * kWItems + 32 * k + lane < tn ? digit_of(kk[k], shift) : 255u;
    const unsigned lp = cw[d] + rank[k];
    st_k[lp] = kk[k];
    st_v[lp] = vv[k];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < tn; q += kSThreads) {
    const K k = st_k[q];
    const unsigned g = goff[digit_of(k, shift)] + (unsigned)q;
    kout[g] = k;
    vout[g] = st_v[q];
  }
}

// ---- per-frame ranks: element p of frame g in sorted order -----------------

// What the duplicate removal asks of a frame: the rank of its last record
// (-1: no records), and the latest earlier frame whose sorted rows reach past
// that rank (-1: none), whose record there is what the reference compares the
// last one with (the candidate table starts zeroed for its first 10485760
// rows, struct.h:10).
struct FrameReq {
  int last, stale_frame, stale, pad;
};
struct FrameFound {
  int4 cells[2];                 // of the last record and of the stale one
  unsigned long long lo, hi;     // key of the last record
};

// Request 2 f: the last record of frame f in sorted order; 2 f + 1: the stale
// one.  One block per request: 256-ary search over the frame's row of tile
// offsets, then the place within the tile by a scan.
template <typename K>
__global__ void __launch_bounds__(kT) k_frame_find(const __grid_constant__ FrameTab ft, const FrameReq* __restrict__ req,
                                                   const unsigned* __restrict__ hoff,
                                                   int nblk, const unsigned* __restrict__ val, long long n,
                                                   const K* __restrict__ key, const int4* __restrict__ cells_in,
                                                   FrameFound* __restrict__ out, int* __restrict__ failed) {
  __shared__ unsigned s_in[kMaxFrames + 1];
  __shared__ unsigned sh[kT / 32];
  const int f = blockIdx.x >> 1, which = blockIdx.x & 1;
  const FrameReq rq = req[f];
  const int g = which ? rq.stale_frame : f, p = which ? rq.stale : rq.last;
  if (g < 0 || p < 0) return;
  load_in_start(ft, s_in);
  const int nf = ft.nframes;
  const unsigned* o = hoff + (long long)g * nblk;
  // last tile b with o[b] <= p (o[0] = 0)
  int lo = 0, hi = nblk;
  while (hi - lo > 1) {
    const int step = (hi - lo + kT - 1) / kT, at = lo + (int)threadIdx.x * step;
    const int c = __syncthreads_count(at < hi && o[at] <= (unsigned)p);
    lo += (c - 1) * step;
    hi = min(hi, lo + step);
  }
  const unsigned need = (unsigned)p - o[lo];
  const long long t0 = (long long)lo * kRTile + threadIdx.x * kRItems;
  unsigned hit = 0;
#pragma unroll
  for (int k = 0; k < kRItems; k++)
    if (t0 + k < n && frame_of_in(val[t0 + k], s_in, nf) == g) hit |= 1u << k;
  const unsigned c = __popc(hit);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned x = c;
#pragma unroll
  for (int q = 1; q < 32; q <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, q);
    if (lane >= q) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  unsigned before = x - c, all = 0;
  for (int k = 0; k < kT / 32; k++) {
    if (k < w) before += sh[k];
    all += sh[k];
  }
  if (need >= all && threadIdx.x == 0) *failed = 1;
  if (need >= before && need < before + c) {
    for (unsigned q = before; q < need; q++) hit &= hit - 1;
    const long long at = t0 + __ffs(hit) - 1;
    out[f].cells[which] = cells_in[val[at]];
    if (!which) key_split(key[at], &out[f].lo, &out[f].hi);
  }
}

// Last run of a frame that is not written (its last record's cells equal the
// stale ones, zeros where there is none).
struct FrameDrop {
  unsigned long long lo, hi;
  int drop, pad;
};
__device__ __forceinline__ FrameDrop frame_drop(const FrameReq& rq, const FrameFound& fd) {
  const int4 a = fd.cells[0], b = rq.stale_frame >= 0 ? fd.cells[1] : make_int4(0, 0, 0, 0);
  return {fd.lo, fd.hi, rq.last >= 0 && a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w, 0};
}

// ---- duplicate removal per (cells, frame) run ------------------------------

// A tile of kTile records a block, with its neighbours, in shared memory: keys
// and frames.  A record that is a run of its own is settled there; the first
// records of longer runs go on a list, whose runs are then shared out among
// the threads, the SNRs of four members in flight at a time.  removed[f]:
// records of frame f that are not kept.  24 x 2^18 records, few duplicates (50
// 000 of 4.7 million) and many (lattice points on 64 lines x 256 positions): 67
// and 94 us with a thread per record and SNRs from a compact array; 41 and
// 55 us here (303 with the runs walked by the threads that found them).
template <typename K>
__global__ void __launch_bounds__(kT) k_dedup(const __grid_constant__ FrameTab ft, const K* __restrict__ key, const unsigned* __restrict__ val,
                                              const double* __restrict__ snr_in, const FrameReq* __restrict__ req,
                                              const FrameFound* __restrict__ found, long long n, uint8_t* __restrict__ keep, unsigned* __restrict__ removed) {
  __shared__ unsigned short list[kTile];
  __shared__ unsigned nlist, hcount[256];
  __shared__ K s_key[kTile + 2];
  __shared__ uint8_t s_frame[kTile + 2];
  __shared__ FrameDrop s_drop[kMaxFrames];
  __shared__ unsigned s_in[kMaxFrames + 1];
  const long long t0 = (long long)blockIdx.x * kTile;
  unsigned v[kIt];
#pragma unroll
  for (int k = 0; k < kIt; k++) {
    const long long i = t0 + k * kT + threadIdx.x;
    v[k] = 0;
    if (i < n) {
      s_key[1 + k * kT + threadIdx.x] = key[i];
      v[k] = val[i];
    }
  }
  if (threadIdx.x == 0) nlist = 0;
  hcount[threadIdx.x] = 0;
  if (threadIdx.x < ft.nframes) s_drop[threadIdx.x] = frame_drop(req[threadIdx.x], found[threadIdx.x]);
  load_in_start(ft, s_in);
  const int nf = ft.nframes;
#pragma unroll
  for (int k = 0; k < kIt; k++) s_frame[1 + k * kT + threadIdx.x] = (uint8_t)frame_of_in(v[k], s_in, nf);
  if (threadIdx.x < 2) {
    const long long i = threadIdx.x ? t0 + kTile : t0 - 1;
    if (i >= 0 && i < n) {
      s_key[threadIdx.x ? kTile + 1 : 0] = key[i];
      s_frame[threadIdx.x ? kTile + 1 : 0] = (uint8_t)frame_of_in(val[i], s_in, nf);
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kIt; k++) {
    const int li = 1 + k * kT + threadIdx.x;
    const long long i = t0 + li - 1;
    if (i >= n) break;
    const K k0 = s_key[li];
    const int f = s_frame[li];
    if (i > 0 && s_key[li - 1] == k0 && s_frame[li - 1] == f) continue;  // not the first of its run
    const bool dropped = s_drop[f].drop && key_is(k0, s_drop[f].lo, s_drop[f].hi);
    const bool single = !(i + 1 < n && s_key[li + 1] == k0 && s_frame[li + 1] == f);
    if (single && !dropped) keep[i] = 1;
    else list[atomicAdd(&nlist, 1u)] = (unsigned short)li;
  }
  __syncthreads();
  const unsigned nl = nlist;
  for (unsigned q = threadIdx.x; q < nl; q += kT) {
    const int li = list[q];
    const long long i = t0 + li - 1;
    const K k0 = s_key[li];
    const int f = s_frame[li];
    // the run [i, j], within the tile and then beyond it
    int le = li;
    while (le <= kTile && t0 + le < n && s_key[le + 1] == k0 && s_frame[le + 1] == f) le++;
    long long j = t0 + le - 1;
    if (le > kTile)
      while (j + 1 < n && key[j + 1] == k0 && frame_of_in(val[j + 1], s_in, nf) == f) j++;
    const bool dropped = s_drop[f].drop && key_is(k0, s_drop[f].lo, s_drop[f].hi);
    atomicAdd(&hcount[f], (unsigned)(j - i + (dropped ? 1 : 0)));
    if (dropped) continue;
    // coincidences.c:317-413 over the pairs (t, t + 1) of the run
    const long long fs = s_in[f];
    long long maxsnridx = 0, maxi = i, idx = 0;
    double candsnr = 0, s0 = 0;
    for (long long t4 = i; t4 <= j; t4 += 4) {
      unsigned v4[4];
      double s4[4];
#pragma unroll
      for (int u = 0; u < 4; u++) v4[u] = t4 + u <= j ? val[t4 + u] : 0u;
#pragma unroll
      for (int u = 0; u < 4; u++) s4[u] = t4 + u <= j ? snr_in[v4[u]] : 0.;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const long long t1 = t4 + u;  // the pair (t1 - 1, t1)
        if (t1 > j) break;
        const double s1 = s4[u];
        const long long idx1 = (long long)v4[u] - fs;
        if (t1 > i) {
          if (!maxsnridx) {
            maxsnridx = (s0 > s1) ? idx : idx1;
            maxi = (s0 > s1) ? t1 - 1 : t1;
            candsnr = (s0 > s1) ? s0 : s1;
          } else {
            if (s0 > candsnr) {
              maxsnridx = idx; maxi = t1 - 1; candsnr = s0;
            } else if (s1 > candsnr) {
              maxsnridx = idx1; maxi = t1; candsnr = s1;
            }
          }
        }
        idx = idx1;
        s0 = s1;
      }
    }
    keep[maxsnridx ? maxi : j] = 1;
  }
  __syncthreads();
  if (hcount[threadIdx.x]) atomicAdd(&removed[threadIdx.x], hcount[threadIdx.x]);
}

// keep flags by in-band index, from the flags by sorted position
__global__ void k_keep_scatter(const uint8_t* __restrict__ keep, const unsigned* __restrict__ val, long long n,
                               uint8_t* __restrict__ keep_in) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) keep_in[val[i]] = keep[i];
}

// per-tile counts of a 0/1 array
__global__ void __launch_bounds__(kT) k_tile_count(const uint8_t* __restrict__ flag, long long n, unsigned* __restrict__ cnt) {
  __shared__ unsigned sh[kT / 32];
  const long long t0 = (long long)blockIdx.x * kTile;
  unsigned c = 0;
  for (int k = 0; k < kIt; k++) {
    const long long i = t0 + (long long)k * kT + threadIdx.x;
    if (i < n) c += flag[i];
  }
  const unsigned tot = block_sum(c, sh);
  if (threadIdx.x == 0) cnt[blockIdx.x] = tot;
}

// survivors in sorted order: key and in-band index
template <typename K>
__global__ void __launch_bounds__(kT) k_compact_surv(const uint8_t* __restrict__ keep, long long n,
                                                     const unsigned* __restrict__ off, const K* __restrict__ key,
                                                     const unsigned* __restrict__ val, K* __restrict__ skey,
                                                     unsigned* __restrict__ sval) {
  __shared__ unsigned sh[kT / 32];
  __shared__ unsigned short list[kTile];
  const long long t0 = (long long)blockIdx.x * kTile;
  const unsigned base = off[blockIdx.x];
  const unsigned tot = tile_list(keep, t0, n, list, sh);
  for (unsigned q = threadIdx.x; q < tot; q += kT) {
    const long long i = t0 + list[q];
    skey[base + q] = key[i];
    sval[base + q] = val[i];
  }
}

// runs of equal cells among the survivors (coincidences.c:449-486)
// (a tile of kTile keys with its neighbours in shared memory; tile counts of
// the stored groups to cnt)
template <typename K>
__global__ void __launch_bounds__(kT) k_groups(const K* __restrict__ skey, long long G, int mincoin,
                                               uint8_t* __restrict__ gflag, unsigned* __restrict__ gend,
                                               unsigned* __restrict__ gw, int* __restrict__ last_unstored,
                                               unsigned* __restrict__ members, unsigned* __restrict__ cnt) {
  __shared__ K s_key[kTile + 2];
  __shared__ unsigned sh[kT / 32];
  const long long t0 = (long long)blockIdx.x * kTile;
#pragma unroll
  for (int k = 0; k < kIt; k++) {
    const long long i = t0 + k * kT + threadIdx.x;
    if (i < G) s_key[1 + k * kT + threadIdx.x] = skey[i];
  }
  if (threadIdx.x < 2) {
    const long long i = threadIdx.x ? t0 + kTile : t0 - 1;
    if (i >= 0 && i < G) s_key[threadIdx.x ? kTile + 1 : 0] = skey[i];
  }
  __syncthreads();
  unsigned stored = 0, mem = 0;
#pragma unroll
  for (int k = 0; k < kIt; k++) {
    const int li = 1 + k * kT + threadIdx.x;
    const long long i = t0 + li - 1;
    if (i >= G) break;
    const K k0 = s_key[li];
    uint8_t fl = 0;
    if ((i == 0 || !(s_key[li - 1] == k0)) && i + 1 < G && s_key[li + 1] == k0) {  // (mincoin >= 2)
      long long j = i + 1;
      while (j + 1 < G && skey[j + 1] == k0) j++;
      const long long w = j - i + 1;
      if (w >= mincoin) {
        if (j < G - 1) {
          fl = 1;
          gend[i] = (unsigned)j;
          gw[i] = (unsigned)w;
          stored++;
          mem += (unsigned)w;
        } else {
          *last_unstored = 1;
        }
      }
    }
    gflag[i] = fl;
  }
  const unsigned tot = block_sum(stored, sh), tm = block_sum(mem, sh);
  if (threadIdx.x == 0) {
    cnt[blockIdx.x] = tot;
    if (tm) atomicAdd(members, tm);
  }
}

__global__ void __launch_bounds__(kT) k_compact_groups(const uint8_t* __restrict__ gflag, long long G,
                                                       const unsigned* __restrict__ off,
                                                       const unsigned* __restrict__ gend, const unsigned* __restrict__ gw,
                                                       unsigned long long* __restrict__ wkey,
                                                       unsigned* __restrict__ cend, unsigned* __restrict__ cw,
                                                       unsigned* __restrict__ cidx) {
  __shared__ unsigned sh[kT / 32];
  __shared__ unsigned short list[kTile];
  const long long t0 = (long long)blockIdx.x * kTile;
  const unsigned base = off[blockIdx.x];
  const unsigned tot = tile_list(gflag, t0, G, list, sh);
  for (unsigned q = threadIdx.x; q < tot; q += kT) {
    const long long i = t0 + list[q];
    const unsigned o = base + q;
    cend[o] = gend[i];
    cw[o] = gw[i];
    wkey[o] = 255ull - gw[i];   // multiplicity <= frames <= 255: one digit
    cidx[o] = o;
  }
}

__global__ void k_gather_w(const unsigned* __restrict__ order, const unsigned* __restrict__ cw, int K,
                           unsigned* __restrict__ w_sorted) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < K) w_sorted[q] = cw[order[q]];
}

// coincidences.c:488-525: means over the members k = end, end - 1, ...  A block
// takes kG coincidences, whose members lie one after the other in the output:
// a thread per member loads and shifts it (a thread per coincidence spent 60 us
// on 12 000 of them, one dependent load after the other), then a thread per
// coincidence and column adds in the reference's order.  (A warp per
// coincidence leaves most lanes of the FP64 pipe idle: 257 000 coincidences 287
// us, 136 with a thread each, 157 here; 12 000: 31, 76 and 31 us.)
constexpr int kG = 32;
__global__ void __launch_bounds__(kT) k_means(const __grid_constant__ FrameTab ft, const unsigned* __restrict__ order, const unsigned* __restrict__ cend,
                                              const unsigned* __restrict__ cw, const unsigned* __restrict__ first,
                                              int K, const unsigned* __restrict__ sval,
                                              const unsigned* __restrict__ rawidx, const double* __restrict__ rec,
                                              double N, int refr, pa_coinc_rec* __restrict__ out,
                                              int* __restrict__ fra, int* __restrict__ ops) {
  __shared__ unsigned s_in[kMaxFrames + 1];
  __shared__ double s_t[5][kT];
  __shared__ unsigned s_first[kG + 1], s_end[kG];
  const int q0 = blockIdx.x * kG, nq = min(kG, K - q0);
  if (threadIdx.x < nq) {
    const unsigned g = order[q0 + threadIdx.x], f = first[q0 + threadIdx.x], w = cw[g];
    s_first[threadIdx.x] = f;
    s_end[threadIdx.x] = cend[g];
    if (threadIdx.x == nq - 1) s_first[nq] = f + w;
  }
  load_in_start(ft, s_in);
  const int nf = ft.nframes;
  const unsigned m0 = s_first[0], m1 = s_first[nq];
  const int sg = threadIdx.x / 5, sk = threadIdx.x % 5;  // the sum of this thread
  double m = 0;
  for (unsigned c0 = m0; c0 < m1; c0 += kT) {
    const unsigned mm = c0 + threadIdx.x;
    if (mm < m1) {
      int lo = 0, hi = nq;  // the member's coincidence: s_first[lo] <= mm < s_first[lo + 1]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_first[mid] <= mm) lo = mid; else hi = mid;
      }
      const unsigned v = sval[s_end[lo] - (mm - s_first[lo])];
      const int f = frame_of_in(v, s_in, nf);
      const long long r = rawidx[v];
      const double* c = rec + 5 * r;
      const double fshift = (double)(refr - ft.frame_no[f]);
      s_t[0][threadIdx.x] = __dadd_rn(c[0], __dmul_rn(__dmul_rn(__dmul_rn(2., c[1]), N), fshift));
      s_t[1][threadIdx.x] = c[1];
      s_t[2][threadIdx.x] = c[2];
      s_t[3][threadIdx.x] = c[3];
      s_t[4][threadIdx.x] = __dmul_rn(c[4], c[4]);
      ops[mm] = (int)(r - (long long)ft.raw_start[f]);
      fra[mm] = ft.frame_no[f];
    }
    __syncthreads();
    if (sg < nq) {
      const unsigned a = max(s_first[sg], c0), b = min(s_first[sg + 1], c0 + kT);
      for (unsigned l = a; l < b; l++) m = __dadd_rn(m, s_t[sk][l - c0]);
    }
    __syncthreads();
  }
  if (sg >= nq) return;
  const int w = (int)(s_first[sg + 1] - s_first[sg]);
  pa_coinc_rec* o = out + q0 + sg;
  o->mean[sk] = sk < 4 ? __ddiv_rn(m, (double)w) : __dsqrt_rn(m);
  if (sk == 0) {
    o->w = w;
    o->first = (int)s_first[sg];
  }
}
static_assert(5 * kG <= kT, "a thread per sum");

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct pa_coinc {
  pa_coinc_cfg cfg;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::string err;
  long long launches = 0;
  double last_ms = 0;
  FrameTab ft;
  std::vector<int> frames;
  std::vector<long long> raw_start;   // per frame, size nframes + 1
  long long nraw = 0;
  // device buffers (grow only)
  struct Buf {
    void* p = nullptr;
    size_t n = 0;
  };
  Buf rec, cells_raw, flag, snr_raw, blkcnt, scan_tmp, minmax, rawidx, cells_in, snr_in, digits, keyA, keyB, valA, valB, hist,
      keep, keep_in, uniq, req, found, skey, sval, gflag, gend, gw, lastu, wkeyA, wkeyB, cend, cw, cidxA, cidxB,
      wsort, means, fra, ops;
  // optional per-kernel profile: events around each launch while on
  bool prof_on = false;
  struct Open {
    int kind;
    cudaEvent_t a, b;
  };
  std::vector<Open> prof_open;
  double prof_ms[16] = {0};
  long long prof_n[16] = {0};
  // results
  pa_coinc_summary sum;
  std::vector<int> frameinfo;
  // results in page-locked host memory (grow only)
  pa_coinc_rec* h_recs = nullptr;
  int* h_fra = nullptr;
  int* h_ops = nullptr;
  size_t h_recs_cap = 0, h_mem_cap = 0;
  long long n_in = 0;
  const unsigned* val_sorted = nullptr;  // in-band index of each sorted position (last run)
  bool ev1_done = false;                 // the run's end event is already on the stream
};

thread_local std::string g_coinc_create_error;  // per host thread, as the other create errors

enum CoincKind { CK_CELLS = 0, CK_INBAND, CK_SORT_HIST, CK_SORT_SCATTER, CK_SCAN, CK_FRAME_RANK, CK_DEDUP,
                 CK_COMPACT, CK_GROUPS, CK_MEANS, CK_COUNT };
static const char* const kCoincKindName[CK_COUNT] = {
    "coinc_cells", "coinc_inband", "coinc_sort_hist", "coinc_sort_scatter", "coinc_scan",
    "coinc_frame_rank", "coinc_dedup", "coinc_compact", "coinc_groups", "coinc_means"};

// CUDA events around the launches of its scope, when profiling is on
struct Span {
  pa_coinc* c;
  int kind;
  cudaEvent_t a = nullptr, b = nullptr;
  Span(pa_coinc* c_, int k) : c(c_), kind(k) {
    if (c->prof_on && cudaEventCreate(&a) == cudaSuccess && cudaEventCreate(&b) == cudaSuccess)
      cudaEventRecord(a, c->stream);
  }
  ~Span() {
    if (a && b) {
      cudaEventRecord(b, c->stream);
      c->prof_open.push_back({kind, a, b});
    }
  }
};

static void prof_collect(pa_coinc* c) {
  for (auto& o : c->prof_open) {
    float ms = 0;
    if (cudaEventSynchronize(o.b) == cudaSuccess && cudaEventElapsedTime(&ms, o.a, o.b) == cudaSuccess) {
      c->prof_ms[o.kind] += ms;
      c->prof_n[o.kind]++;
    }
    cudaEventDestroy(o.a);
    cudaEventDestroy(o.b);
  }
  c->prof_open.clear();
}

static int cfail(pa_coinc* c, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (c) c->err = buf; else g_coinc_create_error = buf;
  return code;
}

#define CCK(call, what)                                                                  \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess) return cfail(c, PA_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e_)); \
  } while (0)

static int ensure(pa_coinc* c, pa_coinc::Buf& b, size_t bytes) {
  if (bytes <= b.n && b.p) return PA_OK;
  size_t nb = bytes < 256 ? 256 : bytes;
  if (b.n) nb = nb > b.n + b.n / 2 ? nb : b.n + b.n / 2;
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, nb);
  if (e != cudaSuccess) return cfail(c, PA_ERR_NOMEM, "cudaMalloc(%zu): %s", nb, cudaGetErrorString(e));
  if (b.p) {
    // work queued on the stream may still read the old buffer
    cudaStreamSynchronize(c->stream);
    cudaFree(b.p);
  }
  b.p = p;
  b.n = nb;
  return PA_OK;
}
#define ENS(buf, bytes)                            \
  do {                                             \
    int rc_ = ensure(c, c->buf, (size_t)(bytes));  \
    if (rc_) return rc_;                           \
  } while (0)

template <typename T>
static T* P(pa_coinc::Buf& b) { return (T*)b.p; }

// exclusive scan of d[0..n) in place; tmp needs room for the block sums of
// every level
static int scan_excl(pa_coinc* c, unsigned* d, long long n, unsigned* tmp) {
  if (n <= 0) return PA_OK;
  if (n <= kScanOne) {
    Span sp_(c, CK_SCAN);
    k_scan_one<<<1, kST, 0, c->stream>>>(d, (int)n);
    c->launches++;
    CCK(cudaGetLastError(), "scan");
    return PA_OK;
  }
  const long long nb = (n + kTile - 1) / kTile;
  {
    Span sp_(c, CK_SCAN);
    k_scan_tiles<<<(unsigned)nb, kT, 0, c->stream>>>(d, n, nb > 1 ? tmp : nullptr);
  }
  c->launches++;
  if (nb > 1) {
    int rc = scan_excl(c, tmp, nb, tmp + nb);
    if (rc) return rc;
    {
      Span sp_(c, CK_SCAN);
      k_scan_add<<<(unsigned)nb, kT, 0, c->stream>>>(d, n, tmp);
    }
    c->launches++;
  }
  CCK(cudaGetLastError(), "scan");
  return PA_OK;
}

static long long scan_tmp_len(long long n) {
  long long t = 0;
  while (n > 1) {
    n = (n + kTile - 1) / kTile;
    t += n;
  }
  return t + 1;
}

template <typename K>
static int radix_sort(pa_coinc* c, K*& k, unsigned*& v, K* k2, unsigned* v2, long long n, int bits) {
  pa::TraceRange trace_("coinc radix sort");
  const int nblk = (int)((n + kRTile - 1) / kRTile);
  ENS(hist, sizeof(unsigned) * 256ll * nblk);
  ENS(digits, sizeof(unsigned) * 256);
  // the staged scatter needs more than the default 48 KB of shared memory
  CCK(cudaFuncSetAttribute(k_radix_scatter<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem<K>()),
      "cudaFuncSetAttribute");
  K* ka = k;
  unsigned* va = v;
  K* kb = k2;
  unsigned* vb = v2;
  for (int s = 0; s < bits; s += 8) {
    {
      Span sp_(c, CK_SORT_HIST);
      k_radix_hist<K><<<nblk, kT, 0, c->stream>>>(ka, n, s, nblk, P<unsigned>(c->hist));
    }
    {
      Span sp_(c, CK_SCAN);
      k_scan_rows<<<256, kT, 0, c->stream>>>(P<unsigned>(c->hist), nblk, P<unsigned>(c->digits));
    }
    c->launches += 2;
    {
      Span sp_(c, CK_SORT_SCATTER);
      k_radix_scatter<K><<<nblk, kSThreads, scatter_smem<K>(), c->stream>>>(
          ka, va, kb, vb, n, s, nblk, P<unsigned>(c->hist), P<unsigned>(c->digits));
    }
    c->launches++;
    CCK(cudaGetLastError(), "radix pass");
    K* tk = ka; ka = kb; kb = tk;
    unsigned* tv = va; va = vb; vb = tv;
  }
  k = ka;
  v = va;
  return PA_OK;
}

extern "C" {

int pa_coinc_vedva(const double* fisher, double* vedva) {
  if (!fisher || !vedva) return PA_ERR_ARG;
  // cyclic Jacobi rotations on a copy (row-major), eigenvectors as columns
  double a[16], v[16];
  memcpy(a, fisher, sizeof(a));
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++) v[4 * i + j] = (i == j);
  for (int sweep = 0; sweep < 64; sweep++) {
    double off = 0;
    for (int i = 0; i < 4; i++)
      for (int j = i + 1; j < 4; j++) off += a[4 * i + j] * a[4 * i + j];
    if (off < 1e-300) break;
    for (int p = 0; p < 4; p++)
      for (int q = p + 1; q < 4; q++) {
        const double apq = a[4 * p + q];
        if (apq == 0.0) continue;
        const double theta = (a[4 * q + q] - a[4 * p + p]) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double cs = 1.0 / sqrt(t * t + 1.0), sn = t * cs;
        for (int k = 0; k < 4; k++) {
          const double akp = a[4 * k + p], akq = a[4 * k + q];
          a[4 * k + p] = cs * akp - sn * akq;
          a[4 * k + q] = sn * akp + cs * akq;
        }
        for (int k = 0; k < 4; k++) {
          const double apk = a[4 * p + k], aqk = a[4 * q + k];
          a[4 * p + k] = cs * apk - sn * aqk;
          a[4 * q + k] = sn * apk + cs * aqk;
        }
        for (int k = 0; k < 4; k++) {
          const double vkp = v[4 * k + p], vkq = v[4 * k + q];
          v[4 * k + p] = cs * vkp - sn * vkq;
          v[4 * k + q] = sn * vkp + cs * vkq;
        }
      }
  }
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++) vedva[4 * i + j] = v[4 * i + j] * sqrt(a[4 * j + j]);
  return PA_OK;
}

const char* pa_coinc_last_error(const pa_coinc* c) {
  return c ? c->err.c_str() : g_coinc_create_error.c_str();
}

pa_coinc* pa_coinc_create(const pa_coinc_cfg* cfg, int* status) {
  auto ret = [&](int st) {
    if (status) *status = st;
    return (pa_coinc*)nullptr;
  };
  pa_coinc* c = nullptr;
  if (!cfg || cfg->N < 1 || cfg->mincoin < 2)
    return cfail(c, PA_ERR_ARG, "pa_coinc_create: invalid configuration (N >= 1, mincoin >= 2)"), ret(PA_ERR_ARG);
  for (int j = 0; j < 4; j++)
    if (cfg->scale[j] == 0) return cfail(c, PA_ERR_ARG, "pa_coinc_create: scale digit 0"), ret(PA_ERR_ARG);
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1)
    return cfail(c, PA_ERR_NODEV, "pa_coinc_create: no CUDA device"), ret(PA_ERR_NODEV);
  if (cfg->device < 0 || cfg->device >= ndev)
    return cfail(c, PA_ERR_ARG, "pa_coinc_create: device %d out of range", cfg->device), ret(PA_ERR_ARG);
  c = new pa_coinc();
  c->cfg = *cfg;
  cudaError_t e;
  if ((e = cudaSetDevice(cfg->device)) != cudaSuccess ||
      (e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaEventCreate(&c->ev0)) != cudaSuccess || (e = cudaEventCreate(&c->ev1)) != cudaSuccess) {
    g_coinc_create_error = std::string("pa_coinc_create: ") + cudaGetErrorString(e);
    pa_coinc_destroy(c);
    if (status) *status = PA_ERR_CUDA;
    return nullptr;
  }
  pa_coinc_reset(c);
  if (status) *status = PA_OK;
  return c;
}

void pa_coinc_destroy(pa_coinc* c) {
  if (!c) return;
  cudaSetDevice(c->cfg.device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  pa_coinc::Buf* bufs[] = {&c->rec, &c->cells_raw, &c->flag, &c->snr_raw, &c->blkcnt, &c->scan_tmp, &c->minmax, &c->rawidx,
                           &c->cells_in, &c->snr_in, &c->digits, &c->keyA, &c->keyB, &c->valA, &c->valB, &c->hist, &c->keep,
                           &c->keep_in, &c->uniq, &c->req, &c->found, &c->skey, &c->sval, &c->gflag, &c->gend,
                           &c->gw, &c->lastu, &c->wkeyA, &c->wkeyB, &c->cend, &c->cw, &c->cidxA, &c->cidxB,
                           &c->wsort, &c->means, &c->fra, &c->ops};
  for (auto* b : bufs)
    if (b->p) cudaFree(b->p);
  for (auto& o : c->prof_open) {
    cudaEventDestroy(o.a);
    cudaEventDestroy(o.b);
  }
  if (c->h_recs) cudaFreeHost(c->h_recs);
  if (c->h_fra) cudaFreeHost(c->h_fra);
  if (c->h_ops) cudaFreeHost(c->h_ops);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

int pa_coinc_reset(pa_coinc* c) {
  if (!c) return PA_ERR_ARG;
  c->frames.clear();
  c->val_sorted = nullptr;
  c->raw_start.assign(1, 0);
  c->nraw = 0;
  c->n_in = 0;
  memset(&c->sum, 0, sizeof(c->sum));
  c->frameinfo.clear();

  return PA_OK;
}

int pa_coinc_add_frame(pa_coinc* c, int frame, const double* records, long long n) {
  pa::TraceRange trace_("pa_coinc_add_frame");
  if (!c || n < 0 || (n > 0 && !records)) return PA_ERR_ARG;
  if ((int)c->frames.size() >= kMaxFrames) return cfail(c, PA_ERR_ARG, "pa_coinc_add_frame: more than %d frames", kMaxFrames);
  if (c->nraw + n >= (1ll << 31)) return cfail(c, PA_ERR_ARG, "pa_coinc_add_frame: more than 2^31 records");
  CCK(cudaSetDevice(c->cfg.device), "cudaSetDevice");
  const size_t need = sizeof(double) * 5 * (size_t)(c->nraw + n);
  if (need > c->rec.n) {
    // grow keeping the frames already uploaded
    size_t nb = need + need / 2;
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, nb);
    if (e != cudaSuccess) return cfail(c, PA_ERR_NOMEM, "cudaMalloc(%zu): %s", nb, cudaGetErrorString(e));
    if (c->rec.p) {
      CCK(cudaMemcpyAsync(p, c->rec.p, sizeof(double) * 5 * (size_t)c->nraw, cudaMemcpyDeviceToDevice, c->stream),
          "cudaMemcpyAsync");
      CCK(cudaStreamSynchronize(c->stream), "sync");
      cudaFree(c->rec.p);
    }
    c->rec.p = p;
    c->rec.n = nb;
  }
  if (n) {
    CCK(cudaMemcpyAsync((double*)c->rec.p + 5 * c->nraw, records, sizeof(double) * 5 * (size_t)n,
                        cudaMemcpyHostToDevice, c->stream),
        "cudaMemcpyAsync");
    // the caller's buffer is free again when the call returns
    CCK(cudaStreamSynchronize(c->stream), "sync");
  }
  c->frames.push_back(frame);
  c->nraw += n;
  c->raw_start.push_back(c->nraw);
  return PA_OK;
}

}  // extern "C"

template <typename K>
static int run_keyed(pa_coinc* c, const KeyLayout& L, int nblk1, std::vector<long long>& nin_f) {
  pa::TraceRange trace_("coinc sort, duplicates, coincidences");
  const int nf = (int)c->frames.size();
  const long long n = c->n_in;
  ENS(snr_in, sizeof(double) * n);
  ENS(keyA, sizeof(K) * n);
  ENS(keyB, sizeof(K) * n);
  ENS(valA, sizeof(unsigned) * n);
  ENS(valB, sizeof(unsigned) * n);
  {
    Span sp_(c, CK_INBAND);
    k_inband<K><<<nblk1, kT, 0, c->stream>>>(c->ft, P<uint8_t>(c->flag), P<int4>(c->cells_raw), P<unsigned>(c->blkcnt), L,
                                             P<unsigned>(c->rawidx), P<int4>(c->cells_in),
                                             P<K>(c->keyA), P<unsigned>(c->valA), P<double>(c->snr_raw),
                                             P<double>(c->snr_in));
  }
  c->launches++;
  CCK(cudaGetLastError(), "k_inband");
  K* key = P<K>(c->keyA);
  unsigned* val = P<unsigned>(c->valA);
  int rc = radix_sort<K>(c, key, val, key == P<K>(c->keyA) ? P<K>(c->keyB) : P<K>(c->keyA),
                         val == P<unsigned>(c->valA) ? P<unsigned>(c->valB) : P<unsigned>(c->valA), n, L.bits);
  if (rc) return rc;

  // per-frame ranks of the sorted order: each frame's last record and the
  // record of an earlier frame at the position one past it
  const int nblkR = (int)((n + kRTile - 1) / kRTile);
  ENS(hist, sizeof(unsigned) * 256ll * nblkR);
  ENS(digits, sizeof(unsigned) * 256);
  ENS(req, sizeof(FrameReq) * nf);
  ENS(found, sizeof(FrameFound) * nf);
  ENS(uniq, sizeof(unsigned) * 257);  // removed records per frame, and the failure flag of the rank lookup
  CCK(cudaMemsetAsync(c->uniq.p, 0, sizeof(unsigned) * 257, c->stream), "memset");
  std::vector<FrameReq> req(nf);
  for (int f = 0; f < nf; f++) {
    req[f] = {(int)(nin_f[f] - 1), -1, -1, 0};
    if (nin_f[f] < 1 || nin_f[f] >= 10485760) continue;
    for (int g = f - 1; g >= 0; g--)
      if (nin_f[g] > nin_f[f]) {
        req[f].stale_frame = g;
        req[f].stale = (int)nin_f[f];
        break;
      }
  }
  CCK(cudaMemcpyAsync(c->req.p, req.data(), sizeof(FrameReq) * nf, cudaMemcpyHostToDevice, c->stream), "copy");
  {
    Span sp_(c, CK_FRAME_RANK);
    k_frame_hist<<<nblkR, kT, 0, c->stream>>>(c->ft, val, n, nblkR, P<unsigned>(c->hist));
  }
  {
    Span sp_(c, CK_SCAN);
    k_scan_rows<<<nf, kT, 0, c->stream>>>(P<unsigned>(c->hist), nblkR, P<unsigned>(c->digits));
  }
  {
    Span sp_(c, CK_FRAME_RANK);
    k_frame_find<K><<<2 * nf, kT, 0, c->stream>>>(c->ft, P<FrameReq>(c->req), P<unsigned>(c->hist), nblkR, val, n, key,
                                                  P<int4>(c->cells_in), P<FrameFound>(c->found),
                                                  (int*)(P<unsigned>(c->uniq) + 256));
  }
  c->launches += 3;
  CCK(cudaGetLastError(), "k_frame_find");

  // duplicate removal
  ENS(keep, n);
  CCK(cudaMemsetAsync(c->keep.p, 0, n, c->stream), "memset");
  c->val_sorted = val;
  {
    Span sp_(c, CK_DEDUP);
    k_dedup<K><<<(unsigned)((n + kTile - 1) / kTile), kT, 0, c->stream>>>(
        c->ft, key, val, P<double>(c->snr_in), P<FrameReq>(c->req), P<FrameFound>(c->found), n,
        P<uint8_t>(c->keep), P<unsigned>(c->uniq));
  }
  c->launches++;
  CCK(cudaGetLastError(), "k_dedup");
  // survivors in sorted order
  const long long nt = (n + kTile - 1) / kTile;
  ENS(blkcnt, sizeof(unsigned) * (nt + 1));
  ENS(scan_tmp, sizeof(unsigned) * scan_tmp_len(nt + 1));
  {
    Span sp_(c, CK_COMPACT);
    k_tile_count<<<(unsigned)nt, kT, 0, c->stream>>>(P<uint8_t>(c->keep), n, P<unsigned>(c->blkcnt));
  }
  c->launches++;
  CCK(cudaMemsetAsync(P<unsigned>(c->blkcnt) + nt, 0, sizeof(unsigned), c->stream), "memset");
  rc = scan_excl(c, P<unsigned>(c->blkcnt), nt + 1, P<unsigned>(c->scan_tmp));
  if (rc) return rc;
  unsigned G = 0;
  std::vector<unsigned> uniq(257, 0);
  CCK(cudaMemcpyAsync(&G, P<unsigned>(c->blkcnt) + nt, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream), "copy");
  CCK(cudaMemcpyAsync(uniq.data(), c->uniq.p, sizeof(unsigned) * 257, cudaMemcpyDeviceToHost, c->stream), "copy");
  CCK(cudaStreamSynchronize(c->stream), "sync");
  if (uniq[256]) return cfail(c, PA_ERR_CUDA, "pa_coinc_run: frame rank lookup failed");
  for (int f = 0; f < nf; f++) c->frameinfo[3 * f + 2] = (int)(nin_f[f] - uniq[f]);
  c->sum.unique = G;
  if (G == 0) return PA_OK;
  ENS(skey, sizeof(K) * G);
  ENS(sval, sizeof(unsigned) * G);
  {
    Span sp_(c, CK_COMPACT);
    k_compact_surv<K><<<(unsigned)nt, kT, 0, c->stream>>>(P<uint8_t>(c->keep), n, P<unsigned>(c->blkcnt), key, val,
                                                           P<K>(c->skey), P<unsigned>(c->sval));
  }
  c->launches++;
  CCK(cudaGetLastError(), "k_compact_surv");

  // coincidences: runs of equal cells
  ENS(gflag, G);
  ENS(gend, sizeof(unsigned) * G);
  ENS(gw, sizeof(unsigned) * G);
  ENS(lastu, 2 * sizeof(int));  // and the number of members of the stored groups
  CCK(cudaMemsetAsync(c->lastu.p, 0, 2 * sizeof(int), c->stream), "memset");
  const long long gt = ((long long)G + kTile - 1) / kTile;
  ENS(blkcnt, sizeof(unsigned) * (gt + 1));
  ENS(scan_tmp, sizeof(unsigned) * scan_tmp_len(gt + 1));
  {
    Span sp_(c, CK_GROUPS);
    k_groups<K><<<(unsigned)gt, kT, 0, c->stream>>>(P<K>(c->skey), G, c->cfg.mincoin, P<uint8_t>(c->gflag),
                                                   P<unsigned>(c->gend), P<unsigned>(c->gw), P<int>(c->lastu),
                                                   P<unsigned>(c->lastu) + 1, P<unsigned>(c->blkcnt));
  }
  c->launches++;
  CCK(cudaGetLastError(), "k_groups");
  CCK(cudaMemsetAsync(P<unsigned>(c->blkcnt) + gt, 0, sizeof(unsigned), c->stream), "memset");
  rc = scan_excl(c, P<unsigned>(c->blkcnt), gt + 1, P<unsigned>(c->scan_tmp));
  if (rc) return rc;
  unsigned Kc = 0;
  int lu[2] = {0, 0};
  CCK(cudaMemcpyAsync(&Kc, P<unsigned>(c->blkcnt) + gt, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream), "copy");
  CCK(cudaMemcpyAsync(lu, c->lastu.p, sizeof(lu), cudaMemcpyDeviceToHost, c->stream), "copy");
  CCK(cudaStreamSynchronize(c->stream), "sync");
  const int lastu = lu[0];
  const unsigned M = (unsigned)lu[1];
  const int ncoin = (int)Kc + (lastu ? 1 : 0);
  if ((size_t)ncoin + 1 > c->h_recs_cap) {
    if (c->h_recs) cudaFreeHost(c->h_recs);
    c->h_recs = nullptr;
    c->h_recs_cap = 0;
    const size_t cap = (size_t)ncoin + 1 + ncoin / 2;
    CCK(cudaMallocHost((void**)&c->h_recs, sizeof(pa_coinc_rec) * cap), "cudaMallocHost");
    c->h_recs_cap = cap;
  }
  if (Kc > 0) {
    ENS(wkeyA, sizeof(unsigned long long) * Kc);
    ENS(wkeyB, sizeof(unsigned long long) * Kc);
    ENS(cend, sizeof(unsigned) * Kc);
    ENS(cw, sizeof(unsigned) * Kc);
    ENS(cidxA, sizeof(unsigned) * Kc);
    ENS(cidxB, sizeof(unsigned) * Kc);
    {
      Span sp_(c, CK_GROUPS);
      k_compact_groups<<<(unsigned)gt, kT, 0, c->stream>>>(P<uint8_t>(c->gflag), G, P<unsigned>(c->blkcnt),
                                                          P<unsigned>(c->gend), P<unsigned>(c->gw),
                                                          P<unsigned long long>(c->wkeyA), P<unsigned>(c->cend),
                                                          P<unsigned>(c->cw), P<unsigned>(c->cidxA));
    }
    c->launches++;
    CCK(cudaGetLastError(), "k_compact_groups");
    // multiplicity descending, stable (coincidences.c:486)
    unsigned long long* wk = P<unsigned long long>(c->wkeyA);
    unsigned* order = P<unsigned>(c->cidxA);
    rc = radix_sort<unsigned long long>(c, wk, order, P<unsigned long long>(c->wkeyB), P<unsigned>(c->cidxB), Kc, 8);
    if (rc) return rc;
    // member offsets
    ENS(wsort, sizeof(unsigned) * (Kc + 1));
    ENS(scan_tmp, sizeof(unsigned) * scan_tmp_len(Kc + 1));
    {
      Span sp_(c, CK_MEANS);
      k_gather_w<<<(Kc + kT - 1) / kT, kT, 0, c->stream>>>(order, P<unsigned>(c->cw), (int)Kc, P<unsigned>(c->wsort));
    }
    c->launches++;
    CCK(cudaMemsetAsync(P<unsigned>(c->wsort) + Kc, 0, sizeof(unsigned), c->stream), "memset");
    rc = scan_excl(c, P<unsigned>(c->wsort), (long long)Kc + 1, P<unsigned>(c->scan_tmp));
    if (rc) return rc;
    ENS(means, sizeof(pa_coinc_rec) * Kc);
    ENS(fra, sizeof(int) * (M + 1));
    ENS(ops, sizeof(int) * (M + 1));
    {
      Span sp_(c, CK_MEANS);
      k_means<<<(Kc + kG - 1) / kG, kT, 0, c->stream>>>(c->ft, order, P<unsigned>(c->cend), P<unsigned>(c->cw),
                                                        P<unsigned>(c->wsort), (int)Kc, P<unsigned>(c->sval),
                                                        P<unsigned>(c->rawidx), P<double>(c->rec),
                                                        (double)c->cfg.N, c->cfg.refr, P<pa_coinc_rec>(c->means),
                                                        P<int>(c->fra), P<int>(c->ops));
    }
    c->launches++;
    CCK(cudaGetLastError(), "k_means");
    if ((size_t)M + 1 > c->h_mem_cap) {
      if (c->h_fra) cudaFreeHost(c->h_fra);
      if (c->h_ops) cudaFreeHost(c->h_ops);
      c->h_fra = c->h_ops = nullptr;
      c->h_mem_cap = 0;
      const size_t cap = (size_t)M + 1 + M / 2;
      CCK(cudaMallocHost((void**)&c->h_fra, sizeof(int) * cap), "cudaMallocHost");
      CCK(cudaMallocHost((void**)&c->h_ops, sizeof(int) * cap), "cudaMallocHost");
      c->h_mem_cap = cap;
    }
    CCK(cudaMemcpyAsync(c->h_recs, c->means.p, sizeof(pa_coinc_rec) * Kc, cudaMemcpyDeviceToHost, c->stream),
        "copy");
    if (M) {
      CCK(cudaMemcpyAsync(c->h_fra, c->fra.p, sizeof(int) * M, cudaMemcpyDeviceToHost, c->stream), "copy");
      CCK(cudaMemcpyAsync(c->h_ops, c->ops.p, sizeof(int) * M, cudaMemcpyDeviceToHost, c->stream), "copy");
    }
    // the device work ends here; what follows is host bookkeeping
    CCK(cudaEventRecord(c->ev1, c->stream), "cudaEventRecord");
    c->ev1_done = true;
    CCK(cudaStreamSynchronize(c->stream), "sync");
    c->sum.nmembers = M;
  }
  if (lastu) {
    // the last group is counted but never stored: a record of multiplicity
    // 0 whose means are 0/0 (coincidences.c:504-512), computed at run time
    volatile double zero = 0.0;
    pa_coinc_rec& r = c->h_recs[ncoin - 1];
    r.w = 0;
    r.first = (int)c->sum.nmembers;
    for (int l = 0; l < 4; l++) r.mean[l] = zero / zero;
    r.mean[4] = sqrt(zero);
  }
  c->sum.ncoin = ncoin;
  // coincidences.c:535-541: the largest multiplicity with the largest SNR
  c->sum.maxcoin = Kc > 0 ? c->h_recs[0].w : 0;
  c->sum.maxcoin_index = 0;
  double maxsnr = 0;
  for (int q = 0; q < ncoin; q++) {
    if (!q) maxsnr = c->h_recs[q].mean[4];
    if (c->h_recs[q].w == c->sum.maxcoin && c->h_recs[q].mean[4] > maxsnr) {
      maxsnr = c->h_recs[q].mean[4];
      c->sum.maxcoin_index = q;
    }
  }
  return PA_OK;
}

extern "C" {

int pa_coinc_run(pa_coinc* c, pa_coinc_summary* sum) {
  pa::TraceRange trace_("pa_coinc_run");
  if (!c) return PA_ERR_ARG;
  CCK(cudaSetDevice(c->cfg.device), "cudaSetDevice");
  const int nf = (int)c->frames.size();
  memset(&c->sum, 0, sizeof(c->sum));

  c->frameinfo.assign(3 * (size_t)nf, 0);
  c->sum.nframes = nf;
  c->sum.raw = c->nraw;
  c->n_in = 0;
  c->val_sorted = nullptr;
  c->ev1_done = false;
  CCK(cudaEventRecord(c->ev0, c->stream), "cudaEventRecord");
  // frame table
  memset(&c->ft, 0, sizeof(c->ft));
  c->ft.nframes = nf;
  int nblk1 = 0;
  for (int f = 0; f < nf; f++) {
    c->ft.frame_no[f] = c->frames[f];
    c->ft.raw_start[f] = (unsigned)c->raw_start[f];
    c->ft.blk_start[f] = nblk1;
    nblk1 += (int)((c->raw_start[f + 1] - c->raw_start[f] + kTile - 1) / kTile);
    c->frameinfo[3 * f] = c->frames[f];
  }
  c->ft.raw_start[nf] = (unsigned)c->nraw;
  c->ft.blk_start[nf] = nblk1;
  int rc = PA_OK;
  if (nblk1 > 0) {
    CellArgs a;
    // as order keys: x > lo with lo = +0 for a zero, x < hi with hi = -0; a
    // NaN is met by nothing
    auto key_of = [](double d, double zero, long long nan) {
      if (d != d) return nan;
      if (d == 0) d = zero;
      long long b;
      memcpy(&b, &d, sizeof(b));
      return order_key(b);
    };
    a.lo_k = key_of(M_PI_2 - c->cfg.narrowdown, 0.0, LLONG_MAX);
    a.hi_k = key_of(M_PI_2 + c->cfg.narrowdown, -0.0, LLONG_MIN);
    a.cut_k = key_of(c->cfg.snrcutoff, 0.0, LLONG_MAX);
    a.N = (double)c->cfg.N;
    a.N2 = 2.0 * a.N;
    a.sqrN = pow(c->cfg.N, 2);
    a.omsN = c->cfg.oms * c->cfg.N;
    volatile double epsm = PA_C_EPSMA;
    a.se = sin(epsm);
    a.ce = cos(epsm);
    for (int j = 0; j < 4; j++) {
      for (int i = 0; i < 4; i++) a.v[i][j] = c->cfg.vedva[i][j] / c->cfg.scale[j];
      a.half_shift[j] = 0.5 * c->cfg.shift[j];
    }
    a.refr = c->cfg.refr;
    a.se_f = (float)a.se;
    a.ce_f = (float)a.ce;
    auto split = [](double d, float* h, float* l) {
      *h = (float)d;
      *l = (float)(d - (double)*h);
    };
    a.fast = c->cfg.N < (1 << 24);
    for (int j = 0; j < 4; j++) {
      split(a.N * a.v[0][j], &a.f_h[j], &a.f_l[j]);
      split(a.sqrN * a.v[1][j], &a.d_h[j], &a.d_l[j]);
      a.hs_f[j] = (float)a.half_shift[j];  // exact: halves of digits
      a.s2_f[j] = (float)(a.omsN * a.v[2][j]);
      a.s3_f[j] = (float)(a.omsN * a.v[3][j]);
      // 2e-6 on be0 and be1, and for the fractions' FP32 sum 2e-6 and two
      // roundings (6e-8 each) of the shift
      const double m = fabs(a.omsN) * (fabs(a.v[2][j]) + fabs(a.v[3][j])) * 2e-6 + 2e-6 +
                       2.4e-7 * fabs(a.half_shift[j]);
      a.margin[j] = m < 1.0 ? (float)m : 1.0f;
    }
    ENS(cells_raw, sizeof(int4) * c->nraw);
    ENS(flag, c->nraw);
    ENS(snr_raw, sizeof(double) * c->nraw);
    ENS(blkcnt, sizeof(unsigned) * (nblk1 + 1));
    ENS(scan_tmp, sizeof(unsigned) * scan_tmp_len(nblk1 + 1));
    ENS(minmax, sizeof(int) * 9);
    const int mm0[9] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, INT_MIN, 0};
    CCK(cudaMemcpyAsync(c->minmax.p, mm0, sizeof(mm0), cudaMemcpyHostToDevice, c->stream), "copy");
    {
      Span sp_(c, CK_CELLS);
      k_cells<<<nblk1, kT, 0, c->stream>>>(c->ft, P<double>(c->rec), a, P<int4>(c->cells_raw), P<uint8_t>(c->flag),
                                          P<unsigned>(c->blkcnt), P<int>(c->minmax),
                                          (unsigned*)(P<int>(c->minmax) + 8), P<double>(c->snr_raw));
    }
    c->launches++;
    CCK(cudaGetLastError(), "k_cells");
    CCK(cudaMemsetAsync(P<unsigned>(c->blkcnt) + nblk1, 0, sizeof(unsigned), c->stream), "memset");
    rc = scan_excl(c, P<unsigned>(c->blkcnt), nblk1 + 1, P<unsigned>(c->scan_tmp));
    if (rc) return rc;
    std::vector<unsigned> boff(nblk1 + 1);
    int mm[9];
    CCK(cudaMemcpyAsync(boff.data(), c->blkcnt.p, sizeof(unsigned) * (nblk1 + 1), cudaMemcpyDeviceToHost, c->stream),
        "copy");
    CCK(cudaMemcpyAsync(mm, c->minmax.p, sizeof(mm), cudaMemcpyDeviceToHost, c->stream), "copy");
    CCK(cudaStreamSynchronize(c->stream), "sync");
    c->n_in = boff[nblk1];
    std::vector<long long> nin_f(nf);
    for (int f = 0; f < nf; f++) {
      c->ft.in_start[f] = boff[c->ft.blk_start[f]];
      nin_f[f] = (long long)boff[c->ft.blk_start[f + 1]] - boff[c->ft.blk_start[f]];
      c->frameinfo[3 * f + 1] = (int)nin_f[f];
    }
    c->ft.in_start[nf] = (unsigned)c->n_in;
    c->sum.inband = c->n_in;
    c->sum.fp64_cells = (unsigned)mm[8];
    if (c->n_in > 0) {
      ENS(rawidx, sizeof(unsigned) * c->n_in);
      ENS(cells_in, sizeof(int4) * c->n_in);
      KeyLayout L;
      int bits[4], tot = 0;
      for (int j = 0; j < 4; j++) {
        const unsigned long long range = (unsigned long long)((long long)mm[4 + j] - (long long)mm[j]);
        int b = 0;
        while (b < 63 && (range >> b)) b++;
        bits[j] = b;
        tot += b;
        L.maxc[j] = mm[4 + j];
      }
      // column 0 is the most significant
      int sh = tot;
      for (int j = 0; j < 4; j++) {
        sh -= bits[j];
        L.shift[j] = sh;
      }
      if (tot <= 64) {
        L.bits = tot;
        rc = run_keyed<unsigned long long>(c, L, nblk1, nin_f);
      } else {
        L.bits = 128;
        rc = run_keyed<U128>(c, L, nblk1, nin_f);
      }
      if (rc) return rc;
    }
  }
  if (!c->ev1_done) CCK(cudaEventRecord(c->ev1, c->stream), "cudaEventRecord");
  CCK(cudaEventSynchronize(c->ev1), "cudaEventSynchronize");
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  c->last_ms = ms;
  prof_collect(c);
  if (sum) *sum = c->sum;
  return PA_OK;
}

int pa_coinc_get(const pa_coinc* c, int* frameinfo, pa_coinc_rec* recs, int* fra, int* ops) {
  if (!c) return PA_ERR_ARG;
  if (frameinfo && !c->frameinfo.empty()) memcpy(frameinfo, c->frameinfo.data(), sizeof(int) * c->frameinfo.size());
  if (recs && c->sum.ncoin > 0) memcpy(recs, c->h_recs, sizeof(pa_coinc_rec) * c->sum.ncoin);
  if (fra && c->sum.nmembers > 0) memcpy(fra, c->h_fra, sizeof(int) * c->sum.nmembers);
  if (ops && c->sum.nmembers > 0) memcpy(ops, c->h_ops, sizeof(int) * c->sum.nmembers);
  return PA_OK;
}

int pa_coinc_cells(pa_coinc* c, int* cells, unsigned char* keep) {
  if (!c) return PA_ERR_ARG;
  if (c->n_in <= 0) return PA_OK;
  CCK(cudaSetDevice(c->cfg.device), "cudaSetDevice");
  if (cells)
    CCK(cudaMemcpyAsync(cells, c->cells_in.p, sizeof(int4) * c->n_in, cudaMemcpyDeviceToHost, c->stream), "copy");
  if (keep) {
    if (!c->val_sorted) return cfail(c, PA_ERR_ARG, "pa_coinc_cells: no completed run");
    // keep flags by in-band index, from those by sorted position
    int rc = ensure(c, c->keep_in, c->n_in);
    if (rc) return rc;
    k_keep_scatter<<<(unsigned)((c->n_in + kT - 1) / kT), kT, 0, c->stream>>>(P<uint8_t>(c->keep), c->val_sorted,
                                                                               c->n_in, P<uint8_t>(c->keep_in));
    c->launches++;
    CCK(cudaGetLastError(), "k_keep_scatter");
    CCK(cudaMemcpyAsync(keep, c->keep_in.p, c->n_in, cudaMemcpyDeviceToHost, c->stream), "copy");
  }
  CCK(cudaStreamSynchronize(c->stream), "sync");
  return PA_OK;
}

double pa_coinc_last_call_ms(const pa_coinc* c) { return c ? c->last_ms : 0.0; }

int pa_coinc_set_profiling(pa_coinc* c, int on) {
  if (!c) return PA_ERR_ARG;
  c->prof_on = on != 0;
  for (int k = 0; k < CK_COUNT; k++) {
    c->prof_ms[k] = 0;
    c->prof_n[k] = 0;
  }
  return PA_OK;
}

int pa_coinc_profile_get(const pa_coinc* c, int kind, const char** name, double* total_ms, long long* launches) {
  if (!c || kind < 0 || kind >= CK_COUNT) return PA_ERR_ARG;
  if (name) *name = kCoincKindName[kind];
  if (total_ms) *total_ms = c->prof_ms[kind];
  if (launches) *launches = c->prof_n[kind];
  return PA_OK;
}
long long pa_coinc_kernel_launches(const pa_coinc* c) { return c ? c->launches : 0; }

}  // extern "C"
