// pa_engine.h -- host-side interface between the C-ABI layer (pa_api.cu) and
// the templated device engines (pa_engine_f32.cu, pa_engine_f64.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pa {

// The FFT passes of the FP32 forms (pa_pair.cuh): L = 256 L2.
// log2 of the rows of a block of the intermediate
constexpr int pair_row_block(int logL) { return logL >= 19 ? 0 : (logL <= 16 ? 3 : 19 - logL); }
// radix of stage `stage` (0, 1, 2) of the row transforms; 1: no such stage
constexpr int pair_radix(int logL, int stage) {
  constexpr int r[9][3] = {{16, 1, 1}, {8, 1, 4}, {8, 1, 8}, {16, 1, 8}, {16, 1, 16},
                           {16, 1, 32}, {16, 8, 8}, {16, 16, 8}, {16, 16, 16}};
  return r[logL - 12][stage];
}
// entries of the row twiddle table: W_{Ns R}^{k r} at r Ns + k for the middle
// stage (if any), then for the last one
constexpr int pair_row_table(int logL) {
  return (pair_radix(logL, 1) > 1 ? pair_radix(logL, 0) * pair_radix(logL, 1) : 0) + (1 << (logL - 8));
}
// samples of room for N of data in a transform of length L: a warp of pass A
// reads four rows wherever the first of them has data
constexpr int pair_pad(int N, int L) { return (N + 4 * (L / 256) + 16 + 7) / 8 * 8; }
// exponent m of W_L^m at entry j of the inter-pass twiddle table: n2 k1 at the
// place of (k1, n2) in the intermediate
inline long pair_pass_exp(long j, int logL) {
  const int lr = pair_row_block(logL);
  const long k1 = (j & ((1L << lr) - 1)) + ((j >> (lr + logL - 8)) << lr);
  const long n2 = (j >> lr) & ((1L << (logL - 8)) - 1);
  return (n2 * k1) & ((1L << logL) - 1);
}
// exponent m of W_{L2}^m at entry j of the row twiddle table
inline long pair_row_exp(int j, int logL) {
  const long L2 = 1L << (logL - 8);
  const int mid = pair_row_table(logL) - (int)L2;
  const long n = j < mid ? mid : L2;                                       // Ns R
  const long Ns = j < mid ? pair_radix(logL, 0) : L2 / (pair_radix(logL, 2) > 1 ? pair_radix(logL, 2) : L2);
  const long q = j < mid ? j : j - mid;
  return (q / Ns) * (q % Ns) * (L2 / n) % L2;
}

constexpr int kMaxDet = 8;

// Per-context constants of one detector (uploaded once).
struct DetConst {
  double amod[9];
  double sig2, inv_sig2;
  double sphir, cphir;
  float amod_f[9], inv_sig2_f;  // FP32 copies (no per-thread conversions)
};

// Per-sky-point scalars, computed on the host in FP64 exactly as
// job_core() does (jobcore.c:243-299) and passed by value to the kernels.
struct SkyArgs {
  double het0;            // fmod(nn M8 + mm M12, M0)
  double oms;
  double sinal, cosal, sindel, cosdel;
  double nS[3];           // unit vector to the source
  double shft1[kMaxDet];  // nS . DetSSB[0..2] per detector
  double shft1_fma[kMaxDet];  // the same with fused multiply-adds (FP32 forms)
  double cosalfr[kMaxDet], sinalfr[kMaxDet];  // modvir rotated angles
  double s1_0;            // nn M9 + mm M13 (0 with --nospindown); over 2 pi
                          // in the fixed-point phase mode
  double M5;              // spindown step (0 with --nospindown); over 2 pi
                          // in the fixed-point phase mode
  double M0, M4;          // frequency step, het1 step
  // FP32 forms: the prelude and spindown phase terms as exact 64-bit
  // fixed-point turns of the FP64 values (turns_fixed)
  unsigned long long h0f; // het0 / 2 pi
  unsigned long long s1f; // s1_0 (already over 2 pi), fixed-point phase mode
  unsigned long long m5f; // M5 (already over 2 pi), fixed-point phase mode
  double oms_t;           // oms / 2 pi
  float cosalfr_f[kMaxDet], sinalfr_f[kMaxDet], cosdel_f, sindel_f;  // FP32 copies
  int ss_base;            // first spindown of the sky point (fixed-point form)
  int task;               // index of the sky point in the current batch
};

// One candidate found on the device (frequency bin ii is absolute).
struct DevCand {
  int task, ss, ii, pad;
  double F;
};

// FP64 form: the coefficients of the spline's elimination, p_i and invp_i = 2 /
// (p_{i-1} + 4), which settle to constants well before i = 63 (auxi.c:71-72).
inline void spline_pivots(double* invp, double* p) {
  p[0] = invp[0] = 0.;
  for (int i = 1; i < 64; i++) {
    invp[i] = 2. / (p[i - 1] + 4.);
    p[i] = -.5 * invp[i];
  }
}
// FP32 forms: sqrt(3) (sqrt(3) - 2)^j as float-float (k_resample).
constexpr int kSplineTaps = 16;
struct SplineTab {
  float ch[kSplineTaps + 1], cl[kSplineTaps + 1];
};
inline SplineTab spline_taps() {
  SplineTab t;
  double c = sqrt(3.);
  const double z = -1. / (2. + sqrt(3.));
  for (int j = 0; j <= kSplineTaps; j++, c *= z) {
    t.ch[j] = (float)c;
    t.cl[j] = (float)(c - (double)t.ch[j]);
  }
  return t;
}

// Device buffers owned by the context and shared with the engine.
struct Buffers {
  int N, nfft, Ninterp, nfftf, nmin, nmax, bins, nblk, nifo, fftpad;
  int NP;                           // FP32 forms: stride of xm's arrays (pair_pad)
  int sbatch;                       // spindowns per fused launch
  const double* xDat;               // [nifo][N]
  const double* DetSSB;             // [nifo][3N]
  const void* cosmodf;              // [N] Real
  const void* sinmodf;              // [N] Real
  const DetConst* dc;               // [nifo]
  const double* spline_invp;        // FP64 form: [64] pivots 2/(p+4) of the spline solve
  const double* spline_p;           // FP64 form: [64] p_i
  SplineTab spl;                    // FP32 forms: the spline's taps
  // FP64 form: arrays of double complex; FP32 forms: of pairs {a.re, b.re,
  // a.im, b.im} (float4)
  void* xin;                        // [nifo][2][N]; FP32: [nifo][N]
  void* spec;                       // [nifo][2][nfft]; FP32: [nifo][nfft]
  void* yint;                       // [nifo][2][Ninterp]; FP32: its odd points, [nifo][nfft]
  double* u;                        // FP64 form: [nifo][2][2N] double2
  void* y2;                         // FP64 form: [nifo][2][2N] double2
  double* shftf;                    // FP64 form: [nifo][N]
  // per-sky prelude outputs, double-buffered (slot 0/1) so that the prelude
  // of one sky point runs while the spindowns of the previous one read the
  // other slot
  void* ph0[2];                     // FP64 form: tmp1 [nifo][N]
  void* xm[2];                      // FP32 forms: [nifo][NP] float4 {a.re, b.re,
                                    // a.im, b.im}, then [nifo][NP] phase terms
                                    // (16 bytes in the fixed-point form, else
                                    // 8), zeros from N on; FP64 form:
                                    // [nifo][2][N] double complex
  double* sums[2];                  // aa, bb, 1/aa, 1/bb
  void* sums_r[2];                  // 1/aa, 1/bb in the working precision
  double* part;                     // partial sums of a^2, b^2
  void* ybuf_pre;                   // FFT intermediate of the prelude, nifo*2*Ninterp
  unsigned int* counter;            // CTA completion counter of the prelude (kept 0)
  void* ybuf;                       // FFT intermediate of the spindown loop, 2*lane_sb*2*nfftf
  void* F;                          // [2*lane_sb][bins] Real
  int lane_sb;                      // spindowns per lane of ybuf and F: lane 1 starts at
                                    // spindown lane_sb (two lanes run on two streams)
  DevCand* cand;
  int* ncand;
  int cand_cap;
  // twiddle tables (Real complex) per transform, FP64 form (FP32 forms: only
  // tw_inv[2] and [3])
  const void* tw_fwd[4];            // nfft forward: tw1, tw2, twlo, twhi
  const void* tw_inv[4];            // Ninterp backward (its twlo/twhi give e^{+i pi j/nfft})
  const void* tw_invh[4];           // nfft backward (the half-length resampling transform)
  const void* tw_main[4];           // nfftf forward
  // FP32 forms (all exp(-2 pi i ...)): W_256^m; the row twiddles and the
  // inter-pass twiddles of the transforms of length nfft (0) and nfftf (1)
  const void* pair_tw1;
  const void* pair_row[2];
  const void* pair_pass[2];
};

// Kernel kinds for the optional per-launch CUDA-event profile.
enum KernelKind {
  KK_PRELUDE_MOD = 0, KK_FFT_FWD_A, KK_FFT_FWD_B, KK_FFT_INV_A, KK_FFT_INV_B, KK_SPLINE_FWD, KK_SPLINE_BWD,
  KK_SPLINT, KK_SPIN_A, KK_SPIN_B, KK_THRESHOLD, KK_COUNT
};
const char* kernel_kind_name(int k);

// Event-bracketed launches recorded while profiling is on.
struct Prof {
  bool on = false;
  struct Rec {
    int kind, items;
    cudaEvent_t a, b;
  };
  Rec* recs = nullptr;
  int n = 0, cap = 0;
  double total_ms[KK_COUNT] = {0};
  long long launches[KK_COUNT] = {0};
  long long items[KK_COUNT] = {0};
};

class Engine {
 public:
  Prof* prof = nullptr;  // owned by the context
  virtual ~Engine() {}
  // Enqueues the per-sky prelude (jobcore.c:270-393) on `st`, outputs to
  // prelude slot `slot`.
  virtual cudaError_t prelude(const SkyArgs& sky, int slot, cudaStream_t st) = 0;
  // Enqueues spindowns ss0 .. ss0+nb-1 reading prelude slot `slot` into
  // lane `lane` of ybuf and F (lane 0: nb <= 2*lane_sb; lane 1, which starts
  // at spindown lane_sb of the buffers: nb <= lane_sb): phase modulation, FFT,
  // F-statistic, normalisation, threshold and candidate compaction.  Fdbg
  // (optional): normalised F of the batch, [nb][bins] Real.
  virtual cudaError_t spindowns(const SkyArgs& sky, int slot, int lane, int ss0, int nb, double trl, int white,
                                int s0_flag, cudaStream_t st, void* Fdbg) = 0;
  virtual long long launches() const = 0;
  virtual size_t real_size() const = 0;
  // Factor split of the FP64 form's spindown FFT (0: L1 = 2^ceil(m/2); 1:
  // swapped, for odd m only; ignored for even m).  The FP32 forms have one
  // factorisation and only keep the value.
  virtual void set_split(int split) = 0;
  virtual int split() const = 0;
  // Per-CTA trace of this engine's kernels into buf (cap records of 48
  // bytes: start/end %globaltimer, start/end clock64, kernel kind, SM id);
  // buf == nullptr switches it off.  trace_count: records written so far
  // (may exceed cap; the excess is dropped).
  virtual cudaError_t set_trace(void* buf, unsigned int cap) = 0;
  virtual cudaError_t trace_count(unsigned int* n) = 0;
};

// Factories (defined in the per-precision translation units).
Engine* make_engine_f32(const Buffers& b, int phase_mode);
Engine* make_engine_f32_fixed_at(void* mem, size_t bytes, const Buffers& b);
Engine* make_engine_f64(const Buffers& b);


}  // namespace pa
