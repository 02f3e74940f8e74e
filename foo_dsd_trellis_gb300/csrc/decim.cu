// DSD -> PCM decimation on sm_103a: the reference's FIR-only engine branch
// (src/engine.c:566-577; chain src/fir.c:523-611 with 63-tap half-band /2
// stages, ipp_downsample_d src/fir.c:467-487; gain ramp src/engine.c:879-889).
//
// Two forms:
//
// The whole chain at once (decim_mma_kernel).  All stages together are one
// filter h of 62 (D - 1) + 1 taps and a decimation by D, over +-1 inputs: with
// the inputs cut into blocks X[n] of B = max(D, 16), an output is
//   y[n] = sum_j sum_r h[B j - r] X[n - j][r]
// a matrix product with the taps on one side and decisions on the other.  The
// taps are rounded to fixed point (to 2^-55 of the largest up to D = 128, 2^-54
// at 256, 2^-53 at 512, where the last bit is 2^-61) and cut into seven 8-bit
// digits, which bf16 holds exactly; every partial sum is a whole number below
// 2^24, so the tensor cores' FP32 accumulators are exact, and the digits' sums
// are joined as 64-bit integers.  Only the taps' own rounding is left (an FP64
// evaluation rounds every sum as well).
// The rows of a product tile are the 16 values of j modulo 16, the four groups
// of j shift the columns, so that 16 (not 63) diagonals are left to add up.
// The decisions are expanded in shared memory to byte selectors (one PRMT makes
// two bf16 of two decisions; "no sample yet" selects zero), one 32-bit load a
// fragment; a warp uses each fragment for two digits, since making it (three
// half-rate integer instructions) takes as long as a product (mma.sync
// m16n8k16: 8.35 cycles a scheduler, measured).  What bounds it: the tensor
// pipe (active 60 % of the time, ncu; 448 multiply-adds an input decision),
// then the taps' loads from L2.  10 s of stereo DSD128 to 44.1 kHz, the whole
// call: 4,560 us stage by stage, 343 us here (7 warps of one digit over all
// columns 573, prmt by an intrinsic that masks its selector 577, one digit a
// warp over half the columns 430, taps loaded a step ahead 428, one CTA of 272
// outputs an SM 371).  Twelve 5-bit digits as e4m3 (exact too) took 609: an
// m16n8k32 product of that type takes 21 cycles a scheduler.
//
// The stages one by one, FP64, y[m] = sum_k h[k] x[2m - k] (the delay line of
// the previous call stands in for negative indices), each followed by a small
// launch that keeps the stage's last 62 consumed inputs.  A stage consumes
// floor(count / 2) * 2 inputs, as the reference's numIters = in_count /
// factor: a call whose length is not a multiple of D drops inputs at some
// stage, and what follows is no longer one filter over the decisions.  The
// next call's first outputs (those whose window reaches back over that point)
// and calls shorter than 128 B then take this form; so do FP64 inputs, captured
// calls, ragged streams up to the sizes of kRaggedFrom and one stage alone from
// kOneStageFrom.  IPP's
// summation order and use of FMA are not known, so the stages take the
// cheapest exact-enough form:
//   * the 63-tap half-band's taps at odd k other than the centre are the
//     design's zeros (|h| < 2e-17: they move an output by ~1e-17 of full scale), so
//     only the 32 even taps and the centre tap are applied;
//   * FP64 stages: those 33 taps as FMAs in ascending tap order;
//   * the first stage reads +-1 decisions: the 32 even taps form 4 groups of
//     8, each group's sum for every pattern of its 8 decisions is a table
//     entry (4 x 256 FP64 values, sums in tap order), so an output is 4 table
//     reads, the centre tap's +-h[31] and 4 adds.
// Either form differs from a tap-order sum of separately rounded products by
// at most a few FP64 ulps (float32 output within 2e-7 of full scale).
#include "api_context.h"
#include "fir_internal.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

using namespace dsdgpu;

namespace {

constexpr int kDecTaps = 63;

struct DecTaps {
  double h[kDecTaps];
};

// nonzero taps: even k and the centre
constexpr int kNzTaps = 33;
struct DecNz {
  double h[kNzTaps];
  int k[kNzTaps];
};

constexpr int kLutGroups = 4;   // 32 even taps in groups of 8

// FP64 stage: the 33 nonzero taps as FMAs in ascending tap order
// (done: nothing is left to do where it is set, see to_lines)
__global__ void decim_stage_kernel(const __grid_constant__ DecNz T, const double* __restrict__ in,
                                   size_t in_stride, long long m_out,
                                   const double* __restrict__ dly, double* __restrict__ out,
                                   size_t out_stride, int nch, const int* __restrict__ done) {
  if (done && *done) return;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m_out * nch) return;
  const long long c = i / m_out, m = i % m_out;
  const double* dl = dly + (size_t)c * (kDecTaps - 1);
  const double* xc = in + (size_t)c * in_stride;
  double acc = 0.0;
#pragma unroll
  for (int q = 0; q < kNzTaps; q++) {
    const long long j = 2 * m - T.k[q];
    const double x = j >= 0 ? xc[j] : dl[kDecTaps - 1 + j];
    acc = __fma_rn(T.h[q], x, acc);
  }
  out[(size_t)c * out_stride + m] = acc;
}

// first stage, decision bytes in: 4 group-table reads + the centre tap
__global__ void __launch_bounds__(256) decim_bits_kernel(const __grid_constant__ DecNz T,
                                                         const double* __restrict__ lut, double h31,
                                                         const uint8_t* __restrict__ bits,
                                                         size_t in_stride, long long m_out,
                                                         const double* __restrict__ dly,
                                                         double* __restrict__ out,
                                                         size_t out_stride, int nch,
                                                         const int* __restrict__ done) {
  __shared__ double tab[kLutGroups * 256];
  if (done && *done) return;
  for (int q = threadIdx.x; q < kLutGroups * 256; q += blockDim.x) tab[q] = lut[q];
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m_out * nch) return;
  const long long c = i / m_out, m = i % m_out;
  const double* dl = dly + (size_t)c * (kDecTaps - 1);
  const uint8_t* bc = bits + (size_t)c * in_stride;
  double acc = 0.0;
  if (2 * m < kDecTaps - 1) {
    // the window reaches the delay line, whose values are zero before the
    // first call: the 33 taps directly
#pragma unroll
    for (int q = 0; q < kNzTaps; q++) {
      const long long j = 2 * m - T.k[q];
      const double x = j >= 0 ? (bc[j] & 1u ? 1.0 : -1.0) : dl[kDecTaps - 1 + j];
      acc = __fma_rn(T.h[q], x, acc);
    }
  } else {
#pragma unroll
    for (int g = 0; g < kLutGroups; g++) {
      unsigned p = 0;
#pragma unroll
      for (int u = 0; u < 8; u++) p |= (unsigned)(bc[2 * m - 16 * g - 2 * u] & 1u) << u;
      acc = __dadd_rn(acc, tab[g * 256 + p]);
    }
    acc = __dadd_rn(acc, (bc[2 * m - 31] & 1u) ? h31 : -h31);
  }
  out[(size_t)c * out_stride + m] = acc;
}

// delay line <- the last 62 consumed inputs of (delay line ++ stage input)
template <bool kBits>
__global__ void decim_dly_kernel(const uint8_t* __restrict__ bits, const double* __restrict__ in,
                                 size_t in_stride, long long used, double* __restrict__ dly,
                                 int nch, const int* __restrict__ done) {
  const int c = blockIdx.x;
  if (c >= nch || (done && *done)) return;
  __shared__ double tmp[kDecTaps - 1];
  double* dl = dly + (size_t)c * (kDecTaps - 1);
  for (int k = threadIdx.x; k < kDecTaps - 1; k += blockDim.x) {
    const long long j = used - (kDecTaps - 1) + k;
    double v;
    if (j >= 0) v = kBits ? (bits[(size_t)c * in_stride + j] ? 1.0 : -1.0) : in[(size_t)c * in_stride + j];
    else v = dl[kDecTaps - 1 + j];
    tmp[k] = v;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kDecTaps - 1; k += blockDim.x) dl[k] = tmp[k];
}

// the delay lines at rest, unless `done`; and `done` itself
__global__ void decim_rest_kernel(double* __restrict__ dly, int n, const int* __restrict__ done) {
  if (*done) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dly[i] = 0.0;
}
__global__ void decim_done_kernel(int* done) { *done = 1; }

__global__ void decim_gain_kernel(const double* __restrict__ y, size_t y_stride, long long n,
                                  int nch, double g_start, double g_step, int apply,
                                  float* __restrict__ out, size_t out_stride) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * nch) return;
  const long long c = i / n, t = i % n;
  double v = y[(size_t)c * y_stride + t];
  if (apply) v = __dmul_rn(v, __dadd_rn(g_start, __dmul_rn(g_step, (double)t)));
  out[(size_t)c * out_stride + t] = (float)v;
}

// FP64 output of the rate-conversion branch (src/engine.c:640-717): gain ramp
// (when either end differs from 1), then the optional soft clip
__global__ void decim_gain_f64_kernel(const double* __restrict__ y, size_t y_stride, long long n,
                                      int nch, double g_start, double g_step, int apply,
                                      int soft_clip, double* __restrict__ out, size_t out_stride) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * nch) return;
  const long long c = i / n, t = i % n;
  double v = y[(size_t)c * y_stride + t];
  if (apply) v = __dmul_rn(v, __dadd_rn(g_start, __dmul_rn(g_step, (double)t)));
  if (soft_clip) v = soft_clip_095(v);
  out[(size_t)c * out_stride + t] = v;
}

// ---- the whole chain as one matrix product ----
constexpr int kMmaDigits = 7;          // 8-bit digits of a tap
constexpr int kMmaParts = 3;           // a warp: two digits over a third of the columns
constexpr int kMmaWarps = (kMmaDigits + 1) / 2 * kMmaParts;
constexpr int kMmaCols = 128;          // output blocks of a CTA
constexpr int kMmaAcc = kMmaCols + 16; // product columns: 16 diagonals end in every output
constexpr int kAccRow = kMmaAcc + 4;   // row of the product tile in shared memory

struct MmaPlan {
  int B;        // inputs a block
  int F;        // outputs a block (1, or 16 / D below D = 16)
  int T;        // groups of 16 lags
  int shift;    // taps are integers over 2^shift
};

// One DoP float's 16 decisions: round(f * 2^23) half away from zero, low 16
// bits (dop_unpack_kernel's FP64 expression; f * 2^23 is exact in FP32, and
// below 2^23 its fraction too).
__device__ __forceinline__ unsigned dop_word(float f) {
  const float y = f * 8388608.0f;
  int v = __float2int_rz(y);
  if (fabsf(y) < 8388608.0f) {
    const float fr = y - (float)v;
    if (fr >= 0.5f) v++;
    else if (fr <= -0.5f) v--;
  }
  return (unsigned)v & 0xffffu;
}

// Byte selectors (PRMT) out of 0x00BF3F80: bf16 +1 = 3F80, -1 = BF80, none = 0.
constexpr unsigned kPool = 0x00bf3f80u;
constexpr unsigned kSelNone = 0x33333333u;
// Selectors of lane c: decisions 2c, 2c+1 (low half) and 2c+8, 2c+9 of a word
// whose bit k is decision k: bit 4 of bytes 0 .. 3, taken from 2 (-1) to 1 (+1).
__device__ __forceinline__ unsigned sel4(unsigned wr, int c) {
  const unsigned x = (wr << 4) >> (2 * c), y = (wr << 3) >> (2 * c);
  return 0x20202020u - (__byte_perm(x, y, 0x5140) & 0x10101010u);
}

// two bf16 by the selector's low half (prmt's plain mode: nibbles 0 .. 3)
__device__ __forceinline__ unsigned two(unsigned sel) {
  unsigned r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(kPool), "r"(sel));
  return r;
}

struct MmaIn {
  const float* dop;        // DoP frames (kDop) or decision bytes
  const uint8_t* bits;
  size_t stride;
  long long count;         // decisions of this call
  const uint8_t* tail;     // decisions before it, newest last, tail_len of them (nullptr: none)
  int tail_len;
  size_t tail_stride;
};

// decision `i` of the stream: 0, 1, or 2 for none
template <bool kDop>
__device__ __forceinline__ unsigned decision(const MmaIn& I, int c, long long i) {
  if (i < 0) {
    const long long k = i + I.tail_len;
    return k >= 0 ? I.tail[(size_t)c * I.tail_stride + k] : 2u;
  }
  if (i >= I.count) return 2u;
  if (kDop) return (dop_word(I.dop[(size_t)c * I.stride + (i >> 4)]) >> (15 - (int)(i & 15))) & 1u;
  return I.bits[(size_t)c * I.stride + i] & 1u;
}

// One warp's products: ND digits (16 rows each) by kN products of 8 columns,
// over all steps, left in the digits' tiles in shared memory.
constexpr int kN = kMmaAcc / 8 / kMmaParts;
template <int ND>
__device__ __forceinline__ void mma_tile(const uint4* __restrict__ A, int steps, int KS, int pitch,
                                         const unsigned* sb, float* tile) {
  float acc[ND][kN][4];
#pragma unroll
  for (int k = 0; k < ND; k++)
#pragma unroll
    for (int n = 0; n < kN; n++)
#pragma unroll
      for (int r = 0; r < 4; r++) acc[k][n][r] = 0.0f;
  const size_t digit = (size_t)steps * 32;
  for (int t = steps / KS; t > 0; t--, sb -= 64) {   // the next 16 lags: 16 columns back
    const unsigned* col = sb;
#pragma unroll 4
    for (int ks = 0; ks < KS; ks++, col += pitch, A += 32) {
      uint4 a[ND];
#pragma unroll
      for (int k = 0; k < ND; k++) a[k] = A[k * digit];
      unsigned sel[kN];
#pragma unroll
      for (int n = 0; n < kN; n++) sel[n] = col[32 * n];
#pragma unroll
      for (int n = 0; n < kN; n++) {
        const unsigned b0 = two(sel[n]), b1 = two(sel[n] >> 16);
#pragma unroll
        for (int k = 0; k < ND; k++)
          asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
              "{%8,%9}, {%0,%1,%2,%3};"
              : "+f"(acc[k][n][0]), "+f"(acc[k][n][1]), "+f"(acc[k][n][2]), "+f"(acc[k][n][3])
              : "r"(a[k].x), "r"(a[k].y), "r"(a[k].z), "r"(a[k].w), "r"(b0), "r"(b1));
      }
    }
  }
#pragma unroll
  for (int k = 0; k < ND; k++)
#pragma unroll
    for (int n = 0; n < kN; n++) {
      float* p = tile + k * 16 * kAccRow + 8 * n;
      *reinterpret_cast<float2*>(p) = make_float2(acc[k][n][0], acc[k][n][1]);
      *reinterpret_cast<float2*>(p + 8 * kAccRow) = make_float2(acc[k][n][2], acc[k][n][3]);
    }
}

template <bool kDop>
__global__ void __launch_bounds__(32 * kMmaWarps, 2)
decim_mma_kernel(const MmaPlan M, const MmaIn I, const uint4* __restrict__ taps, int col_first,
                 unsigned col_tiles, unsigned per_ch, long long n_out, double scale, double g_start, double g_step,
                 int apply, float* __restrict__ out, size_t out_stride,
                 uint8_t* __restrict__ new_tail, int keep, long long total) {
  extern __shared__ __align__(16) unsigned mma_smem[];
  const int c = (int)(blockIdx.x / per_ch);
  const unsigned bx = blockIdx.x - (unsigned)c * per_ch;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (bx >= col_tiles) {
    // the decisions the next call looks back to: the last `keep` of (tail ++ input)
    const int part = (int)(bx - col_tiles), parts = (int)(per_ch - col_tiles);
    for (int k = part * (int)blockDim.x + tid; k < keep; k += parts * (int)blockDim.x)
      new_tail[(size_t)c * I.tail_stride + k] =
          (uint8_t)decision<kDop>(I, c, total - keep + k - I.tail_len);
    return;
  }
  const int ksh = 31 - __clz(M.B >> 4);          // 16-decision steps of a block: 2^ksh
  const int KS = 1 << ksh;
  const long long n0 = col_first + (long long)bx * kMmaCols;
  const int cols = kMmaCols + 16 * M.T;          // columns n0 - 16 T .. n0 + 127
  // selectors as [step][column][4 lanes]: a fragment is 32 consecutive words,
  // and the columns of the next product lie at a fixed distance; a step's rows
  // are 16 bytes further than whole, so that the words of one column (written
  // by neighbouring threads) fall on different banks
  const int pitch = 4 * cols + 4;
  const long long i0 = (n0 - 16 * M.T) * M.B;
  constexpr int kLoads = 4;                      // words of a thread on their way at once
  for (int k0 = tid; k0 < cols * KS; k0 += kLoads * 32 * kMmaWarps) {
    unsigned w[kLoads], none[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; u++) {
      const int k = k0 + u * 32 * kMmaWarps;
      const long long i = i0 + 16ll * k;
      w[u] = none[u] = 0u;
      if (k >= cols * KS) continue;
      if (kDop && i >= 0 && i + 16 <= I.count)
        w[u] = __float_as_uint(I.dop[(size_t)c * I.stride + (i >> 4)]);
    }
#pragma unroll
    for (int u = 0; u < kLoads; u++) {
      const int k = k0 + u * 32 * kMmaWarps;
      const long long i = i0 + 16ll * k;
      if (k >= cols * KS) continue;
      unsigned wr = 0u;                          // bit b: decision b of the word
      if (i >= 0 && i + 16 <= I.count) {
        if (kDop) {
          wr = __brev(dop_word(__uint_as_float(w[u]))) >> 16;
        } else {
          const uint8_t* b = I.bits + (size_t)c * I.stride + i;
#pragma unroll
          for (int e = 0; e < 16; e++) wr |= (unsigned)(b[e] & 1u) << e;
        }
      } else {
        for (int e = 0; e < 16; e++) {
          const unsigned d = decision<kDop>(I, c, i + e);
          wr |= (d & 1u) << e;
          none[u] |= (d >> 1) << e;
        }
      }
      uint4 sel = make_uint4(sel4(wr, 0), sel4(wr, 1), sel4(wr, 2), sel4(wr, 3));
      if (none[u]) {
        auto blank = [&](unsigned v, int q) {    // bytes of the decisions that are not there
          const unsigned m = ((none[u] << 4) >> (2 * q)), o = ((none[u] << 3) >> (2 * q));
          const unsigned at = (__byte_perm(m, o, 0x5140) & 0x10101010u) >> 4;
          return (v & ~(at * 0xffu)) | (kSelNone & (at * 0xffu));
        };
        sel = make_uint4(blank(sel.x, 0), blank(sel.y, 1), blank(sel.z, 2), blank(sel.w, 3));
      }
      *reinterpret_cast<uint4*>(&mma_smem[(k & (KS - 1)) * pitch + 4 * (k >> ksh)]) = sel;
    }
  }
  __syncthreads();
  // product tiles: two digits of one output phase over a third of the columns
  // a warp (the decisions' fragments cost as much as a product, so each serves
  // two; the last pair has one digit)
  const int dg = 2 * (warp / kMmaParts), part = warp % kMmaParts;
  const int steps = M.T * KS;
  // the tiles lie behind the selectors, which further phases still read
  float* const tiles = reinterpret_cast<float*>(mma_smem + KS * pitch);
  int* const sums = reinterpret_cast<int*>(tiles + kMmaDigits * 16 * kAccRow);
  for (int ph = 0; ph < M.F; ph++) {
    const uint4* A = taps + ((size_t)(ph * kMmaDigits + dg) * steps) * 32 + lane;
    const unsigned* sb = mma_smem + 64 * (M.T - 1) + 32 * kN * part + lane;
    float* tile = tiles + dg * 16 * kAccRow + (lane >> 2) * kAccRow + 8 * kN * part + 2 * (lane & 3);
    if (dg + 1 < kMmaDigits) mma_tile<2>(A, steps, KS, pitch, sb, tile);
    else mma_tile<1>(A, steps, KS, pitch, sb, tile);
    __syncthreads();
    for (int k = tid; k < kMmaDigits * kMmaCols; k += 32 * kMmaWarps) {
      const int at = k % kMmaCols;
      const float* tile = tiles + k / kMmaCols * 16 * kAccRow;
      float y = 0.0f;
#pragma unroll
      for (int i = 0; i < 16; i++) y += tile[i * kAccRow + 16 + at - i];
      sums[k] = (int)y;
    }
    __syncthreads();
    if (tid < kMmaCols) {
      const long long m = (n0 + tid) * M.F + ph;
      if (m < n_out) {
        long long y = 0;
#pragma unroll
        for (int k = 0; k < kMmaDigits; k++) y += (long long)sums[k * kMmaCols + tid] << (8 * k);
        double v = __dmul_rn((double)y, scale);
        if (apply) v = __dmul_rn(v, __dadd_rn(g_start, __dmul_rn(g_step, (double)m)));
        out[(size_t)c * out_stride + m] = (float)v;
      }
    }
    if (ph + 1 < M.F) __syncthreads();
  }
}

__host__ size_t mma_smem_bytes(const MmaPlan& M) {
  return sizeof(unsigned) * (size_t)(M.B >> 4) * (4 * (kMmaCols + 16 * M.T) + 4) +
         sizeof(float) * (size_t)kMmaDigits * 16 * kAccRow + sizeof(int) * kMmaDigits * kMmaCols;
}

// The plan of `stages` stages (all but its shift, which the taps' peak decides).
int mma_len(int stages) { return 62 * ((1 << stages) - 1) + 1; }
size_t mma_words(const MmaPlan& M) { return (size_t)M.F * kMmaDigits * M.T * (M.B / 16) * 32 * 4; }
MmaPlan mma_plan(int stages) {
  const int D = 1 << stages;
  MmaPlan M{};
  M.B = D < 16 ? 16 : D;
  M.F = M.B / D;
  const int J = (mma_len(stages) - 1 + M.B - 1) / M.B + 1;
  M.T = (J + 15) / 16;
  return M;
}

// The plan's taps, formed on the device: on the host they took 1.8 ms of a
// setup at ratio 512.  One stage's taps, `gap` inputs apart, times the response
// of the stages before it, h of `len` taps (nullptr: the unit impulse):
__global__ void decim_conv_kernel(const __grid_constant__ DecNz T, const double* __restrict__ h, int len,
                                  int gap, double* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= len + 62 * gap) return;
  double acc = 0.0;
  for (int q = kNzTaps - 1; q >= 0; q--) {
    const int i = j - T.k[q] * gap;
    if (i >= 0 && i < len) acc = __dadd_rn(acc, __dmul_rn(h ? h[i] : 1.0, T.h[q]));
  }
  out[j] = acc;
}

__global__ void __launch_bounds__(1024) decim_peak_kernel(const double* __restrict__ h, int len,
                                                          double* __restrict__ peak) {
  __shared__ double part[32];
  double m = 0.0;
  for (int i = threadIdx.x; i < len; i += blockDim.x) m = fmax(m, fabs(h[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = part[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) *peak = m;
  }
}

// the taps in the order of the A fragments:
// [phase][digit][16-lag group][step][lane][4 registers of two bf16]
__global__ void decim_frag_kernel(const MmaPlan M, int D, const double* __restrict__ h, int len, double one,
                                  unsigned* __restrict__ out, int words) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= words) return;
  const int r = w & 3, lane = (w >> 2) & 31, KS = M.B / 16;
  int at = w >> 7;
  const int ks = at % KS;
  at /= KS;
  const int t = at % M.T;
  at /= M.T;
  const int k = at % kMmaDigits, ph = at / kMmaDigits;
  const int row = lane / 4 + (r & 1) * 8;
  unsigned word = 0;
  for (int e = 0; e < 2; e++) {
    const int kk = 2 * (lane % 4) + e + (r >> 1) * 8;
    const int tap = D * ph + M.B * (16 * t + row) - (16 * ks + kk);
    if (tap < 0 || tap >= len) continue;
    long long v = __double2ll_rn(h[tap] * one);   // the product is exact
    int d = 0;
    for (int i = 0; i <= k; i++) {                // balanced digits, -128 .. 127
      d = (int)(signed char)(v & 255);
      v = (v - d) >> 8;
    }
    word |= (__float_as_uint((float)d) >> 16) << (16 * e);   // bf16: exact
  }
  out[w] = word;
}

unsigned nb(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

struct dsdgpu_decim_state {
  int stages = 0;
  int nch = 0;
  DecTaps taps{};
  DecNz nz{};
  double* d_lut = nullptr;      // [group][pattern] sums of the first stage
  double* d_dly = nullptr;      // [stage][nch][62]
  double* d_buf = nullptr;      // ping-pong [2][nch][row]
  size_t row = 0;
  // the whole-chain form: its plan, taps, and the decisions before the next
  // call (two buffers in turn)
  MmaPlan mma{};
  uint4* d_taps = nullptr;
  uint8_t* d_tail = nullptr;    // [2][nch][tail_cap]
  int tail_cap = 0, tail_len = 0, tail_buf = 0;
  // what the next call continues from: nothing yet, the decisions in the tail
  // (`ragged`: their last call's length was not whole blocks), or the stages'
  // delay lines
  enum { kFresh, kTail, kLines } from = kFresh;
  bool ragged = false;
  // Calls captured into a graph run later and more than once, so they may not
  // rest on what the host knows of the stream: from the first one on, every
  // call takes the stages, whose whole state is the delay lines, and a device
  // word says whether these are valid yet (see to_lines).
  bool on_device = false;
  bool capturing = false;       // this call is captured
  int* d_done = nullptr;
  bool buf_in_graph = false;    // a captured call has named d_buf
  std::vector<double*> old_bufs;
  uint8_t* tail() const { return d_tail + (size_t)tail_buf * nch * tail_cap; }
  ~dsdgpu_decim_state() {
    if (d_done) cudaFree(d_done);
    if (d_taps) cudaFree(d_taps);
    if (d_tail) cudaFree(d_tail);
    if (d_lut) cudaFree(d_lut);
    if (d_dly) cudaFree(d_dly);
    if (d_buf) cudaFree(d_buf);
    for (double* b : old_bufs) cudaFree(b);
  }
};

void decim_free(dsdgpu_decim_state* s) { delete s; }

// The FP64 chain from fresh state without a context (the batch plan's DSD
// input to a lower rate): `stages` 63-tap half-band /2 stages over `count`
// inputs through the ping-pong rows of `buf` (2 x nch rows of `row` doubles,
// row >= count / 2 + 1), with the zero delay lines `zero_dly` (nch x 62
// zeros, read only: a fresh stream has nothing before its first sample), then
// gain and the optional soft clip into `out`.  *out_count = count >> stages.
// out32 non-null: FP32 output instead (the gain, no clip, narrowed to
// nearest: the PreCorr walk's input), `out` unused.
int launch_decim_f64_fresh(const double* in, size_t in_stride, long long count, int stages,
                           int nch, double* buf, size_t row, const double* zero_dly,
                           double g_start, double g_step, int apply, int soft_clip, double* out,
                           size_t out_stride, cudaStream_t st, float* out32) {
  if (count < 2 || stages < 1) return 0;
  DecTaps taps{};
  DecNz nz{};
  design_taps(kDecTaps, false, taps.h);
  for (int q = 0, k = 0; k < kDecTaps; k++)
    if ((k & 1) == 0 || k == kDecTaps / 2) { nz.h[q] = taps.h[k]; nz.k[q] = k; q++; }
  double* pp[2] = {buf, buf + row * (size_t)nch};
  long long cur = count;
  const double* x = in;
  size_t xs = in_stride;
  for (int k = 0; k < stages; k++) {
    const long long m = cur / 2;
    if (m > 0)
      decim_stage_kernel<<<nb(m * nch, 256), 256, 0, st>>>(nz, x, xs, m, zero_dly, pp[k & 1], row,
                                                           nch, nullptr);
    x = pp[k & 1];
    xs = row;
    cur = m;
  }
  if (cur > 0 && out32)
    decim_gain_kernel<<<nb(cur * nch, 256), 256, 0, st>>>(x, xs, cur, nch, g_start, g_step, apply,
                                                          out32, out_stride);
  else if (cur > 0)
    decim_gain_f64_kernel<<<nb(cur * nch, 256), 256, 0, st>>>(x, xs, cur, nch, g_start, g_step,
                                                              apply, soft_clip ? 1 : 0, out,
                                                              out_stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

namespace {

// The stages' rows.  Calls that took the product have not allocated them, so the
// first captured call may have to: allowed in this thread's relaxed mode.  Rows
// that a graph may name, or that a captured call outgrows, are kept until the
// state goes.
int ensure_rows(dsdgpu_context_t* c, dsdgpu_decim_state* s, size_t count) {
  const size_t row = ((count / 2 + 1) + 31) & ~(size_t)31;
  if (s->row >= row) {
    s->buf_in_graph |= s->capturing;
    return DSDGPU_OK;
  }
  if (s->d_buf && (s->buf_in_graph || s->capturing)) s->old_bufs.push_back(s->d_buf);
  else if (s->d_buf) cudaFree(s->d_buf);
  s->d_buf = nullptr;
  s->row = 0;
  s->buf_in_graph = s->capturing;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  const cudaError_t e = cudaMalloc(&s->d_buf, sizeof(double) * 2 * row * (size_t)s->nch);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return c->cuda_fail(e, "decimation buffers");
  }
  s->row = row;
  return DSDGPU_OK;
}

// The whole-chain form's taps in s->d_taps, and the plan's shift.
int form_taps(dsdgpu_context_t* c, dsdgpu_decim_state* s) {
  const int len = mma_len(s->stages), words = (int)mma_words(s->mma);
  const int rc = c->ensure_scratch(sizeof(double) * (2 * (size_t)len + 1));
  if (rc) return rc;
  double* buf[2] = {(double*)c->d_scratch, (double*)c->d_scratch + len};
  double* d_peak = buf[1] + len;
  const double* h = nullptr;
  for (int k = 0; k < s->stages; k++) {
    const int n = mma_len(k + 1);
    decim_conv_kernel<<<nb(n, 128), 128, 0, c->stream>>>(s->nz, h, mma_len(k), 1 << k, buf[k & 1]);
    h = buf[k & 1];
  }
  decim_peak_kernel<<<1, 1024, 0, c->stream>>>(h, len, d_peak);
  double peak = 0.0;
  cudaMemcpyAsync(&peak, d_peak, sizeof peak, cudaMemcpyDeviceToHost, c->stream);
  const cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->cuda_fail(e, "decimation taps");
  // a tap stays below 2^54 (seven digits), and with at most 61 the joined sum
  // below 1.9 x 2^61, a bit within 64 (sum |h| < 1.9 at every ratio)
  s->mma.shift = 61;
  while (std::ldexp(peak, s->mma.shift) > std::ldexp(1.0, 54)) s->mma.shift--;
  decim_frag_kernel<<<nb(words, 256), 256, 0, c->stream>>>(s->mma, 1 << s->stages, h, len,
                                                           std::ldexp(1.0, s->mma.shift), (unsigned*)s->d_taps,
                                                           words);
  c->launches += s->stages + 2;
  return DSDGPU_OK;
}

// `count` decisions through the stages and their delay lines; the last
// stage's outputs in *y (rows of s->row), *m of them.  Nothing where *done is set.
int staged(dsdgpu_context_t* c, dsdgpu_decim_state* s, const uint8_t* d_bits, size_t bits_stride,
           size_t count, const double** y, size_t* m_out, const int* done = nullptr) {
  const int nch = s->nch;
  cudaStream_t st = c->stream;
  const int rc = ensure_rows(c, s, count);
  if (rc) return rc;
  double* buf[2] = {s->d_buf, s->d_buf + s->row * (size_t)nch};
  size_t cur = count;
  const double* in = nullptr;
  for (int k = 0; k < s->stages; k++) {
    const long long m = (long long)(cur / 2);
    double* out = buf[k & 1];
    double* dly = s->d_dly + (size_t)k * nch * (kDecTaps - 1);
    if (m > 0) {
      if (k == 0) {
        decim_bits_kernel<<<nb(m * nch, 256), 256, 0, st>>>(s->nz, s->d_lut, s->taps.h[kDecTaps / 2], d_bits,
                                                            bits_stride, m, dly, out, s->row, nch, done);
        decim_dly_kernel<true><<<nch, 64, 0, st>>>(d_bits, nullptr, bits_stride, 2 * m, dly, nch, done);
      } else {
        decim_stage_kernel<<<nb(m * nch, 256), 256, 0, st>>>(s->nz, in, s->row, m, dly, out, s->row,
                                                             nch, done);
        decim_dly_kernel<false><<<nch, 64, 0, st>>>(nullptr, in, s->row, 2 * m, dly, nch, done);
      }
      c->launches += 2;
    }
    in = out;
    cur = (size_t)m;
  }
  *y = in;
  *m_out = cur;
  return DSDGPU_OK;
}

// Whether this call is captured; from then on the stream's state is on the device.
void look_for_capture(dsdgpu_context_t* c, dsdgpu_decim_state* s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(c->stream, &cap);
  s->capturing = cap != cudaStreamCaptureStatusNone;
  if (s->capturing) s->on_device = true;
}

// The stages' delay lines as the calls so far leave them: zero at a stream's
// start, else the stages run over the tail from rest.  The tail starts on a
// whole block and is 64 blocks long (or the whole stream), which is longer
// than any line's window, so its last values are the same as in one run.
// A captured call carries these launches into its graph, and they have to run
// once, whichever of the graph's replays and of the calls after it comes first:
// they look at *d_done, which the first of them sets.
int to_lines(dsdgpu_context_t* c, dsdgpu_decim_state* s) {
  if (s->from == dsdgpu_decim_state::kLines) return DSDGPU_OK;
  const int lines = s->stages * s->nch * (kDecTaps - 1);
  const int* done = s->on_device ? s->d_done : nullptr;
  if (done) {
    decim_rest_kernel<<<std::min(nb(lines, 256), 64u), 256, 0, c->stream>>>(s->d_dly, lines, done);
    c->launches++;
  } else {
    cudaMemsetAsync(s->d_dly, 0, sizeof(double) * (size_t)lines, c->stream);
  }
  if (s->from == dsdgpu_decim_state::kTail && s->tail_len > 0) {
    const double* y = nullptr;
    size_t m = 0;
    const int rc = staged(c, s, s->tail(), (size_t)s->tail_cap, (size_t)s->tail_len, &y, &m, done);
    if (rc) return rc;
  }
  if (done) {
    decim_done_kernel<<<1, 1, 0, c->stream>>>(s->d_done);
    c->launches++;
  }
  if (s->capturing) return DSDGPU_OK;   // as far as the host knows, it has not run
  s->from = dsdgpu_decim_state::kLines;
  s->ragged = false;
  s->tail_len = 0;
  return DSDGPU_OK;
}

}  // namespace

// Decisions of a call (over all channels) from which the product pays though it
// costs more launches than the stages, by the number of stages: a ragged call of
// a stream whose last one was ragged too, which would run the tail through the
// stages (a launch costs 4.9 us here) to get the first outputs.  Measured, calls
// of one length, 1 / 2 / 6 channels alike, us by stages alone / with the
// product: 4 stages 1.0 M decisions 95 / 110, 2.0 M 129 / 117; 7 stages 20 k
// 94 / 168, 2.5 M 184 / 186, 4.0 M 234 / 185; 9 stages 4.0 M 254 / 250.
constexpr double kRaggedFrom[] = {0, 0.5e6, 4.0e6, 2.0e6, 1.8e6, 2.0e6, 2.2e6, 2.6e6, 3.1e6, 4.0e6};
static_assert(sizeof kRaggedFrom / sizeof(double) == kMaxStages + 1, "one for every number of stages");
// One stage (a product tile for every output of a block, eight of them): also
// the calls that follow whole blocks; 0.5 M decisions 27 / 34 us, 6.0 M 83 / 214.
constexpr double kOneStageFrom = 0.5e6;

// Whether [a, a + na) and [b, b + nb) share a byte.
static bool overlap(const void* a, size_t na, const void* b, size_t nb) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + nb && y < x + na;
}

// One call of the decimation from DoP frames (d_dop, rows of `stride` floats)
// or decision bytes (d_bits): the route by what the stream continues from (see
// the head of the file).  DoP frames that have to take the stages are unpacked
// into the context's scratch memory.  So is an input of the product that shares
// memory with the output (a call in place): its CTAs read what others write
// over.  (The stages have read the whole input before the first output is
// written.)
int decim_run(dsdgpu_context_t* c, int nch, const float* d_dop, const uint8_t* d_bits, size_t stride,
              size_t count, float* d_pcm, size_t pcm_stride, double gain_start, double gain_end,
              size_t* out_count) {
  if (!c) return DSDGPU_ERR_ARG;
  dsdgpu_decim_state* s = c->decim;
  if (!s) return c->fail(DSDGPU_ERR_STATE, "decimation not set up");
  if (nch != s->nch) return c->fail(DSDGPU_ERR_ARG, "channel count differs from the setup");
  size_t n = count;
  for (int k = 0; k < s->stages; k++) n /= 2;
  if (out_count) *out_count = n;
  if (count < 2) return DSDGPU_OK;
  if ((!d_bits && !d_dop) || !d_pcm) return c->fail(DSDGPU_ERR_ARG, "null buffer");
  if (pcm_stride < n) return c->fail(DSDGPU_ERR_ARG, "output stride too small");
  cudaSetDevice(c->device);
  cudaStream_t st = c->stream;
  // gain ramp of engine_process_fir_gain (src/engine.c:879-889), then float
  double gs = gain_start;
  if (gs == 0.0) gs = gain_end;
  const int apply = (gs != 1.0 || gain_end != 1.0) ? 1 : 0;
  const double step = n > 1 ? (gain_end - gs) / (double)(n - 1) : 0.0;

  const MmaPlan& M = s->mma;
  look_for_capture(c, s);
  const int rag = (int)(count % (size_t)M.B);
  const double work = (double)count * nch;
  // stages at the start of the call, and to its end
  const bool only = s->on_device || (s->stages == 1 && work >= kOneStageFrom);
  const bool stages = s->from == dsdgpu_decim_state::kLines || s->ragged || only;
  const bool all = only || (stages && (count < (size_t)128 * M.B || (rag && work < kRaggedFrom[s->stages])));
  const size_t in_row = d_dop ? count / 16 * sizeof(float) : count;
  const size_t in_step = d_dop ? stride * sizeof(float) : stride;
  if (!all && n > 0 &&
      overlap(d_dop ? (const void*)d_dop : d_bits, in_step * (size_t)(nch - 1) + in_row, d_pcm,
              sizeof(float) * (pcm_stride * (size_t)(nch - 1) + n))) {
    const size_t row = (count + 255) & ~(size_t)255;
    int rc = c->ensure_scratch(row * (size_t)nch);
    if (rc) return rc;
    uint8_t* copy = (uint8_t*)c->d_scratch;
    if (d_dop) {
      rc = dsdgpu_dop_unpack(c, nch, d_dop, stride, count / 16, copy, row);
      if (rc) return rc;
    } else {
      for (int ch = 0; ch < nch; ch++) {
        const cudaError_t e = cudaMemcpyAsync(copy + row * (size_t)ch, d_bits + stride * (size_t)ch, count,
                                              cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return c->cuda_fail(e, "decimation input copy");
      }
    }
    d_dop = nullptr;
    d_bits = copy;
    stride = row;
  }

  int col_first = 0;
  if (stages) {
    int rc = to_lines(c, s);
    if (rc) return rc;
    const size_t part = all ? count : (size_t)64 * M.B;
    const uint8_t* bits = d_bits;
    size_t bstride = stride;
    if (d_dop) {
      bstride = (part + 255) & ~(size_t)255;
      rc = c->ensure_scratch(bstride * (size_t)nch);
      if (rc) return rc;
      rc = dsdgpu_dop_unpack(c, nch, d_dop, stride, part / 16, (uint8_t*)c->d_scratch, bstride);
      if (rc) return rc;
      bits = (const uint8_t*)c->d_scratch;
    }
    const double* y = nullptr;
    size_t m = 0;
    rc = staged(c, s, bits, bstride, part, &y, &m);
    if (rc) return rc;
    if (m > 0) {
      decim_gain_kernel<<<nb((long long)m * nch, 256), 256, 0, st>>>(y, s->row, (long long)m, nch, gs,
                                                                   step, apply, d_pcm, pcm_stride);
      c->launches++;
    }
    if (all) {
      const cudaError_t e = cudaGetLastError();
      return e == cudaSuccess ? DSDGPU_OK : c->cuda_fail(e, "decimation launch");
    }
    col_first = 64;   // the windows of the outputs from here on lie in this call
  }
  MmaIn I{};
  I.dop = d_dop;
  I.bits = d_bits;
  I.stride = stride;
  I.count = (long long)count;
  I.tail = s->tail();
  I.tail_len = s->tail_len;
  I.tail_stride = (size_t)s->tail_cap;
  const long long total = (long long)s->tail_len + (long long)count;
  const int keep = (int)std::min<long long>(total, 64ll * M.B + rag);
  uint8_t* next = s->d_tail + (size_t)(s->tail_buf ^ 1) * nch * s->tail_cap;
  const long long cols = ((long long)n + M.F - 1) / M.F - col_first;
  const unsigned tiles = (unsigned)((std::max(cols, 0ll) + kMmaCols - 1) / kMmaCols);
  const unsigned per = tiles + (unsigned)((keep + 4095) / 4096);
  const dim3 grid(per * (unsigned)nch);
  const size_t smem = mma_smem_bytes(M);
  const double scale = std::ldexp(1.0, -M.shift);
  if (d_dop)
    decim_mma_kernel<true><<<grid, 32 * kMmaWarps, smem, st>>>(M, I, s->d_taps, col_first, tiles, per, (long long)n,
                                                               scale, gs, step, apply, d_pcm, pcm_stride,
                                                               next, keep, total);
  else
    decim_mma_kernel<false><<<grid, 32 * kMmaWarps, smem, st>>>(M, I, s->d_taps, col_first, tiles, per, (long long)n,
                                                                scale, gs, step, apply, d_pcm, pcm_stride,
                                                                next, keep, total);
  c->launches++;
  s->tail_buf ^= 1;
  s->tail_len = keep;
  s->ragged = rag != 0;
  s->from = dsdgpu_decim_state::kTail;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? DSDGPU_OK : c->cuda_fail(e, "decimation launch");
}

extern "C" {

int dsdgpu_decim_setup(dsdgpu_context_t* c, unsigned fs_in, unsigned fs_out, int nch) {
  if (!c || nch < 1) return DSDGPU_ERR_ARG;
  if (fs_out == 0 || fs_in <= fs_out || fs_in % fs_out) return c->fail(DSDGPU_ERR_ARG, "decimation needs fs_in = fs_out * 2^k");
  unsigned r = fs_in / fs_out;
  if (r & (r - 1)) return c->fail(DSDGPU_ERR_ARG, "decimation ratio must be a power of two");
  int S = 0;
  while (r > 1) { S++; r >>= 1; }
  if (S > kMaxStages) return c->fail(DSDGPU_ERR_ARG, "too many stages");
  cudaSetDevice(c->device);
  dsdgpu_decim_state* s = new (std::nothrow) dsdgpu_decim_state();
  if (!s) return DSDGPU_ERR_NOMEM;
  s->stages = S;
  s->nch = nch;
  design_taps(kDecTaps, false, s->taps.h);
  for (int q = 0, k = 0; k < kDecTaps; k++)
    if ((k & 1) == 0 || k == kDecTaps / 2) { s->nz.h[q] = s->taps.h[k]; s->nz.k[q] = k; q++; }
  // group g, pattern p: sum over u = 0..7 of h[16 g + 2 u] * (bit u of p ? 1 : -1)
  double lut[kLutGroups * 256];
  for (int g = 0; g < kLutGroups; g++)
    for (int p = 0; p < 256; p++) {
      double acc = 0.0;
      for (int u = 0; u < 8; u++) {
        const double h = s->taps.h[16 * g + 2 * u];
        acc += ((p >> u) & 1) ? h : -h;
      }
      lut[g * 256 + p] = acc;
    }
  const size_t dbytes = sizeof(double) * (size_t)S * nch * (kDecTaps - 1);
  s->mma = mma_plan(S);
  s->tail_cap = 65 * s->mma.B;
  if (cudaMalloc(&s->d_dly, dbytes) != cudaSuccess || cudaMalloc(&s->d_lut, sizeof lut) != cudaSuccess ||
      cudaMalloc(&s->d_taps, mma_words(s->mma) * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&s->d_tail, (size_t)2 * nch * s->tail_cap) != cudaSuccess ||
      cudaMalloc(&s->d_done, sizeof(int)) != cudaSuccess) {
    delete s;
    return c->cuda_fail(cudaGetLastError(), "decimation buffers");
  }
  // The attribute belongs to the kernel, not to the context: the widest plan's
  // size, so that no context's setup takes another's away.
  MmaPlan widest = s->mma;
  widest.B = 1 << kMaxStages;
  widest.T = 4;   // 62 blocks of lags, and no plan has more
  const int smem = (int)mma_smem_bytes(widest);
  if (cudaFuncSetAttribute(decim_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaFuncSetAttribute(decim_mma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    delete s;
    return c->cuda_fail(cudaGetLastError(), "decimation kernel attributes");
  }
  cudaMemcpyAsync(s->d_lut, lut, sizeof lut, cudaMemcpyHostToDevice, c->stream);
  const int rc = form_taps(c, s);
  if (rc) {
    delete s;
    return rc;
  }
  cudaMemsetAsync(s->d_dly, 0, dbytes, c->stream);
  cudaMemsetAsync(s->d_done, 0, sizeof(int), c->stream);
  decim_free(c->decim);
  c->decim = s;
  return c->check_status();
}

int dsdgpu_decim_reset(dsdgpu_context_t* c) {
  if (!c) return DSDGPU_ERR_ARG;
  if (!c->decim) return c->fail(DSDGPU_ERR_STATE, "decimation not set up");
  dsdgpu_decim_state* s = c->decim;
  s->tail_len = 0;
  s->ragged = false;
  s->from = dsdgpu_decim_state::kFresh;
  // nothing on the device has to change (the next call starts from no history),
  // unless a graph may run next
  if (!s->on_device) return DSDGPU_OK;
  cudaSetDevice(c->device);
  cudaMemsetAsync(s->d_dly, 0, sizeof(double) * (size_t)s->stages * s->nch * (kDecTaps - 1), c->stream);
  decim_done_kernel<<<1, 1, 0, c->stream>>>(s->d_done);
  c->launches++;
  s->from = dsdgpu_decim_state::kLines;
  return c->check_status();
}

int dsdgpu_decim_process_async(dsdgpu_context_t* c, int nch, const uint8_t* d_bits,
                               size_t bits_stride, size_t count, float* d_pcm, size_t pcm_stride,
                               double gain_start, double gain_end, size_t* out_count) {
  return decim_run(c, nch, nullptr, d_bits, bits_stride, count, d_pcm, pcm_stride, gain_start,
                   gain_end, out_count);
}

int dsdgpu_decim_process_f64_async(dsdgpu_context_t* c, int nch, const double* d_in,
                                   size_t in_stride, size_t count, double* d_out,
                                   size_t out_stride, double gain_start, double gain_end,
                                   int soft_clip, size_t* out_count) {
  if (!c) return DSDGPU_ERR_ARG;
  dsdgpu_decim_state* s = c->decim;
  if (!s) return c->fail(DSDGPU_ERR_STATE, "decimation not set up");
  if (nch != s->nch) return c->fail(DSDGPU_ERR_ARG, "channel count differs from the setup");
  size_t n = count;
  for (int k = 0; k < s->stages; k++) n /= 2;
  if (out_count) *out_count = n;
  if (count < 2) return DSDGPU_OK;
  if (!d_in || !d_out) return c->fail(DSDGPU_ERR_ARG, "null buffer");
  if (nch > 1 && (in_stride < count || out_stride < n))
    return c->fail(DSDGPU_ERR_ARG, "row stride shorter than the count");
  cudaSetDevice(c->device);
  cudaStream_t st = c->stream;
  look_for_capture(c, s);
  int rc = to_lines(c, s);
  if (rc) return rc;
  rc = ensure_rows(c, s, count);
  if (rc) return rc;
  double* buf[2] = {s->d_buf, s->d_buf + s->row * (size_t)nch};
  size_t cur = count;
  const double* in = d_in;
  size_t istride = in_stride;
  for (int k = 0; k < s->stages; k++) {
    const long long m = (long long)(cur / 2);
    double* out = buf[k & 1];
    double* dly = s->d_dly + (size_t)k * nch * (kDecTaps - 1);
    if (m > 0) {
      decim_stage_kernel<<<nb(m * nch, 256), 256, 0, st>>>(s->nz, in, istride, m, dly, out, s->row, nch,
                                                           nullptr);
      decim_dly_kernel<false><<<nch, 64, 0, st>>>(nullptr, in, istride, 2 * m, dly, nch, nullptr);
      c->launches += 2;
    }
    in = out;
    istride = s->row;
    cur = (size_t)m;
  }
  // gain ramp of the rate-conversion branch (src/engine.c:646-651), soft clip (:704-717)
  double gs = gain_start;
  if (gs == 0.0) gs = gain_end;
  const int apply = (gs != 1.0 || gain_end != 1.0) ? 1 : 0;
  const double step = n > 1 ? (gain_end - gs) / (double)(n - 1) : 0.0;
  if (n > 0) {
    decim_gain_f64_kernel<<<nb((long long)n * nch, 256), 256, 0, st>>>(
        in, istride, (long long)n, nch, gs, step, apply, soft_clip ? 1 : 0, d_out, out_stride);
    c->launches++;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? DSDGPU_OK : c->cuda_fail(e, "decimation launch");
}

int dsdgpu_decim_process_f64(dsdgpu_context_t* c, int nch, const double* d_in, size_t in_stride,
                             size_t count, double* d_out, size_t out_stride, double gain_start,
                             double gain_end, int soft_clip, size_t* out_count) {
  const int rc = dsdgpu_decim_process_f64_async(c, nch, d_in, in_stride, count, d_out, out_stride,
                                                gain_start, gain_end, soft_clip, out_count);
  return rc ? rc : c->check_status();
}

int dsdgpu_decim_process(dsdgpu_context_t* c, int nch, const uint8_t* d_bits, size_t bits_stride,
                         size_t count, float* d_pcm, size_t pcm_stride, double gain_start,
                         double gain_end, size_t* out_count) {
  const int rc = dsdgpu_decim_process_async(c, nch, d_bits, bits_stride, count, d_pcm, pcm_stride,
                                            gain_start, gain_end, out_count);
  return rc ? rc : c->check_status();
}

}  // extern "C"
