// Trellis (Viterbi look-ahead) 1-bit sigma-delta modulator for sm_103a.
//
// One warp runs one SDM job (a channel block or a DAS segment); a persistent
// grid pulls jobs from an atomic counter, so one launch covers any mix of
// channels, segments and streams.  Lane i owns the candidate at rank i
// (K <= 32): its NTF state, cost, path, traceback bit and a lat-bit traceback
// ring live in registers.  Each input sample:
//
//   1. expansion   every live lane advances its NTF (FP64, reference order,
//                  no contraction: __dadd_rn/__dmul_rn) and forms both
//                  children: slots 2i (bit 0, state[0] + 1) and 2i + 1
//                  (bit 1, state[0] - 1)          (reference src/trellis.c:37-191)
//   2. selection   the 2n children sorted by int64 cost bits and index, as
//                  one 32-bit word each where those tell, the whole pairs
//                  where they do not; majority vote on the traceback bit with
//                  the 1.1x override; without equal paths the sorted
//                  positions of the eligible children are their ranks, else
//                  the reference's ordered insertion with path-hash dedup,
//                  the hash chains walked in shared memory
//                                                  (src/trellis.c:582-731)
//   3. commit      survivors pull their parent's state, path, traceback bit
//                  and ring with shuffles, normalise cost by the new minimum
//                  and write their decision bit into the ring
//                                                  (src/trellis.c:938-972)
//
// The shared-memory slot arrays (path, cost bits, chain link for both banks)
// reproduce the reference's slot memory, including the K = 32 store one past
// act[] that lands on path_hash[0] while bank 1 is sorted (src/trellis.c:668-673).
//
// The kernels are instantiated twice: in sdm_trellis.cu with the products that
// both children share on the integer pipe (IM), and in sdm_warp_fp64.cu with
// all products in FP64, for filters whose coefficients are out of the integer
// products' range.
#pragma once
#include "sdm_internal.h"
#include "sdm_intmul.h"

#include <climits>

namespace dsdgpu {

// One warp per CTA (one job, or 32 / LPJ jobs side by side for K <= 16): a
// few thousand long-running jobs spread evenly over the SMs.  At 32 lanes a
// launch bound of 13 CTAs per SM holds the kernel at 128 registers (up to 112
// bytes of spills), one of 12 at 168 without spills, for launches that fit it;
// at narrower widths the compiler takes at most 168 (up to 36 bytes of spills at
// orders 7 to 10), of which 12 CTAs fit.
constexpr int kRegRingWords = 8;      // rings held in registers: lat <= 256
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ long long key_of(double c) { return __double_as_longlong(c); }

// A ring word kept opaque in a register: without it the word-select loops over
// a 64-word ring compile to an indexed local-memory array.
template <int RW>
__device__ __forceinline__ uint32_t reg_word(uint32_t v) {
  if constexpr (RW > kRegRingWords) asm volatile("" : "+r"(v));
  return v;
}

template <int LPJ>
__device__ __forceinline__ unsigned long long shfl64(unsigned long long v, int src, unsigned hm) {
  return (unsigned long long)__shfl_sync(hm, (long long)v, src, LPJ);
}

// ballot / match over the job's lanes, as bits of the job's lane numbers
#define BALLOT(p) (__ballot_sync(hm, (p)) >> sh)
#define MATCH(v) (__match_any_sync(hm, (v)) >> sh)

// The NTF advance with y = 0 (src/trellis.c:37-151; every order has the
// same shape): d[0] = (s0 - g0 s1) + x; d[i] = (s[i] + s[i-1]) - g[i] s[i+1];
// d[N-1] = s[N-1] + s[N-2]; v = ((x + a0 d0) + a1 d1) + ...  The two children
// of a candidate share s[1..N-1], so everything that does not involve s[0]
// (g0 s1, g1 s2, d[2..N-1] and a[i] d[i] for i >= 2) is the same for both
// siblings: it is computed once per parent, while the next selection runs,
// and handed to the surviving children as a Pack.  Each sample then keeps only
// the s[0]-dependent operations on its critical path.  Every operation is the
// reference's, in the reference's order, rounded separately (no contraction).
//
// A loop filter's resonators make every second g zero: the odd ones for even
// orders, the even ones for odd orders, but the odd ones in the table's filters
// of odd order above DSD512 (FLIP: the builds for filters whose coefficients the
// integer products do not take, such as these, go by that pattern).  While
// that holds and no value is infinite or NaN, g[i] s[i+1] is a zero and
// subtracting it leaves its operand as it is (up to the sign of a zero, which
// no cost depends on), so those products and differences are not issued: 35
// of the 41 + 1 FP64 instructions of a step at order 7.  `zg` says that they
// may be left out; a non-finite cost or state, or other g, takes them all.
template <int N>
struct Pack {
  double G0;      // g0 * s1
  double G1;      // g1 * s2          (N >= 3)
  double D[N];    // d[i], i = 2..N-1
  double A[N];    // a[i] * d[i], i = 2..N-1
};

template <int N, bool FLIP>
__host__ __device__ constexpr bool g_zero(int i) { return (i & 1) == ((N & 1) && !FLIP ? 0 : 1); }

// middle indices i = 2..N-2 with a nonzero g
template <int N, bool FLIP>
__host__ __device__ constexpr int mid_g() {
  int c = 0;
  for (int i = 2; i <= N - 2; i++) c += g_zero<N, FLIP>(i) ? 0 : 1;
  return c;
}

template <int N, bool FLIP>
__host__ __device__ constexpr int shared_ops() {
  return N >= 3 ? 1 + 2 * mid_g<N, FLIP>() + (N - 3) + 1 + (N - 2) : 1;
}

// index of the k-th middle g that is not zero
template <int N, bool FLIP>
__host__ __device__ constexpr int mid_g_at(int k) {
  int c = 0;
  for (int i = 2; i <= N - 2; i++)
    if (!g_zero<N, FLIP>(i)) {
      if (c == k) return i;
      c++;
    }
  return 2;
}

// FP64 operations that stay under the branch they are written under, and the
// count of that branch's passes (0 or 1): a loop stays a branch, while a short
// condition becomes a predicate, under which an FP64 instruction costs its 64
// cycles whether its result is wanted or not (measured).
__device__ __forceinline__ double vmul(double a, double b) {
  double r;
  asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}
__device__ __forceinline__ double vadd(double a, double b) {
  double r;
  asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}
__device__ __forceinline__ double vsub(double a, double b) {
  double r;
  asm volatile("sub.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}
__device__ __forceinline__ int all_products(bool zg) {
  int z = zg ? 0 : 1;
  asm volatile("" : "+r"(z));
  return z;
}

// Operation k of the shared part, inputs S[1..N-1] (a child's state), into
// np (with scratch tg).  Orders respect the dependencies when k runs
// 0, 1, 2, ...
template <int N, bool IM, bool FLIP>
__device__ __forceinline__ void shared_op(int k, const SdmParams& P, const double (&S)[N],
                                          Pack<N>& np, double (&tg)[N], bool zg) {
  auto mulg = [&](int i, double x) { return IM ? int_mul(P.ig[i], x) : __dmul_rn(P.g[i], x); };
  auto mula = [&](int i, double x) { return IM ? int_mul(P.ia[i], x) : __dmul_rn(P.a[i], x); };
  if (N < 3) {
    if (k == 0) np.G0 = mulg(0, S[1]);
    return;
  }
  constexpr int M = N - 3;   // middle indices i = 2..N-2
  constexpr int Z = mid_g<N, FLIP>();
  if (k == 0) {
    if (g_zero<N, FLIP>(0)) np.G1 = mulg(1, S[2]);
    else np.G0 = mulg(0, S[1]);
    return;
  }
  k -= 1;
  if (k < Z) { const int i = mid_g_at<N, FLIP>(k); tg[i] = mulg(i, S[i + 1]); return; }
  k -= Z;
  if (k < M) { const int i = 2 + k; np.D[i] = __dadd_rn(S[i], S[i - 1]); return; }
  k -= M;
  if (k == 0) { np.D[N - 1] = __dadd_rn(S[N - 1], S[N - 2]); return; }
  k -= 1;
  if (k < Z) { const int i = mid_g_at<N, FLIP>(k); np.D[i] = __dsub_rn(np.D[i], tg[i]); return; }
  k -= Z;
  if (k == 0) {
    // the products with the g that are zero in the table's filters
#pragma unroll 1
    for (int z = all_products(zg); __builtin_expect(z > 0, 0); z--) {
      if (g_zero<N, FLIP>(0)) np.G0 = vmul(P.g[0], S[1]);
      else np.G1 = vmul(P.g[1], S[2]);
#pragma unroll
      for (int i = 2; i <= N - 2; i++)
        if (g_zero<N, FLIP>(i)) np.D[i] = vsub(np.D[i], vmul(P.g[i], S[i + 1]));
    }
  }
  if (k < N - 2) { const int i = 2 + k; np.A[i] = mula(i, np.D[i]); return; }
}

template <int N, bool FLIP>
__device__ __forceinline__ void shared_all(const SdmParams& P, const double (&S)[N], Pack<N>& np,
                                           bool zg) {
  double tg[N];
#pragma unroll
  for (int k = 0; k < shared_ops<N, FLIP>(); k++) shared_op<N, false, FLIP>(k, P, S, np, tg, zg);
}

// Whether this filter's g has the zero pattern and no a is zero (a state that
// is not finite then always shows in a cost that is not finite).
__device__ __forceinline__ bool zero_pattern(const SdmParams& P, int N, bool flip) {
  bool ok = true;
  for (int i = 0; i < N; i++) {
    const long long a = __double_as_longlong(P.a[i]) & 0x7fffffffffffffffll;
    const long long g = __double_as_longlong(P.g[i]) & 0x7fffffffffffffffll;
    if (a == 0 || a >= 0x7ff0000000000000ll || g >= 0x7ff0000000000000ll) ok = false;
    if (i <= N - 2 && (i & 1) == ((N & 1) && !flip ? 0 : 1) && g != 0) ok = false;
  }
  return ok;
}

__device__ __forceinline__ bool not_finite(double v) {
  return ((unsigned)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u;
}

// Shared memory of one job run by LPJ lanes: the slot memory of both banks
// for its 2 * LPJ children (K <= LPJ, so children 2K.. are never touched),
// the 128-bucket path hash and the selection scratch.
template <int LPJ>
struct WarpSmem {
  static constexpr int S = 2 * LPJ;
  unsigned long long path[2][S];
  long long key[2][S];
  int8_t link[2][S];
  int8_t heads[kBuckets];
  int8_t act[LPJ];             // scatter target of the fast selection
  uint8_t hashmark[S];         // children the serial path hashed (verify mode)
  uint8_t hashmark2[S];        // children the fast path deems hashed
  int8_t pos[S];               // sorted position of each child (serial path)
  int8_t idx_at[S];            // child at each sorted position (serial path)
  // lanes by path, for the search of equal paths: 64 entries a lane, so that
  // two different paths seldom share one (32 lanes, 2,048 entries: 0.24 pairs
  // a sample)
  static constexpr int kTab = 64 * LPJ;
  uint8_t tab[kTab];
  // the run's counts (conv_fail, next_filter_drops, total_children), added to
  // once a block: out of the step loop's registers
  unsigned long long count[3];
};

// Lanes per job: the smallest power of two >= K (at least 2) is the tightest
// packing, 32 / LPJ jobs per warp; a requested width (SdmParams::lanes) is
// raised to it.
__host__ __device__ constexpr int min_lanes(int K) {
  return K > 16 ? 32 : K > 8 ? 16 : K > 4 ? 8 : K > 2 ? 4 : 2;
}

template <int LPJ>
__host__ __device__ constexpr unsigned job_mask(int sh) {
  return LPJ == 32 ? 0xffffffffu : (((1u << LPJ) - 1u) << sh);
}

// (key, index) order of the survivor selection: cost bits as int64, then slot.
__device__ __forceinline__ bool key_less(long long ka, int ia, long long kb, int ib) {
  return ka < kb || (ka == kb && ia < ib);
}

// A child's cost and index as one 32-bit word: 26 bits of the cost (its key
// from 2^-24 to 2^8 in 2^21 steps an octave, clamped outside) over 6 bits of
// index.  Words order like (key, index) wherever their cost parts differ.
constexpr unsigned kWordBase = (1023u - 24u) << 21;
constexpr unsigned kWordTop = 0x3fffffeu;    // largest cost part of a child
constexpr unsigned kWordNone = 0x3ffffffu;   // no child

__device__ __forceinline__ unsigned key_word(long long key, int idx) {
  const unsigned hi = (unsigned)((unsigned long long)key >> 32);
  const unsigned u = __funnelshift_l((unsigned)key, hi, 1);   // key >> 31 for keys >= 0
  const unsigned w = min(max(u, kWordBase) - kWordBase, kWordTop);
  return (w << 6) | (unsigned)idx;
}

// Bitonic sort of the 2 * LPJ words of one job, two per lane (sorted positions
// 2*lane and 2*lane + 1), ascending: each merge starts with the mirrored
// exchange, so every exchange keeps the smaller word at the lower position.
template <int LPJ, typename Hook>
__device__ __forceinline__ void word_sort(unsigned& c0, unsigned& c1, int lane, unsigned hm,
                                          Hook&& hook) {
  int stage = 0;
#pragma unroll
  for (int k = 2; k <= 2 * LPJ; k <<= 1) {
    hook(stage++);
    if (k > 2) {
      const bool low = (lane & (k >> 2)) == 0;
      const unsigned p1 = __shfl_xor_sync(hm, c1, (k >> 1) - 1, LPJ);
      const unsigned p0 = __shfl_xor_sync(hm, c0, (k >> 1) - 1, LPJ);
      c0 = low ? min(c0, p1) : max(c0, p1);
      c1 = low ? min(c1, p0) : max(c1, p0);
#pragma unroll
      for (int j = k >> 2; j > 1; j >>= 1) {
        hook(stage++);
        const bool lo = (lane & (j >> 1)) == 0;
        const unsigned q0 = __shfl_xor_sync(hm, c0, j >> 1, LPJ);
        const unsigned q1 = __shfl_xor_sync(hm, c1, j >> 1, LPJ);
        c0 = lo ? min(c0, q0) : max(c0, q0);
        c1 = lo ? min(c1, q1) : max(c1, q1);
      }
      hook(stage++);
    }
    const unsigned mn = min(c0, c1), mx = max(c0, c1);
    c0 = mn;
    c1 = mx;
  }
}

// The same order by the whole (key, index) pairs.  Not unrolled: it is rare.
template <int LPJ>
__device__ __forceinline__ void full_sort(long long& kA, int& iA, long long& kB, int& iB, int lane,
                                          unsigned hm) {
#pragma unroll 1
  for (int k = 2; k <= 2 * LPJ; k <<= 1) {
    const bool asc = ((2 * lane) & k) == 0;
#pragma unroll 1
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j == 1) {
        const bool sw = asc ? key_less(kB, iB, kA, iA) : key_less(kA, iA, kB, iB);
        if (sw) {
          const long long tk = kA; kA = kB; kB = tk;
          const int ti = iA; iA = iB; iB = ti;
        }
      } else {
        const int lj = j >> 1;
        const bool keep_min = (((lane & lj) == 0) == asc);
        long long pk = __shfl_xor_sync(hm, kA, lj, LPJ);
        int pi = __shfl_xor_sync(hm, iA, lj, LPJ);
        if (keep_min == key_less(pk, pi, kA, iA)) { kA = pk; iA = pi; }
        pk = __shfl_xor_sync(hm, kB, lj, LPJ);
        pi = __shfl_xor_sync(hm, iB, lj, LPJ);
        if (keep_min == key_less(pk, pi, kB, iB)) { kB = pk; iB = pi; }
      }
    }
  }
}

// The order of the children of n candidates (their keys in shared memory) for the
// samples whose words do not tell: two children within 2^-21 of each other's
// cost, a cost out of the words' range, or one that is not finite.  The words of
// the keys' distances from the least one tell nearly always, above all once a
// modulator has run away (its costs agree to many places on every sample, for
// good); else the whole pairs are sorted.  Out of line: its code stays out of the
// step loop's registers.  Returns the children at sorted positions 2 * lane and
// 2 * lane + 1 as bits 0 .. 5 and 6 ..  K = 32, order 7, a signal that overloads
// the modulator: 4.4 us a step, 5.7 with the pairs' sort alone.
template <int LPJ>
static __device__ __noinline__ int order_again(const long long* key, int n, int lane, unsigned hm) {
  __syncwarp(hm);
  const long long k0 = lane < n ? key[2 * lane] : LLONG_MAX, k1 = lane < n ? key[2 * lane + 1] : LLONG_MAX;
  // the least key and the largest distance from it, of those that are costs
  const bool c0 = (unsigned long long)k0 < 0x7ff0000000000000ull, c1 = (unsigned long long)k1 < 0x7ff0000000000000ull;
  const unsigned h0 = c0 ? (unsigned)(k0 >> 32) : ~0u, h1 = c1 ? (unsigned)(k1 >> 32) : ~0u;
  const unsigned mh = __reduce_min_sync(hm, min(h0, h1));
  const unsigned ml = __reduce_min_sync(hm, min(h0 == mh ? (unsigned)k0 : ~0u, h1 == mh ? (unsigned)k1 : ~0u));
  const unsigned long long least = (unsigned long long)mh << 32 | ml;
  const unsigned long long d0 = c0 ? (unsigned long long)k0 - least : 0ull, d1 = c1 ? (unsigned long long)k1 - least : 0ull;
  const unsigned rh = __reduce_max_sync(hm, (unsigned)(max(d0, d1) >> 32));
  const unsigned rl = __reduce_max_sync(hm, rh ? 0u : (unsigned)max(d0, d1));
  const int bits = rh ? 64 - __clz((int)rh) : 32 - __clz((int)rl);
  const int shift = bits > 25 ? bits - 25 : 0;
  unsigned w0 = ((c0 ? (unsigned)(d0 >> shift) : kWordNone) << 6) | (unsigned)(2 * lane);
  unsigned w1 = ((c1 ? (unsigned)(d1 >> shift) : kWordNone) << 6) | (unsigned)(2 * lane + 1);
  word_sort<LPJ>(w0, w1, lane, hm, [](int) {});
  int i0 = (int)(w0 & 63u), i1 = (int)(w1 & 63u);
  auto key_at = [&](int i) { return (i >> 1) < n ? key[i] : LLONG_MAX; };
  long long s0 = key_at(i0), s1 = key_at(i1);
  const long long after = __shfl_down_sync(hm, s0, 1, LPJ);
  const int ia = __shfl_down_sync(hm, i0, 1, LPJ);
  const bool wrong = key_less(s1, i1, s0, i0) || (lane < LPJ - 1 && key_less(after, ia, s1, i1));
  if (__any_sync(hm, wrong)) {
    s0 = k0;
    s1 = k1;
    i0 = 2 * lane;
    i1 = 2 * lane + 1;
    full_sort<LPJ>(s0, i0, s1, i1, lane, hm);
  }
  return i0 | i1 << 6;
}

// Stages of the bitonic sort of 2 * LPJ keys: log2(2 LPJ) (log2(2 LPJ) + 1) / 2
// (21 for 64 keys, 15 for 32, 10, 6, 3).
template <int LPJ>
__host__ __device__ constexpr int sort_stages() {
  return LPJ == 32 ? 21 : LPJ == 16 ? 15 : LPJ == 8 ? 10 : LPJ == 4 ? 6 : 3;
}

// LPJ lanes run one job (lanes_per_job(K)): a whole warp for K > 16, else
// 32 / LPJ jobs side by side in one warp, so small trellises do not leave
// most of every FP64 warp instruction idle.  `lane` is the lane within the
// job, `hm` the job's lanes; warp intrinsics use hm and width LPJ, ballots
// are shifted to the job's bits.
template <int N, int LPJ, int RW, bool IM>
__device__ void run_job(const SdmParams& P, const SdmJob& job, SdmCtx* __restrict__ ctxs,
                        WarpSmem<LPJ>& sm, int* __restrict__ status) {
  constexpr int S = WarpSmem<LPJ>::S;
  constexpr bool FLIP = !IM && RW == kRegRingWords && (N & 1);   // see Pack
  const int wl = threadIdx.x & 31;
  const int lane = wl & (LPJ - 1);
  const unsigned sh = (unsigned)(wl - lane);
  const unsigned hm = job_mask<LPJ>((int)sh);
  // ctx < 0: the job's end state goes to a scratch context, one per job slot
  // of the launch, at (-ctx - 1) + slot (jobs whose end state nobody reads)
  const int slot_id = (int)blockIdx.x * (32 / LPJ) + wl / LPJ;
  const int dst_i = job.ctx >= 0 ? job.ctx : (-job.ctx - 1) + slot_id;
  const SdmCtx* src = &ctxs[job.copy_from >= 0 ? job.copy_from : dst_i];
  SdmCtx* dst = &ctxs[dst_i];
  const int K = P.cands;
  const int W = (P.lat + 31) >> 5;
  const unsigned long long mask = P.mask;

  int n = src->n, bank = src->bank, pos = src->pos;
  double s[N];
  double cost = 0.0;
  unsigned long long path = 0;
  uint32_t ring[RW];
  int nxt = 0, slot = 0;
#pragma unroll
  for (int k = 0; k < N; k++) s[k] = 0.0;
#pragma unroll
  for (int w = 0; w < RW; w++) ring[w] = 0;
  if (lane < n) {
#pragma unroll
    for (int k = 0; k < N; k++) s[k] = src->s[lane][k];
    cost = src->cost[lane];
    path = src->path[lane];
    nxt = src->next[lane];
    slot = src->slot[lane];
#pragma unroll
    for (int w = 0; w < RW; w++)
      if (w < W) ring[w] = src->ring[lane][w];
  }
  for (int i = lane; i < 2 * S; i += LPJ) {
    const int b = i / S, j = i % S;
    sm.path[b][j] = src->spath[b][j];
    sm.key[b][j] = (long long)src->skey[b][j];
    sm.link[b][j] = src->slink[b][j];
  }
  if (lane == 0) {
    const bool go_on = job.copy_from < 0;
    sm.count[0] = go_on ? src->conv_fail : 0ull;   // cands_collapse counts with it
    sm.count[1] = go_on ? src->next_filter_drops : 0ull;
    sm.count[2] = go_on ? src->total_children : 0ull;
  }
  const unsigned long long coll_over =
      job.copy_from < 0 ? src->cands_collapse - src->conv_fail : 0ull;
  __syncwarp(hm);
  if (job.seed_state) {
    // DAS temp seeding: every live candidate gets the estimated state, cost 0.
    if (lane < n) {
#pragma unroll
      for (int k = 0; k < N; k++) s[k] = job.seed_state[k];
      cost = 0.0;
      sm.key[bank][slot] = key_of(0.0);
    }
    __syncwarp(hm);
  }
  // the products with the filter's zero g are left out while every value is
  // finite (see Pack)
  bool zg = zero_pattern(P, N, FLIP);
  {
    bool nf = false;
#pragma unroll
    for (int k = 0; k < N; k++) nf |= not_finite(s[k]);
    if (__any_sync(hm, nf)) zg = false;
  }
  // the candidate as (s0, s1, shared part of its next advance)
  double cs0 = s[0], cs1 = s[1];
  Pack<N> pk;
  pk.G0 = pk.G1 = 0.0;
  shared_all<N, FLIP>(P, s, pk, zg);
  // whether the states in hand are operands for integer products (a step that
  // finds one that is not forms its products, and the next step's, in FP64)
  bool int_in = false;

  // the traceback ring's word being written, and for the other words the lane
  // whose ring they were when that word was entered: they are moved between
  // lanes once per word, not once per sample
  uint32_t cur = 0;
#pragma unroll
  for (int w = 0; w < RW; w++) {
    const uint32_t r = reg_word<RW>(ring[w]);
    if (w == (pos >> 5)) cur = r;
  }
  int perm = lane;
  // equal paths are searched by a table of paths: the path itself where the
  // masked paths number no more than its entries
  constexpr int kTabBits = LPJ == 32 ? 11 : LPJ == 16 ? 10 : LPJ == 8 ? 9 : LPJ == 4 ? 8 : 7;
  const bool tab_direct = P.depth - 1 <= kTabBits;

  const long long n_in = job.n_in;
  const double* __restrict__ in = job.in;
  double x_cur = 0.0, x_nxt = 0.0;
  if (in) {
    if (lane < n_in) x_cur = in[lane];
    if (LPJ + lane < n_in) x_nxt = in[LPJ + lane];
  }
  int err = 0;
  const bool lim_on = P.state_limit > 0.0;

  for (long long t0 = 0; t0 < n_in; t0 += LPJ) {
   // a block of LPJ inputs, one a lane (the next block's loads in flight)
   const int tn = (int)(n_in - t0 < LPJ ? n_in - t0 : LPJ);
   if (t0 > 0) {
     x_cur = x_nxt;
     x_nxt = (in && t0 + LPJ + lane < n_in) ? in[t0 + LPJ + lane] : 0.0;
   }
   unsigned obits = 0u, k_conv = 0u, k_drop = 0u, k_tot = 0u;
#pragma unroll 1
   for (int tl = 0; tl < tn; tl++) {
    const double x = __shfl_sync(hm, x_cur, tl, LPJ);
    const int nb = bank ^ 1;
    int next_pos = pos + 1;
    if (next_pos == P.lat) next_pos = 0;
    const bool live = lane < n;
    const unsigned livemask = n >= 32 ? 0xffffffffu : ((1u << n) - 1u);
    // only at K = 32 while bank 1 is sorted can a slot's path, cost and chain
    // link be read in a later sample (see the selection)
    const bool links_matter = (K == kMaxCands && nb == 1);

    // ---- 1. expansion: the s0-dependent part of the advance ----
    const unsigned long long q = (path << 1) & mask;
    double S[N];          // the children's shared state s[1..N-1] (clamped)
    S[0] = 0.0;
    double d0 = __dadd_rn(g_zero<N, FLIP>(0) ? cs0 : __dsub_rn(cs0, pk.G0), x);
    double d1 = __dadd_rn(cs1, cs0);
    if (N >= 3 && !g_zero<N, FLIP>(1)) d1 = __dsub_rn(d1, pk.G1);
    for (int z = all_products(zg); __builtin_expect(z > 0, 0); z--) {
      if (g_zero<N, FLIP>(0)) d0 = vadd(vsub(cs0, pk.G0), x);
      else if (N >= 3) d1 = vsub(d1, pk.G1);
    }
    double v = __dadd_rn(x, __dmul_rn(P.a[0], d0));
    v = __dadd_rn(v, __dmul_rn(P.a[1], d1));

    // equal paths: children of two candidates share a path iff their q are
    // equal.  Every live lane leaves its number at its path's table entry; a
    // lane that reads another's number there compares the paths, and a second
    // round tells the other lane.  More than one such lane at one entry takes
    // the warp's match instruction, which costs 270 to 510 cycles (measured)
    // and used to run on every sample.
    int partner = -1;       // the live lane with this lane's q
    bool multi = false;     // three or more live lanes share a q
    unsigned ti;
    if (tab_direct) {
      ti = (unsigned)(q >> 1) & (WarpSmem<LPJ>::kTab - 1);
    } else {
      const unsigned m = ((unsigned)q + (unsigned)(q >> 32) * 0x85ebca77u) * 0x9e3779b1u;
      ti = m >> (32 - kTabBits);
    }
    if (live) sm.tab[ti] = (uint8_t)lane;
    const unsigned nx1 = BALLOT(live && nxt);   // traceback bits of the candidates
    __syncwarp(hm);
    const int holder = live ? (int)sm.tab[ti] : lane;
    const bool pany = __any_sync(hm, holder != lane);

#pragma unroll
    for (int i = 2; i < N; i++) v = __dadd_rn(v, pk.A[i]);
    S[1] = d1;
#pragma unroll
    for (int i = 2; i < N; i++) S[i] = pk.D[i];
    if (lim_on) {
#pragma unroll
      for (int k = 1; k < N; k++) S[k] = clamp_state(S[k], P.state_limit);
    }
    if (pany) {
      const unsigned long long qh = shfl64<LPJ>(q, holder, hm);
      const bool lose = holder != lane;
      __syncwarp(hm);
      if (lose) sm.tab[ti] = (uint8_t)lane;
      __syncwarp(hm);
      const int second = live ? (int)sm.tab[ti] : lane;
      const unsigned long long q2 = shfl64<LPJ>(q, second, hm);
      if (__any_sync(hm, lose && second != lane)) {
        const unsigned mm = MATCH(live ? q : ~(unsigned long long)lane) & livemask;
        const unsigned oth = mm & ~(1u << lane);
        if (live && __popc(mm) == 2) partner = __ffs(oth) - 1;
        multi = __any_sync(hm, live && __popc(mm) > 2);
      } else if (lose) {
        if (qh == q) partner = holder;
      } else if (live && second != lane && q2 == q) {
        partner = second;
      }
    }
    // the parent's traceback bit at next_pos
    uint32_t wv = cur;
    const bool cross = (next_pos >> 5) != (pos >> 5);
    if (cross) {
#pragma unroll
      for (int w = 0; w < RW; w++) {
        const uint32_t r = reg_word<RW>(ring[w]);
        if (w == (next_pos >> 5)) wv = r;
      }
      wv = __shfl_sync(hm, wv, perm, LPJ);
    }
    const int new_next = (int)((wv >> (next_pos & 31)) & 1u);

    const double e0 = __dadd_rn(v, P.a[0]);
    const double e1 = __dsub_rn(v, P.a[0]);
    const long long key0 = key_of(__dadd_rn(cost, __dmul_rn(e0, e0)));
    const long long key1 = key_of(__dadd_rn(cost, __dmul_rn(e1, e1)));
    if (live) {
      sm.key[nb][2 * lane] = key0;
      sm.key[nb][2 * lane + 1] = key1;
      if (links_matter) {
        sm.path[nb][2 * lane] = q;
        sm.path[nb][2 * lane + 1] = q | 1ull;
      }
    }
    const bool odd_key = live && ((unsigned)(key0 >> 32) >= 0x7ff00000u ||
                                  (unsigned)(key1 >> 32) >= 0x7ff00000u);
    // a state that is not finite shows in the cost; with integer products the
    // shared part's range check finds it
    if (!IM && __any_sync(hm, odd_key)) zg = false;

    // the children's shared part, spread over the sort's stages below
    Pack<N> npk;
    double tg[N];
    // ---- 2. selection ----
    // All 2n children sorted by (cost bits as int64, slot index): position 0
    // is the reference's minimum (first index among equal costs), the first
    // sorted child carrying the majority bit is its best_maj, and the
    // eligible children keep their (cost, index) order (src/trellis.c:628-652).
    // The sort runs on 32-bit words (key_word): one shuffle and one min / max
    // an exchange where the whole (key, index) pairs took three shuffles and a
    // 64-bit comparison (1,000 of a step's 7,400 cycles).
    unsigned c0 = live ? key_word(key0, 2 * lane) : (kWordNone << 6) | (unsigned)(2 * lane);
    unsigned c1 = live ? key_word(key1, 2 * lane + 1) : (kWordNone << 6) | (unsigned)(2 * lane + 1);
    // The shared-part operations ride on the sort stages, except the last
    // kDeferOps, which are issued at the start of the selection so that its
    // integer work runs while they occupy the FP64 unit.
    constexpr int kOps = shared_ops<N, FLIP>();
    constexpr int kStages = sort_stages<LPJ>();
    constexpr int kDeferOps = 6;
    constexpr int kSortOps = (kOps < kStages ? kOps : kStages) > kDeferOps
                                 ? (kOps < kStages ? kOps : kStages) - kDeferOps : 0;
    word_sort<LPJ>(c0, c1, lane, hm, [&](int st) {
      if (st < kSortOps) shared_op<N, IM, FLIP>(st, P, S, npk, tg, zg);
    });
    int si0 = (int)(c0 & 63u), si1 = (int)(c1 & 63u);
    {
      const unsigned after = __shfl_down_sync(hm, c0, 1, LPJ);
      const bool same = (c0 >> 6) == (c1 >> 6) && (c1 >> 6) != kWordNone;
      const bool same2 = lane < LPJ - 1 && (c1 >> 6) == (after >> 6) && (c1 >> 6) != kWordNone;
      if (__any_sync(hm, same || same2 || odd_key)) {
        const int both = order_again<LPJ>(sm.key[nb], n, lane, hm);
        si0 = both & 63;
        si1 = both >> 6;
      }
    }
    // All candidates carry one traceback bit nearly always (they share their
    // history lat samples back): it is the wanted one, every child is eligible,
    // and without equal paths the sorted positions are the ranks.
    const bool uni = (nx1 == 0u || nx1 == livemask) && !pany && P.mode == kModeFast;
    int want = nx1 != 0u ? 1 : 0;
    const bool sl0 = (si0 >> 1) < n, sl1 = (si1 >> 1) < n;
    if (!uni) {
    const int sn0 = (int)((nx1 >> (si0 >> 1)) & 1u);   // traceback bit of each sorted child
    const int sn1 = (int)((nx1 >> (si1 >> 1)) & 1u);
    const int votes1 = 2 * __popc(nx1);
    const int majority = (votes1 > 2 * n - votes1) ? 1 : 0;
    const int first = __shfl_sync(hm, si0, 0, LPJ);
    want = (int)((nx1 >> (first >> 1)) & 1u);
    if (want != majority) {
      __syncwarp(hm);
      const unsigned mA = BALLOT(sl0 && sn0 == majority);
      const unsigned mB = BALLOT(sl1 && sn1 == majority);
      int at = 1 << 20;
      if (mA) at = 2 * (__ffs(mA) - 1);
      if (mB) at = min(at, 2 * (__ffs(mB) - 1) + 1);
      if (at < (1 << 20)) {
        const int bA = __shfl_sync(hm, si0, at >> 1, LPJ);
        const int bB = __shfl_sync(hm, si1, at >> 1, LPJ);
        const double cbm = __longlong_as_double(sm.key[nb][(at & 1) ? bB : bA]);
        if (cbm < __dmul_rn(__longlong_as_double(sm.key[nb][first]), 1.1)) want = majority;
      }
    }
    }
#pragma unroll
    for (int k = kSortOps; k < kOps; k++) shared_op<N, IM, FLIP>(k, P, S, npk, tg, zg);
    if (IM) {
      // operands of this step's integer products and of the next one's (the
      // clamped ones lie between them and the limit): out of range in some lane,
      // and the shared part is formed in FP64
      unsigned w = range_word(d1);
#pragma unroll
      for (int i = 2; i < N; i++) w = max(w, range_word(npk.D[i]));
      bool in = !__any_sync(hm, live && w > kRangeSpan);
      int z = in && int_in ? 0 : 1;
      asm volatile("" : "+r"(z));
#pragma unroll 1
      for (; __builtin_expect(z > 0, 0); z--) {
        bool nf = not_finite(d0) || not_finite(d1);
#pragma unroll
        for (int i = 2; i < N; i++) nf |= not_finite(pk.D[i]);
        if (__any_sync(hm, live && nf)) zg = false;
        shared_all<N, FLIP>(P, S, npk, zg);
        w = range_word(d1);
#pragma unroll
        for (int i = 2; i < N; i++) w = max(w, range_word(npk.D[i]));
        in = !__any_sync(hm, live && w > kRangeSpan);
      }
      int_in = in && P.int_ok;
    }
    const unsigned elig = want ? nx1 : (livemask & ~nx1);
    k_drop += 2u * (unsigned)(n - __popc(elig));
    k_tot += 2u * (unsigned)n;

    // ---- 2b. fast selection ----
    // Without equal paths, the reference's ordered insertion with path-hash
    // dedup keeps exactly the first K eligible children of the (cost, index)
    // order: every insert is new to the hash, evictions drop the largest, ties
    // keep insertion (index) order, skips are children that would not be among
    // the K smallest.  Where two candidates share a q, of each pair of children
    // with one path only the first in that order stays: the later one either
    // finds it hashed, or replaces it, or finds it gone because the list's
    // worst was better already.  (Three or more on one path keep their reference
    // order in the serial path: a child replaced there stays in the hash.)
    // A child is hashed iff fewer than K eligible children with a lower index
    // precede it in that order; only at K = 32 while bank 1 is sorted can the
    // stored chain links be read in a later sample (through the act[32] store
    // onto path_hash[0]), so only then are they written, as "previous hashed
    // child of the same bucket".  There, equal paths, or a bucket-0 child once
    // the list can be full, take the serial path.
    const bool me = live && ((elig >> lane) & 1u);
    bool fast_ok = (P.mode != kModeExact) && !multi;
    unsigned rem0 = 0u, rem1 = 0u;   // lanes whose child 0 / 1 loses to its equal
    if (pany) {
      const bool dup = me && partner >= 0 && ((elig >> (partner & 31)) & 1u);
      if (links_matter) {
        if (__any_sync(hm, dup)) fast_ok = false;
      } else {
        const int ps = partner >= 0 ? partner : lane;
        const long long o0 = (long long)shfl64<LPJ>((unsigned long long)key0, ps, hm);
        const long long o1 = (long long)shfl64<LPJ>((unsigned long long)key1, ps, hm);
        rem0 = BALLOT(dup && key_less(o0, ps, key0, lane));
        rem1 = BALLOT(dup && key_less(o1, ps, key1, lane));
      }
    }
    bool f0 = sl0, f1 = sl1;
    unsigned EA = livemask, EB = livemask;
    int m2 = 2 * n;
    if (!uni) {
      f0 = sl0 && ((elig >> (si0 >> 1)) & 1u) &&
           !((((si0 & 1) ? rem1 : rem0) >> (si0 >> 1)) & 1u);
      f1 = sl1 && ((elig >> (si1 >> 1)) & 1u) &&
           !((((si1 & 1) ? rem1 : rem0) >> (si1 >> 1)) & 1u);
      EA = BALLOT(f0);
      EB = BALLOT(f1);
      m2 = __popc(EA) + __popc(EB);
    }
    int f_cnt = 0, f_Ls = -1, f_link0 = -1, f_link1 = -1;
    long long f_Lk = LLONG_MAX;
    bool f_h0 = false, f_h1 = false;
    if (links_matter && m2 > K && __any_sync(hm, me && (q & (kBuckets - 1)) == 0)) fast_ok = false;
    if (fast_ok) {
      const unsigned below = (1u << lane) - 1u;
      int u0 = 0, u1 = 0;
      if (uni) {
        u0 = __shfl_sync(hm, si0, lane >> 1, LPJ);
        u1 = __shfl_sync(hm, si1, lane >> 1, LPJ);
      } else {
        const int r0 = __popc(EA & below) + __popc(EB & below);
        const int r1 = r0 + (f0 ? 1 : 0);
        if (f0 && r0 < K) sm.act[r0] = (int8_t)si0;
        if (f1 && r1 < K) sm.act[r1] = (int8_t)si1;
      }
      if (links_matter) {
        // eligible children sorted before, with a lower index: OR-scan of
        // one-hot index masks over the sorted positions
        const unsigned long long mine = (f0 ? (1ull << si0) : 0ull) | (f1 ? (1ull << si1) : 0ull);
        unsigned long long inc = mine;
#pragma unroll
        for (int o = 1; o < LPJ; o <<= 1) {
          const unsigned long long u = (unsigned long long)__shfl_up_sync(hm, (long long)inc, o, LPJ);
          if (lane >= o) inc |= u;
        }
        const unsigned long long before0 = inc & ~mine;
        const unsigned long long before1 = before0 | (f0 ? (1ull << si0) : 0ull);
        const int p0 = __popcll(before0 & ((1ull << si0) - 1ull));
        const int p1 = __popcll(before1 & ((1ull << si1) - 1ull));
        sm.hashmark2[si0] = (uint8_t)(f0 && p0 < K);
        sm.hashmark2[si1] = (uint8_t)(f1 && p1 < K);
      }
      __syncwarp(hm);
      f_cnt = m2 < K ? m2 : K;
      if (lane < f_cnt) {
        f_Ls = uni ? ((lane & 1) ? u1 : u0) : (int)sm.act[lane];
        f_Lk = sm.key[nb][f_Ls];
      }
      if (links_matter) {
        f_h0 = live && sm.hashmark2[2 * lane] != 0;
        f_h1 = live && sm.hashmark2[2 * lane + 1] != 0;
        const unsigned H0 = BALLOT(f_h0), H1 = BALLOT(f_h1);
        // lanes whose children fall in this lane's buckets (bits 1..6 of q; the
        // children of bit 0 and 1 have a bucket each): one ballot per bit
        unsigned bm = 0xffffffffu;
#pragma unroll
        for (int k = 1; k < 7; k++) {
          const bool on = ((unsigned)q >> k) & 1u;
          const unsigned bb = __ballot_sync(hm, on);
          bm &= on ? bb : ~bb;
        }
        bm >>= sh;
        const unsigned s0 = bm & H0 & below;
        const unsigned s1 = bm & H1 & below;
        f_link0 = s0 ? 2 * (31 - __clz(s0)) : -1;
        f_link1 = s1 ? 2 * (31 - __clz(s1)) + 1 : -1;
      }
      __syncwarp(hm);
    }

    // ---- 2c. serial selection (exact reference order) ----
    // The reference's act list is always ordered by (cost, index) (children are
    // inserted in index order, after every element of equal cost), so it is
    // held as a set of sorted positions: insertion, eviction of the worst,
    // replacement and the "list full and worst <= s" skip are bit operations.
    // Children are visited in index order and the path hash is walked in
    // shared memory exactly as sdm_check_path does, stale links included.
    int cnt = 0;
    long long Lk = LLONG_MAX;
    int Ls = -1;
    if (!fast_ok || P.mode == kModeVerify) {
      sm.pos[si0] = (int8_t)(2 * lane);
      sm.pos[si1] = (int8_t)(2 * lane + 1);
      sm.idx_at[2 * lane] = (int8_t)si0;
      sm.idx_at[2 * lane + 1] = (int8_t)si1;
      if (live) {
        // every lookup below is in a bucket of this sample's children
        sm.path[nb][2 * lane] = q;
        sm.path[nb][2 * lane + 1] = q | 1ull;
        sm.heads[q & (kBuckets - 1)] = -1;
        sm.heads[(q | 1ull) & (kBuckets - 1)] = -1;
      }
      if (P.mode == kModeVerify && live) { sm.hashmark[2 * lane] = 0; sm.hashmark[2 * lane + 1] = 0; }
      __syncwarp(hm);
      const int nch = 2 * n;
      unsigned long long Lm = 0ull;   // the act list, as sorted positions
      unsigned el = elig;
      while (el) {
        const int p = __ffs(el) - 1;
        el &= el - 1;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = 2 * p + h;
          const int ps = sm.pos[c];
          const long long sk = sm.key[nb][c];
          const unsigned long long sp = sm.path[nb][c];
          if (cnt == K && (63 - __clzll((long long)Lm)) < ps) continue;
          const int b = (int)(sp & (kBuckets - 1));
          int t = sm.heads[b];
          int hops = 0;
          const int hop_limit = P.hop_limit > 0 ? P.hop_limit : 4 * kSlots;
          while (t >= 0) {
            if (sm.path[nb][t] == sp) break;
            t = sm.link[nb][t];
            if (++hops > hop_limit) { err = kStatusChainLimit; t = -1; break; }
          }
          if (t < 0) {
            __syncwarp(hm);
            if (lane == 0) {
              sm.link[nb][c] = sm.heads[b];
              sm.heads[b] = (int8_t)c;
              sm.hashmark[c] = 1;
            }
            __syncwarp(hm);
            if (cnt == K) {
              const int wp = 63 - __clzll((long long)Lm);
              if (K == kMaxCands && nb == 1) {
                // the store to act[32] hits path_hash[0] in the reference layout
                if (lane == 0) sm.heads[0] = sm.idx_at[wp];
                __syncwarp(hm);
              }
              Lm = (Lm & ~(1ull << wp)) | (1ull << ps);
            } else {
              Lm |= 1ull << ps;
              cnt++;
            }
            continue;
          }
          if (sm.key[nb][t] <= sk) continue;
          const bool t_in = t < nch && ((Lm >> sm.pos[t]) & 1ull);
          if (t_in) {
            Lm = (Lm & ~(1ull << sm.pos[t])) | (1ull << ps);      // replace t by s
          } else if (cnt == K) {
            Lm = (Lm & ~(1ull << (63 - __clzll((long long)Lm)))) | (1ull << ps);
          } else {
            Lm |= 1ull << ps;
            cnt++;
          }
        }
      }
      // act[rank] = the child at the rank-th set position
      const unsigned long long lowA = (1ull << (2 * lane)) - 1ull;
      if ((Lm >> (2 * lane)) & 1ull) sm.act[__popcll(Lm & lowA)] = (int8_t)si0;
      if ((Lm >> (2 * lane + 1)) & 1ull) sm.act[__popcll(Lm & (lowA | (1ull << (2 * lane))))] = (int8_t)si1;
      __syncwarp(hm);
      if (lane < cnt) {
        Ls = sm.act[lane];
        Lk = sm.key[nb][Ls];
      }
      __syncwarp(hm);
    }

    if (fast_ok) {
      if (P.mode == kModeVerify) {
        bool vbad = (cnt != f_cnt) || (lane < cnt && (Ls != f_Ls || Lk != f_Lk));
        if (links_matter) {
          if (live && (sm.hashmark[2 * lane] != 0) != f_h0) vbad = true;
          if (live && (sm.hashmark[2 * lane + 1] != 0) != f_h1) vbad = true;
          if (f_h0 && sm.link[nb][2 * lane] != f_link0) vbad = true;
          if (f_h1 && sm.link[nb][2 * lane + 1] != f_link1) vbad = true;
        }
        if (__any_sync(hm, vbad)) err = max(err, (int)kStatusVerifyMismatch);
      } else {
        cnt = f_cnt;
        Ls = f_Ls;
        Lk = f_Lk;
        if (links_matter) {
          if (f_h0) sm.link[nb][2 * lane] = (int8_t)f_link0;
          if (f_h1) sm.link[nb][2 * lane + 1] = (int8_t)f_link1;
        }
      }
    }

    // ---- 3. commit ----
    const int n_old = n;
    const int n_new = cnt;
    const double min_cost = __longlong_as_double(__shfl_sync(hm, Lk, 0, LPJ));
    const bool surv = lane < n_new;
    const int pp = surv ? (Ls >> 1) : lane;
    const int hh = surv ? (Ls & 1) : 0;
    const double fd0 = __shfl_sync(hm, d0, pp, LPJ);
    const double fS1 = __shfl_sync(hm, S[1], pp, LPJ);
    if (N < 3 || !(g_zero<N, FLIP>(0) && zg)) pk.G0 = __shfl_sync(hm, npk.G0, pp, LPJ);
    if (N >= 3 && !(g_zero<N, FLIP>(1) && zg)) pk.G1 = __shfl_sync(hm, npk.G1, pp, LPJ);
#pragma unroll
    for (int i = 2; i < N; i++) {
      pk.D[i] = __shfl_sync(hm, npk.D[i], pp, LPJ);
      pk.A[i] = __shfl_sync(hm, npk.A[i], pp, LPJ);
    }
    // the child's own s0 (both siblings share d0)
    cs0 = __dadd_rn(fd0, hh ? -1.0 : 1.0);
    if (lim_on) cs0 = clamp_state(cs0, P.state_limit);
    cs1 = fS1;
    if (t0 + tl == n_in - 1) {
      // the full child state is only needed when the context is stored
      if (surv) {
        dst->s[lane][0] = cs0;
        dst->s[lane][1] = cs1;
      }
#pragma unroll
      for (int i = 2; i < N; i++) {
        const double f = __shfl_sync(hm, S[i], pp, LPJ);
        if (surv) dst->s[lane][i] = f;
      }
    }
    path = shfl64<LPJ>(q, pp, hm) | (unsigned long long)hh;
    const unsigned pn = __shfl_sync(hm, (unsigned)perm | ((unsigned)new_next << 5), pp, LPJ);
    perm = (int)(pn & 31u);
    nxt = (int)(pn >> 5);
    cur = __shfl_sync(hm, cur, pp, LPJ);
    cur = (cur & ~(1u << (pos & 31))) | ((uint32_t)hh << (pos & 31));
    if (surv) {
      cost = __dsub_rn(__longlong_as_double(Lk), min_cost);
      slot = Ls;
      if (links_matter) sm.key[nb][Ls] = key_of(cost);
    }
    if (cross) {
      // the word is complete: bring the ring's words to their lanes, and enter
      // the next one
#pragma unroll
      for (int w = 0; w < RW; w++) {
        uint32_t r = reg_word<RW>(ring[w]);
        if (w < W) r = __shfl_sync(hm, r, perm, LPJ);
        if (w == (pos >> 5)) r = cur;
        ring[w] = r;
      }
      perm = lane;
#pragma unroll
      for (int w = 0; w < RW; w++) {
        const uint32_t r = reg_word<RW>(ring[w]);
        if (w == (next_pos >> 5)) cur = r;
      }
    }
    __syncwarp(hm);
    k_conv += n_new < n_old ? 1u : 0u;
    n = n_new;
    bank = nb;
    pos = next_pos;
    obits |= (unsigned)want << tl;
   }
   // ---- output: the block's decisions, and its counts ----
   const long long o = t0 + lane - job.skip_out;
   if (lane < tn && o >= 0) job.out[o] = (uint8_t)((obits >> lane) & 1u);
   if (lane == 0) {
     sm.count[0] += k_conv;
     sm.count[1] += k_drop;
     sm.count[2] += k_tot;
   }
  }

  // ---- store the context (the states were stored at the last sample) ----
  if (job.flags & kJobNoStore) {
    err = __reduce_max_sync(hm, err);
    if (err && lane == 0) atomicMax(status, err);
    return;
  }
#pragma unroll
  for (int w = 0; w < RW; w++) {
    uint32_t r = reg_word<RW>(ring[w]);
    if (w < W) r = __shfl_sync(hm, r, perm, LPJ);
    if (w == (pos >> 5)) r = cur;
    ring[w] = r;
  }
  if (lane < n) {
    dst->cost[lane] = cost;
    dst->path[lane] = path;
    dst->next[lane] = (uint8_t)nxt;
    dst->slot[lane] = (uint8_t)slot;
#pragma unroll
    for (int w = 0; w < RW; w++)
      if (w < W) dst->ring[lane][w] = ring[w];
  }
  __syncwarp(hm);
  for (int i = lane; i < 2 * S; i += LPJ) {
    const int b = i / S, j = i % S;
    dst->spath[b][j] = sm.path[b][j];
    dst->skey[b][j] = (unsigned long long)sm.key[b][j];
    dst->slink[b][j] = sm.link[b][j];
  }
  if (lane == 0) {
    dst->n = n;
    dst->bank = bank;
    dst->pos = pos;
    dst->conv_fail = sm.count[0];
    dst->cands_collapse = sm.count[0] + coll_over;
    dst->next_filter_drops = sm.count[1];
    dst->total_children = sm.count[2];
  }
  err = __reduce_max_sync(hm, err);
  if (err && lane == 0) atomicMax(status, err);
}

// kCtas: CTAs that an SM must hold (at 32 lanes 13, which leaves 128 registers
// and some spills, or 12 and 168; a launch takes 12 where its CTAs fit).
template <int N, int LPJ, int kCtas, bool IM>
__global__ void __launch_bounds__(32, kCtas)
sdm_jobs_kernel(SdmParams P, const SdmJob* __restrict__ jobs, int njobs,
                int* __restrict__ job_counter, SdmCtx* __restrict__ ctxs,
                int* __restrict__ status, int groups) {
  extern __shared__ __align__(16) unsigned char sdm_smem_raw[];
  const int wl = threadIdx.x & 31;
  if (wl / LPJ >= groups) return;   // jobs per warp of this launch
  const int lane = wl & (LPJ - 1);
  const unsigned hm = job_mask<LPJ>(wl - lane);
  WarpSmem<LPJ>& sm =
      reinterpret_cast<WarpSmem<LPJ>*>(sdm_smem_raw)[(threadIdx.x >> 5) * (32 / LPJ) + wl / LPJ];
  for (;;) {
    int j = 0;
    if (lane == 0) j = atomicAdd(job_counter, 1);
    j = __shfl_sync(hm, j, 0, LPJ);
    if (j >= njobs) break;
    const SdmJob job = jobs[j];
    run_job<N, LPJ, kRegRingWords, IM>(P, job, ctxs, sm, status);
    __syncwarp(hm);
  }
}

// ---- balanced launches: jobs cut into parts, parts queued ----
// One job per warp pins a job to one SM sub-partition, and every FP64 warp
// instruction of the warps there shares its FP64 pipe.  1,874 DAS segments
// over 152 SMs put 4 warps on 50 sub-partitions and 3 on the rest, and the
// launch lasts as long as the slowest 4-warp pipe (measured: 1,824 jobs, 3 per
// sub-partition, ran at 0.86 of the FP64 rate, 1,874 at 0.79).  A balanced
// launch holds exactly w warps per sub-partition, cuts every job into parts
// of part_len samples, and queues the parts: a warp that finishes part p of
// job j stores the context (as a streamed block boundary does), publishes
// part p + 1 at the queue's tail, and takes the next entry at its head, so
// the jobs move between warps and every pipe stays loaded to the end.
// Queue layout: [0] head, [1] tail, [2 ..] entries (part << 32 | job; empty
// ~0).  A wait for an entry that is not yet published is bounded.
constexpr long long kPartWaitCycles = 8000000000ll;   // ~4 s at 2 GHz

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// The rare wait for an entry not yet published (out of line: inlined, its
// loop changes the register allocation of the step loop).
static __device__ __noinline__ unsigned long long wait_entry(const unsigned long long* p, int* status,
                                                     long long limit) {
  unsigned long long e = ~0ull;
  const long long t0 = clock64();
  if (limit <= 0) limit = kPartWaitCycles;
  do {
    __nanosleep(1000);
    e = ld_acquire_u64(p);
  } while (e == ~0ull && clock64() - t0 < limit);
  if (e == ~0ull && (threadIdx.x & 31) == 0) atomicMax(status, kStatusQueueWait);
  return e;
}

template <int N, bool IM>
__global__ void __launch_bounds__(32, 12)
sdm_parts_kernel(SdmParams P, const SdmJob* __restrict__ jobs, long long part_len,
                 unsigned long long* __restrict__ queue, long long total,
                 SdmCtx* __restrict__ ctxs, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char sdm_smem_raw[];
  WarpSmem<32>& sm = reinterpret_cast<WarpSmem<32>*>(sdm_smem_raw)[0];
  const int lane = threadIdx.x & 31;
  unsigned long long* head = queue;
  unsigned long long* tail = queue + 1;
  unsigned long long* ent = queue + 2;
  for (;;) {
    unsigned long long idx = 0;
    if (lane == 0) idx = atomicAdd(head, 1ull);
    idx = __shfl_sync(kFull, idx, 0);
    if (idx >= (unsigned long long)total) break;
    // every lane reads the entry with acquire semantics (one transaction)
    unsigned long long e = ld_acquire_u64(ent + idx);
    if (e == ~0ull) e = wait_entry(ent + idx, status, P.part_wait_cycles);
    if (e == ~0ull) break;
    __threadfence();   // the previous part's context is read after the entry
    const int j = (int)(e & 0xffffffffull);
    const long long p = (long long)(e >> 32);
    const SdmJob jb = jobs[j];
    const long long off = p * part_len;
    const long long rem = jb.n_in - off;
    SdmJob pj = jb;
    pj.n_in = rem < part_len ? rem : part_len;
    if (jb.in) pj.in = jb.in + off;
    const long long sk = jb.skip_out - off;
    pj.skip_out = sk <= 0 ? 0 : (sk < pj.n_in ? sk : pj.n_in);
    pj.out = jb.out + (off > jb.skip_out ? off - jb.skip_out : 0);
    if (p > 0) {
      // later parts continue from the job's own context
      pj.copy_from = -1;
      pj.seed_state = nullptr;
    }
    const bool more = off + pj.n_in < jb.n_in;
    run_job<N, 32, kRegRingWords, IM>(P, pj, ctxs, sm, status);
    __threadfence();   // this part's context and decisions before its successor's entry
    __syncwarp();
    if (lane == 0 && more) {
      const unsigned long long t = atomicAdd(tail, 1ull);
      atomicExch(ent + t, ((unsigned long long)(p + 1) << 32) | (unsigned long long)(unsigned)j);
    }
    __syncwarp();
  }
}

// ---- launches ----
struct WarpLaunch {
  int lanes;          // a job
  int groups;         // jobs a warp
  bool full_regs;     // at 32 lanes: the build of 12 CTAs an SM
  unsigned blocks;
};

template <bool IM, int LPJ, int kCtas>
int launch_lpj(const SdmParams& P, const WarpLaunch& W, const SdmJob* d_jobs, int njobs, int* d_counter,
               SdmCtx* d_ctxs, int* d_status, cudaStream_t stream) {
  const size_t smem = sizeof(WarpSmem<LPJ>) * (size_t)W.groups;
  switch (P.order) {
#define DSD_CASE(NN)                                                                              \
  case NN:                                                                                        \
    sdm_jobs_kernel<NN, LPJ, kCtas, IM><<<W.blocks, 32, smem, stream>>>(P, d_jobs, njobs, d_counter, \
                                                                        d_ctxs, d_status, W.groups); \
    return 0;
    DSD_CASE(2) DSD_CASE(3) DSD_CASE(4) DSD_CASE(5) DSD_CASE(6)
    DSD_CASE(7) DSD_CASE(8) DSD_CASE(9) DSD_CASE(10)
#undef DSD_CASE
  }
  return -1;
}

template <bool IM>
int launch_warp(const SdmParams& P, const WarpLaunch& W, const SdmJob* d_jobs, int njobs, int* d_counter,
                SdmCtx* d_ctxs, int* d_status, cudaStream_t s) {
  switch (W.lanes) {
    case 32:
      return W.full_regs ? launch_lpj<IM, 32, 12>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, s)
                         : launch_lpj<IM, 32, 13>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, s);
    case 16: return launch_lpj<IM, 16, 10>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, s);
    case 8: return launch_lpj<IM, 8, 10>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, s);
    case 4: return launch_lpj<IM, 4, 10>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, s);
  }
  return launch_lpj<IM, 2, 10>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, s);
}

template <bool IM>
int launch_parts(const SdmParams& P, unsigned blocks, const SdmJob* d_jobs, long long part_len,
                 unsigned long long* d_queue, long long total, SdmCtx* d_ctxs, int* d_status,
                 cudaStream_t stream) {
  const size_t smem = sizeof(WarpSmem<32>);
  switch (P.order) {
#define DSD_CASE(NN)                                                                          \
  case NN:                                                                                    \
    sdm_parts_kernel<NN, IM><<<blocks, 32, smem, stream>>>(P, d_jobs, part_len, d_queue, total, \
                                                           d_ctxs, d_status);                 \
    return 0;
    DSD_CASE(2) DSD_CASE(3) DSD_CASE(4) DSD_CASE(5) DSD_CASE(6)
    DSD_CASE(7) DSD_CASE(8) DSD_CASE(9) DSD_CASE(10)
#undef DSD_CASE
  }
  return -1;
}

// sdm_warp_fp64.cu: the launches above with IM = false
int launch_warp_fp64(const SdmParams& P, const WarpLaunch& W, const SdmJob* d_jobs, int njobs, int* d_counter,
                     SdmCtx* d_ctxs, int* d_status, cudaStream_t stream);
int launch_parts_fp64(const SdmParams& P, unsigned blocks, const SdmJob* d_jobs, long long part_len,
                      unsigned long long* d_queue, long long total, SdmCtx* d_ctxs, int* d_status,
                      cudaStream_t stream);

}  // namespace dsdgpu
