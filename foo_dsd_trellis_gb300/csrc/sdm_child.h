// Trellis SDM for K <= 16 with one child per lane group and the next advance
// run ahead of the selection.
//
// What bounds a small trellis on this part is the chain of one step: an FP64
// instruction takes its warp 64 cycles (76 with all four schedulers of the SM
// busy) whatever the number of active lanes, and a selection of a few hundred
// dependent integer instructions takes as long again.  Here
//
//   * every child of the step owns H lanes (2 KC H lanes a job, 32 / (2 KC H)
//     jobs a warp), and lane q of a child holds the state components
//     q C .. q C + C - 1 (C = ceil(N / H)), so one FP64 instruction forms both
//     children's costs, and H components of every child's advance;
//   * the NTF advance of the next sample is formed for every child before it
//     is known which of them survive: it needs the child's state and the next
//     input only.  The selection runs beside it, and a step costs about the
//     larger of the two instead of their sum.  The survivors gather their
//     advance (d, v) from the child they descend from.
//   * the selection ranks the children by counting: each child's cost as one
//     31-bit word under its traceback bit, the words of all children read from
//     shared memory, and the number of smaller ones is the child's place among
//     the children with its bit, whichever bit is then wanted.  Two children
//     with equal words fall on one place, which their owners notice: those
//     steps rank by the whole (cost, index) pairs.
//
// The operations and their order are the reference's (src/trellis.c:37-191,
// 621-731, 868-973), every one rounded separately:
//   m = g_i s_{i+1};  u = s_i + (i == 0 ? -m : s_{i-1});
//   d_i = u + (i == 0 ? x : i < N-1 ? -m : -0.0);   p_i = a_i d_i
//   v = ((x + p_0) + p_1) + ...;  children: s_0 = d_0 +- 1, e = v +- a_0
// (adding -m is subtracting m, adding -0.0 leaves any value as it is).  The
// products with the filter's structurally zero g are left out while every v
// is finite (see sdm_warp.h).
//
// What bounds a step now is its FP64 instructions (child_ops in
// sdm_trellis.cu, 64 cycles each) and about 500 cycles of the selection that
// they do not cover.  Measured cycles a step, one job (before: the lane-split
// kernel at K <= 4, the warp kernel above): K = 2, order 6 2,668 -> 1,498;
// K = 4 4,720 -> 1,659; K = 8, depth 4 5,548 -> 2,500; K = 16, order 8
// 5,630 -> 2,883.
//
// With one lane a child (H = 1) the step has the most FP64 instructions, and
// with several warps a scheduler the FP64 unit's rate is all there is: there the
// products go to the integer pipe (sdm_intmul.h), a third of the FP64
// instructions.  Measured cycles a step, products in FP64 -> on the integer pipe:
// K = 16, order 8 2,883 -> 2,790 with one job, 7,600 -> 5,697 with 1,500; K = 2,
// order 6 3,011 -> 2,186 with 1,722 jobs; K = 8 3,393 -> 2,567 with 1,216.
#pragma once
#include "sdm_internal.h"
#include "sdm_intmul.h"

#include <climits>

namespace dsdgpu {

namespace child {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBlock = 32;   // samples between loads of inputs and stores of decisions

template <int N>
__host__ __device__ constexpr bool g_zero(int i) { return (i & 1) == ((N & 1) ? 0 : 1); }

// whether any lane's j-th component has a g that the table's filters keep
template <int N, int H, int C>
__host__ __device__ constexpr bool need_g(int j) {
  for (int q = 0; q < H; q++) {
    const int i = q * C + j;
    if (i <= N - 2 && !g_zero<N>(i)) return true;
  }
  return false;
}

__device__ __forceinline__ double neg(double v) {
  return __longlong_as_double(__double_as_longlong(v) ^ (long long)0x8000000000000000ull);
}

// FP64 operations of the advance
template <int N, int H, int C, bool IM>
__host__ __device__ constexpr int advance_ops() {
  int m = 0, d = 1;
  for (int j = 0; j < C; j++) {
    m += need_g<N, H, C>(j) ? 1 : 0;
    d += need_g<N, H, C>(j) && j > 0 ? 1 : 0;
  }
  return (IM ? 0 : m + C) + (H == 1 && !need_g<N, H, C>(0) ? C - 1 : C) + d + N;
}

// FP64 operations that stay where they are written: an FP64 instruction holds
// its unit for 64 cycles, and the selection's integer instructions are written
// between them, a handful behind each (left to itself the compiler puts the
// advance behind the selection, and a step costs the sum of both).
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

// Branches that are seldom taken: their code is placed behind the step's.
#define DSD_RARE(c) __builtin_expect((c), 0)

__device__ __forceinline__ unsigned long long shfl_u64(unsigned long long v, int src) {
  return (unsigned long long)__shfl_sync(kFull, (long long)v, src);
}

__device__ __forceinline__ bool key_less(long long ka, int ia, long long kb, int ib) {
  return ka < kb || (ka == kb && ia < ib);
}

// 30 bits of a cost: its bit pattern from 2^-24 to 2^8 in 2^25 steps an octave,
// clamped outside (equal words are told apart by the whole cost).  With the
// traceback bit above, words stay below 2^31, so the sign of a difference is
// the comparison.
constexpr unsigned long long kWordBase = (unsigned long long)(1023 - 24) << 25;
constexpr unsigned kWordTop = 0x3ffffffeu;
constexpr unsigned kWordNone = 0x7fffffffu;

__device__ __forceinline__ unsigned cost_word(long long key) {
  const unsigned hi = (unsigned)((unsigned long long)key >> 32);
  const unsigned u = __funnelshift_l((unsigned)key, hi, 5);     // key >> 27, its low 32 bits
  // exponents below 2^-24 and above 2^8 (1023 - 24 = 0x3e7, 1023 + 8 = 0x407)
  if (hi < ((1023u - 24u) << 20)) return 0u;
  if (hi >= ((1023u + 8u) << 20)) return kWordTop;
  return min(u - (unsigned)kWordBase, kWordTop);
}

__device__ __forceinline__ int below4(const uint4& w, unsigned word) {
  const unsigned a = (w.x - word) >> 31, b = (w.y - word) >> 31;
  const unsigned c = (w.z - word) >> 31, d = (w.w - word) >> 31;
  return (int)((a + b) + (c + d));
}

// The reference's insertion over the children in index order
// (src/trellis.c:653-731) for one job, by one lane: keys, paths and next bits
// of the children in shared memory, the act list out.  For the samples whose
// equal paths are more than pairs, and for the selection modes that ask for it.
struct SerialIn {
  long long* key;
  unsigned long long* path;
  unsigned char* next;
  int* act;
};

static __device__ __noinline__ int serial_select(const SerialIn& I, int nchild, int K, int want) {
  int na = 0;
  unsigned hashed = 0;
  for (int c = 0; c < nchild; c++) {
    if (I.next[c] != want) continue;
    const long long ks = I.key[c];
    if (na == K && I.key[I.act[na - 1]] <= ks) continue;
    int t = -1;
    for (int h = 0; h < c; h++)
      if (((hashed >> h) & 1u) && I.path[h] == I.path[c]) t = h;
    if (t < 0) {
      hashed |= 1u << c;
    } else {
      if (I.key[t] <= ks) continue;
      for (int i = 0; i < na; i++)
        if (I.act[i] == t) {
          for (int k = i; k + 1 < na; k++) I.act[k] = I.act[k + 1];
          na--;
          break;
        }
    }
    int j = na;   // inserted after every entry with key <= ks; a full list drops its last
    while (j > 0 && I.key[I.act[j - 1]] > ks) j--;
    if (j < K) {
      for (int k = (na < K ? na : K - 1); k > j; k--) I.act[k] = I.act[k - 1];
      I.act[j] = c;
    }
    if (na < K) na++;
  }
  return na;
}

// ring words of one job in shared memory: [2 buffers][W words][KC candidates]
__host__ __device__ inline size_t ring_words(int lat, int KC) {
  return (size_t)2 * ((lat + 31) >> 5) * KC;
}

// the advance of this lane's candidate or child by input x: d and v.  The
// operations that do not wait for one another come first; hook(k) runs behind
// the k-th.
// IM (H = 1): the products on the integer pipe, those with a one at a time in
// the shadow of v's sums.
template <int N, int H, int C, bool IM, typename Hook>
__device__ __forceinline__ void advance(const SdmParams& P, const double (&st)[C], double x, double (&d)[C], double& v,
                                        const double (&gl)[C], const double (&al)[C], double d0, int q,
                                        int lane0, bool zg, Hook&& hook) {
  constexpr bool kPad = H * C > N;
  double sn_q = 0.0, sp_q = 0.0;
  if (H > 1) {
    sn_q = __shfl_down_sync(kFull, d0, 1, H);   // lanes q >= 1: s_0's sum has not moved them
    sp_q = __shfl_up_sync(kFull, st[C - 1], 1, H);
  }
  int k = 0;
  double mm[C], p[C];                       // -m, p
#pragma unroll
  for (int j = 0; j < C; j++) {
    mm[j] = 0.0;
    if (need_g<N, H, C>(j)) {
      const double sn = j < C - 1 ? st[j + 1 < C ? j + 1 : j] : sn_q;
      if (IM) {
        mm[j] = neg(int_mul(P.ig[j], sn));
      } else {
        mm[j] = neg(vmul(gl[j], sn));
        hook(k++);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < C; j++) {
    const bool have = need_g<N, H, C>(j);
    double t1 = j > 0 ? st[j > 0 ? j - 1 : 0] : sp_q;
    if (j == 0 && q == 0) t1 = have ? mm[j] : -0.0;
    if (H == 1 && j == 0 && !have) {
      d[0] = st[0];
    } else {
      d[j] = vadd(st[j], t1);
      hook(k++);
    }
  }
#pragma unroll
  for (int j = 0; j < C; j++) {
    const bool have = need_g<N, H, C>(j);
    const int i = q * C + j;
    if (H == 1 ? j == 0 || (have && j <= N - 2) : j == 0 || have) {
      double t2 = have && (H == 1 || i <= N - 2) ? mm[j] : -0.0;
      if (j == 0 && q == 0) t2 = x;
      d[j] = vadd(d[j], t2);
      hook(k++);
    }
  }
  // the structurally zero products where they may not be left out: written as
  // a loop of no or one pass, which stays a branch (under a predicate, an FP64
  // instruction costs its 64 cycles all the same)
  int nz = zg ? 0 : 1;
  asm volatile("" : "+r"(nz));
#pragma unroll 1
  for (; DSD_RARE(nz > 0); nz--) {
#pragma unroll
    for (int j = 0; j < C; j++) {
      if (need_g<N, H, C>(j)) continue;
      const int i = q * C + j;
      const double m0 = neg(vmul(gl[j], j < C - 1 ? st[j + 1 < C ? j + 1 : j] : sn_q));
      const double t2 = i <= N - 2 ? m0 : -0.0;
      if (j == 0) d[0] = vadd(vadd(st[0], q == 0 ? m0 : sp_q), q == 0 ? x : t2);
      else d[j] = vadd(d[j], t2);
    }
  }
  if (kPad) {
#pragma unroll
    for (int j = 0; j < C; j++)
      if (q * C + j >= N) d[j] = 0.0;
  }
  double acc = x;
  if constexpr (IM) {
    // without g_0 (odd orders) d_0 is 0 on every second step of a silence from rest
    p[0] = need_g<N, H, C>(0) ? int_mul(P.ia[0], d[0]) : int_mul0(P.ia[0], d[0]);
#pragma unroll
    for (int j = 0; j < N; j++) {
      acc = vadd(acc, p[j]);
      if (j + 1 < N) p[j + 1] = int_mul(P.ia[j + 1], d[j + 1]);
      hook(k++);
    }
  } else {
#pragma unroll
    for (int j = 0; j < C; j++) {
      p[j] = vmul(al[j], d[j]);
      hook(k++);
    }
    double pn = H == 1 ? p[0] : __shfl_sync(kFull, p[0], lane0);
#pragma unroll
    for (int i = 0; i < N; i++) {
      const double pi = pn;
      const int i1 = i + 1 < N ? i + 1 : i;
      if (i + 1 < N) pn = H == 1 ? p[i1 % C] : __shfl_sync(kFull, p[i1 % C], lane0 + i1 / C);
      acc = vadd(acc, pi);
      hook(k++);
    }
  }
  v = acc;
}

// (several lanes a child: launches of at most 8 CTAs an SM, which leaves the
// registers to do without spills; 5 s of stereo DSD64 at K = 4 64.2 -> 61.1 ms)
template <int N, int KC, int H, bool IM>
__global__ void __launch_bounds__(32, H == 1 ? 12 : 8)
sdm_child_kernel(const __grid_constant__ SdmParams P, const SdmJob* __restrict__ jobs, int njobs,
                 SdmCtx* __restrict__ ctxs, int* __restrict__ status) {
  constexpr int NC = 2 * KC;            // children
  constexpr int G = NC * H;             // lanes of a job
  constexpr int JPW = 32 / G;           // jobs of a warp
  constexpr int C = (N + H - 1) / H;    // state components of a lane
  __shared__ __align__(16) unsigned s_word[32 / H];
  __shared__ int s_act[32 / H];
  __shared__ long long s_key[32 / H];
  __shared__ unsigned long long s_path[32 / H];
  __shared__ unsigned char s_next[32 / H];
  __shared__ int s_sact[32 / H];
  __shared__ double s_x[JPW][2 * kBlock];
  extern __shared__ uint32_t s_ring[];

  const int wl = threadIdx.x & 31;
  const int js = wl / G, jl = wl % G, jb = js * G;
  const int c = jl / H, q = jl % H, r = c >> 1, b = c & 1;
  const int jid = (int)blockIdx.x * JPW + js;
  const bool has = jid < njobs;
  SdmJob job;
  if (has) {
    job = jobs[jid];
  } else {
    job.in = nullptr; job.out = nullptr; job.n_in = 0; job.skip_out = 0; job.ctx = 0;
    job.copy_from = -1; job.seed_state = nullptr; job.flags = kJobNoStore;
  }
  const SdmCtx* src = &ctxs[job.copy_from >= 0 ? job.copy_from : job.ctx];
  SdmCtx* dst = &ctxs[job.ctx];
  const int K = P.cands, lat = P.lat, W = (lat + 31) >> 5;
  const unsigned long long mask = P.mask;
  const bool lim_on = P.state_limit > 0.0;
  const double lim = P.state_limit;
  const double a0b = b ? -P.a[0] : P.a[0];          // e = v + a0 (bit 0), v - a0 (bit 1)
  const double s0b = q == 0 ? (b ? -1.0 : 1.0) : -0.0;   // s_0 = d_0 +- 1, the others as they are
  const unsigned jobmask = G == 32 ? kFull : (((1u << (G & 31)) - 1u) << jb);
  const unsigned ownmask = (2 * H == 32 ? kFull : ((1u << (2 * H & 31)) - 1u)) << (jb + 2 * H * r);
  const int lane0 = wl - q;                          // the child's first lane
  const bool short_path = P.depth <= 28;             // the match's words hold the whole path

  // this lane's coefficients (constant bank operands where a lane has them all)
  double al[C], gl[C];
#pragma unroll
  for (int j = 0; j < C; j++) {
    if (H == 1) {
      al[j] = P.a[j];
      gl[j] = P.g[j];
    } else {
      al[j] = gl[j] = 0.0;
#pragma unroll
      for (int i = 0; i < N; i++)
        if (i == q * C + j) { al[j] = P.a[i]; gl[j] = P.g[i]; }
    }
  }

  int n = 1, pos = 0, bank0 = 0;
  double s[C], cost = 0.0;
  unsigned long long path = 0;
  int nxt = 0;
  uint32_t cur = 0;
  int buf = 0;
  const size_t rw = ring_words(lat, KC);
  uint32_t* ring = s_ring + (size_t)js * rw;         // [buf][w][r]
#pragma unroll
  for (int j = 0; j < C; j++) s[j] = 0.0;
  if (has) {
    n = src->n;
    bank0 = src->bank;
    pos = src->pos;
    if (r < n) {
#pragma unroll
      for (int j = 0; j < C; j++) {
        const int i = q * C + j;
        if (i < N) s[j] = job.seed_state ? job.seed_state[i] : src->s[r][i];
      }
      cost = job.seed_state ? 0.0 : src->cost[r];    // DAS temp seeding: cost 0
      path = src->path[r];
      nxt = src->next[r];
      cur = src->ring[r][pos >> 5];
    }
  }
  for (int w = jl / KC; w < W; w += G / KC) {
    const int rr = jl % KC;
    ring[w * KC + rr] = (has && rr < n) ? src->ring[rr][w] : 0u;
    ring[(W + w) * KC + rr] = 0u;
  }
  unsigned long long c_conv = 0, c_drop = 0, c_tot = 0, coll_over = 0;
  if (has && job.copy_from < 0) {
    c_conv = src->conv_fail;
    coll_over = src->cands_collapse - src->conv_fail;   // they count together
    c_drop = src->next_filter_drops;
    c_tot = src->total_children;
  }
  int perm = r;   // the candidate this one descends from when the ring's word was entered

  bool int_in = false;   // IM: the states in hand are operands for integer products
  bool zg;        // the structurally zero products may be left out
  {
    bool ok = true;
    for (int i = 0; i < N; i++) {
      const long long a = __double_as_longlong(P.a[i]) & 0x7fffffffffffffffll;
      const long long g = __double_as_longlong(P.g[i]) & 0x7fffffffffffffffll;
      if (a == 0 || a >= 0x7ff0000000000000ll || g >= 0x7ff0000000000000ll) ok = false;
      if (i <= N - 2 && (i & 1) == ((N & 1) ? 0 : 1) && g != 0) ok = false;
    }
#pragma unroll
    for (int j = 0; j < C; j++)
      if (((unsigned)__double2hiint(s[j]) & 0x7ff00000u) == 0x7ff00000u) ok = false;
    zg = __all_sync(kFull, ok);
  }

  constexpr int kOps = advance_ops<N, H, C, IM>();

  const long long n_in = job.n_in;
  long long n_max = n_in;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long m = __shfl_xor_sync(kFull, n_max, o);
    n_max = m > n_max ? m : n_max;
  }
  // inputs: this block's and the next one's in shared memory, the one after
  // that on its way in registers
  constexpr int XL = kBlock / G;
  const double* __restrict__ in = job.in;
  double xr[XL];
  auto load_x = [&](long long t) {
#pragma unroll
    for (int i = 0; i < XL; i++) {
      const long long k = t + i * G + jl;
      xr[i] = (in && k < n_in) ? in[k] : 0.0;
    }
  };
  auto put_x = [&](long long t) {
#pragma unroll
    for (int i = 0; i < XL; i++) s_x[js][(int)(t & kBlock) + i * G + jl] = xr[i];
  };
  load_x(0);
  put_x(0);
  load_x(kBlock);
  double d[C], v = 0.0;
  const bool stored = !(job.flags & kJobNoStore);
  __syncwarp();
  advance<N, H, C, false>(P, s, s_x[js][0], d, v, gl, al, s[0], q, lane0, zg, [](int) {});

  // steps from step t to the next at which a job leaves its ring's word or ends
  auto next_event = [&](long long t) {
    long long e = 1 << 30;
    if (t < n_in) {
      e = min(e, n_in - 1 - t);
      if (W > 1) e = min(e, (long long)(min(pos | 31, lat - 1) - pos));
    }
    return (int)__reduce_min_sync(kFull, (unsigned)e);
  };
  int togo = next_event(0);
  unsigned k_conv = 0, k_drop = 0, k_tot = 0;
  unsigned obits = 0;
  int err = 0;
  double e = vadd(v, a0b);
  // the decisions t0 .. t0 + m - 1 of this lane's job
  auto put_bits = [&](long long t0, int m) {
#pragma unroll
    for (int i = 0; i < XL; i++) {
      const int k = i * G + jl;
      const long long o = t0 + k - job.skip_out;
      if (k < m && o >= 0) job.out[o] = (uint8_t)((obits >> k) & 1u);
    }
  };

  for (long long t0 = 0; t0 < n_max; t0 += kBlock) {
   const int tn = (int)min((long long)kBlock, n_max - t0);
   const int xo = (int)(t0 & kBlock);
   put_x(t0 + kBlock);
   __syncwarp();
   load_x(t0 + 2 * kBlock);
   obits = 0u;
#pragma unroll 1
   for (int tb = 0; tb < tn; tb++) {
    // ---- the children's costs (e: behind the last step's gather) ----
    const double x1 = s_x[js][(xo + tb + 1) & (2 * kBlock - 1)];
    const bool live = r < n;
    const unsigned long long qv = (path << 1) & mask;
    const unsigned livemask = (2 * H * n >= 32 ? kFull : ((1u << (2 * H * n & 31)) - 1u)) << jb;
    // equal paths: the other live candidate with this one's q
    unsigned oth = 0u;
    unsigned long long qo = 0ull;
    if (KC == 2) {
      qo = (unsigned long long)__shfl_xor_sync(kFull, (long long)qv, 2 * H);
    } else {
      const unsigned mv = ((unsigned)qv + (unsigned)(qv >> 32) * 0x85ebca77u) * 2u + (unsigned)js;
      oth = __match_any_sync(kFull, mv);
    }
    const bool fin = ((unsigned)__double2hiint(v) & 0x7ff00000u) != 0x7ff00000u;
    const bool nonfin = __any_sync(kFull, live && !fin);
    // candidates with traceback bit 1
    const int ones = __popc(__ballot_sync(kFull, live && nxt && b == 0 && q == 0) & jobmask);
    if (nonfin) zg = false;
    const double sq = vmul(e, e);
    int next_pos = pos + 1;
    if (next_pos == lat) next_pos = 0;
    const bool event = togo == 0;
    uint32_t wv = cur;
    bool cross = false;
    if (DSD_RARE(event)) {
      cross = t0 + tb < n_in && (next_pos >> 5) != (pos >> 5);
      if (cross) wv = ring[(buf * W + (next_pos >> 5)) * KC + perm];
    }
    const int new_next = (int)((wv >> (next_pos & 31)) & 1u);
    const double costs = vadd(cost, sq);
    int partner = -1;
    bool multi = false, pany = false;
    bool same = false;    // KC = 2: both candidates on one path, with one traceback bit
    if (KC == 2) {
      same = n == 2 && qo == qv && (ones == 0 || ones == 2);
    } else {
      oth &= livemask & ~ownmask;
      const bool twin = live && oth != 0u;
      const unsigned twins = __ballot_sync(kFull, twin);
      // more than a pair (or, of paths longer than the match's words, words
      // that only look equal)
      const unsigned more = __ballot_sync(kFull, twin && __popc(oth) != 2 * H);
      pany = twins != 0u;
      if (DSD_RARE(pany)) {
        multi = more != 0u;
        const int ol = oth ? __ffs(oth) - 1 : wl;
        if (twin) partner = (ol - jb) / (2 * H);
        if (!short_path && shfl_u64(qv, ol) != qv) partner = -1;
      }
    }
#pragma unroll
    for (int j = 0; j < C; j++) s[j] = d[j];
    double first = s[0];
    s[0] = vadd(s[0], s0b);
    if (DSD_RARE(lim_on)) {
      first = clamp_state(first, lim);
#pragma unroll
      for (int j = 0; j < C; j++) s[j] = clamp_state(s[j], lim);
    }

    // ---- selection, beside the children's advance by the next input ----
    const long long key = __double_as_longlong(costs);
    bool valid = live;   // a child that its equal does not beat
    unsigned word = 0u;
    uint4 o[NC / 4];
    int rank = 0, cnt0 = 0, cnt1 = 0, chk = 0, want = 0, n_new = 1, ac = 0, a_first = 0;
    constexpr int kRankParts = NC / 8 > 0 ? NC / 8 : 1;   // eight comparisons behind an operation
    constexpr int kP = 3 + kRankParts;
    auto piece = [&](int k) {
      if (k == 0) {
        word = cost_word(key) | ((unsigned)nxt << 30);
        if (KC == 2) {
          // (as below, without a branch: short paths are often equal at K = 2)
          const long long ko = __shfl_xor_sync(kFull, key, 2 * H);
          if (same && key_less(ko, c ^ 2, key, c)) valid = false;
        } else if (DSD_RARE(pany)) {
          // of a pair with one path and one traceback bit only the first in
          // (cost, index) order can stay in the list
          const int pc = partner >= 0 ? 2 * partner + b : c;
          const long long ko = (long long)shfl_u64((unsigned long long)key, jb + pc * H);
          const int no = __shfl_sync(kFull, nxt, jb + pc * H);
          if (live && partner >= 0 && no == nxt && key_less(ko, pc, key, c)) valid = false;
        }
        if (!valid) word = kWordNone;
        if (q == 0) s_word[wl / H] = word;
        __syncwarp();
      } else if (k == 1) {
        const uint4* wp = reinterpret_cast<const uint4*>(&s_word[js * NC]);
#pragma unroll
        for (int i = 0; i < NC / 4; i++) o[i] = wp[i];
      } else if (k < 2 + kRankParts) {
        const int i = k - 2;
        rank += below4(o[2 * i < NC / 4 ? 2 * i : 0], word);
        if (2 * i + 1 < NC / 4) rank += below4(o[2 * i + 1 < NC / 4 ? 2 * i + 1 : 0], word);
      } else if (k == kP - 1) {
        // children of each bit that stay
        cnt0 = 2 * (n - ones);
        cnt1 = 2 * ones;
        if (KC == 2) {
          if (same) {   // one of each pair
            cnt0 >>= 1;
            cnt1 >>= 1;
          }
        } else if (DSD_RARE(pany)) {
          const unsigned gone = __ballot_sync(kFull, live && !valid && q == 0) & jobmask;
          const unsigned gone1 = __ballot_sync(kFull, live && !valid && q == 0 && nxt) & jobmask;
          cnt0 -= __popc(gone & ~gone1);
          cnt1 -= __popc(gone1);
        }
        if (valid && q == 0) s_act[js * NC + rank] = c;
        __syncwarp();
      } else if (k == kP) {
        if (valid) chk = s_act[js * NC + rank];
        want = ones > 0 ? 1 : 0;
        n_new = min(want ? cnt1 : cnt0, K);
        ac = s_act[js * NC + (want ? cnt0 : 0) + min(r, n_new - 1)];
        a_first = s_act[js * NC + (want ? cnt0 : 0)];
      } else if (k == kP + 1) {
        const bool odd = valid && (chk != c || (unsigned long long)key >= 0x7ff0000000000000ull);
        const bool both = ones > 0 && ones < n;
        if (DSD_RARE(__any_sync(kFull, odd || both || multi || P.mode != kModeFast))) {
          if (DSD_RARE(__any_sync(kFull, odd))) {
            // two equal words (or a cost that is not finite): the whole order
            int lo = 0;
#pragma unroll 1
            for (int i = 0; i < NC; i++) {
              const long long kk = (long long)shfl_u64((unsigned long long)key, jb + i * H);
              const int kf = __shfl_sync(kFull, (valid ? 2 : 0) | nxt, jb + i * H);
              if ((kf & 2) && (kf & 1) == nxt && key_less(kk, i, key, c)) lo++;
            }
            rank = lo + (nxt ? cnt0 : 0);
            __syncwarp();
            if (valid && q == 0) s_act[js * NC + rank] = c;
            __syncwarp();
          }
          // both bits among the candidates: the wanted one is the cheapest
          // child's, or the majority's if its best is within 1.1 of that
          const int b0 = cnt0 > 0 ? s_act[js * NC] : 0;
          const int b1 = cnt1 > 0 ? s_act[js * NC + cnt0] : 0;
          const long long k0 = (long long)shfl_u64((unsigned long long)key, jb + b0 * H);
          const long long k1 = (long long)shfl_u64((unsigned long long)key, jb + b1 * H);
          if (both) {
            const int major = (2 * ones > 2 * n - 2 * ones) ? 1 : 0;
            want = key_less(k0, b0, k1, b1) ? 0 : 1;
            if (want != major &&
                __longlong_as_double(major ? k1 : k0) <
                    __dmul_rn(__longlong_as_double(want ? k1 : k0), 1.1))
              want = major;
          }
          n_new = min(want ? cnt1 : cnt0, K);
          ac = s_act[js * NC + (want ? cnt0 : 0) + min(r, n_new - 1)];
          a_first = s_act[js * NC + (want ? cnt0 : 0)];
          if (DSD_RARE(P.mode != kModeFast || multi)) {
            if (q == 0) {
              s_key[js * NC + c] = key;
              s_path[js * NC + c] = qv | (unsigned long long)b;
              s_next[js * NC + c] = (unsigned char)nxt;
            }
            __syncwarp();
            int ns = 0;
            if (jl == 0) {
              SerialIn I{s_key + js * NC, s_path + js * NC, s_next + js * NC, s_sact + js * NC};
              ns = serial_select(I, 2 * n, K, want);
            }
            __syncwarp();
            ns = __shfl_sync(kFull, ns, jb);
            const int as = s_sact[js * NC + min(r, ns - 1)];
            const int as0 = s_sact[js * NC];
            if (P.mode == kModeVerify && !multi) {
              if (t0 + tb < n_in && (ns != n_new || (r < ns && as != ac))) err = kStatusVerifyMismatch;
            }
            n_new = ns;
            ac = as;
            a_first = as0;
            __syncwarp();
          }
        }
      } else if (k == kP + 2) {
        // candidate r descends from child ac: what the advance does not touch
        const int sl = jb + ac * H;
        const int ab = ac & 1;
        const long long kme = (long long)shfl_u64((unsigned long long)key, sl);
        const long long kmin = (long long)shfl_u64((unsigned long long)key, jb + a_first * H);
        path = shfl_u64(qv, sl) | (unsigned long long)ab;
        const unsigned pn = __shfl_sync(kFull, (unsigned)perm | ((unsigned)new_next << 8), sl);
        const uint32_t cc = __shfl_sync(kFull, cur, sl);
        cost = vadd(__longlong_as_double(kme), neg(__longlong_as_double(kmin)));
        perm = (int)(pn & 0xffu);
        nxt = r < n_new ? (int)(pn >> 8) : 0;
        cur = (cc & ~(1u << (pos & 31))) | ((uint32_t)ab << (pos & 31));
        k_tot += 2u * (unsigned)n;
        k_drop += 2u * (unsigned)(want ? n - ones : ones);
        if (n_new < n) k_conv++;
        n = n_new;
        obits |= (unsigned)want << tb;
      }
    };
    constexpr int kPieces = kP + 3;
    double dn[C], vn;
    advance<N, H, C, IM>(P, s, x1, dn, vn, gl, al, first, q, lane0, zg, [&](int k) {
      if (k < kPieces) piece(k);
    });
#pragma unroll
    for (int k = kOps; k < kPieces; k++) piece(k);
    if (IM) {
      // operands of the integer products (the clamped ones lie between them and
      // the limit): out of range in some lane, and the advance is formed in FP64
      auto in_range = [&]() {
        unsigned w = need_g<N, H, C>(0) ? range_word(dn[0]) : range_word0(dn[0]);
#pragma unroll
        for (int j = 1; j < C; j++) w = max(w, range_word(dn[j]));
        return !__any_sync(kFull, live && w > kRangeSpan);
      };
      bool in = in_range();
      int z = in && int_in ? 0 : 1;
      asm volatile("" : "+r"(z));
#pragma unroll 1
      for (; DSD_RARE(z > 0); z--) {
        advance<N, H, C, false>(P, s, x1, dn, vn, gl, al, first, q, lane0, zg, [](int) {});
        in = in_range();
      }
      int_in = in;
    }

    // ---- commit: the survivors' advance ----
    const int sl = jb + ac * H;
    v = __shfl_sync(kFull, vn, sl);
    e = vadd(v, a0b);
#pragma unroll
    for (int j = 0; j < C; j++) d[j] = __shfl_sync(kFull, dn[j], sl + q);

    // ---- rare: a job's ring enters its next word, or the job ends ----
    if (DSD_RARE(event)) {
      const long long t = t0 + tb;
      double keep[C];
#pragma unroll
      for (int j = 0; j < C; j++) keep[j] = __shfl_sync(kFull, s[j], sl + q);
      if (t < n_in) {
        c_conv += k_conv;
        c_drop += k_drop;
        c_tot += k_tot;
      }
      k_conv = k_drop = k_tot = 0;
      if (cross) {
        // the word is complete: bring the ring's words to their candidates
        for (int w = jl - 2 * H * r; w < W; w += 2 * H)
          ring[((buf ^ 1) * W + w) * KC + r] =
              w == (pos >> 5) ? cur : ring[(buf * W + w) * KC + perm];
      }
      if (t == n_in - 1) {
        put_bits(t0, tb + 1);
        if (stored) {
          if (r < n && b == 0) {
#pragma unroll
            for (int j = 0; j < C; j++)
              if (q * C + j < N) dst->s[r][q * C + j] = keep[j];
            if (q == 0) {
              dst->cost[r] = cost;
              dst->path[r] = path;
              dst->next[r] = (uint8_t)nxt;
              dst->slot[r] = (uint8_t)r;
              for (int w = 0; w < W; w++)
                dst->ring[r][w] = w == (pos >> 5) ? cur : ring[(buf * W + w) * KC + perm];
            }
          }
          if (jl == 0) {
            dst->n = n;
            dst->bank = bank0 ^ (int)(n_in & 1);
            dst->pos = next_pos;
            dst->conv_fail = c_conv;
            dst->cands_collapse = c_conv + coll_over;
            dst->next_filter_drops = c_drop;
            dst->total_children = c_tot;
          }
        }
      }
      __syncwarp();
      if (cross) {
        buf ^= 1;
        perm = r;
        cur = ring[(buf * W + (next_pos >> 5)) * KC + r];
      }
      pos = next_pos;
      togo = next_event(t + 1) + 1;
    }
    pos = next_pos;
    togo--;
   }
   // the block's bits (a job that ended inside it has written its own)
   if (t0 + kBlock <= n_in) {
     put_bits(t0, kBlock);
     c_conv += k_conv;
     c_drop += k_drop;
     c_tot += k_tot;
   }
   k_conv = k_drop = k_tot = 0;
  }

  if (has && job.copy_from >= 0 && stored) {
    for (int i = jl; i < 2 * kSlots; i += G) {
      const int bk = i / kSlots, j = i % kSlots;
      dst->spath[bk][j] = src->spath[bk][j];
      dst->skey[bk][j] = src->skey[bk][j];
      dst->slink[bk][j] = src->slink[bk][j];
    }
  }
  err = __reduce_max_sync(kFull, err);
  if (err && wl == 0) atomicMax(status, err);
}

template <int KC, int H, bool IM = false>
int launch(const SdmParams& P, const SdmJob* d_jobs, int njobs, SdmCtx* d_ctxs, int* d_status,
           cudaStream_t stream) {
  // one lane has all of a child's components: its step is bound by its FP64
  // instructions, and the products go to the integer pipe
  if constexpr (H == 1 && !IM) {
    if (P.int_ok) return launch<KC, H, true>(P, d_jobs, njobs, d_ctxs, d_status, stream);
  }
  const int jpw = 32 / (2 * KC * H);
  const dim3 grid((unsigned)((njobs + jpw - 1) / jpw)), block(32);
  const size_t smem = sizeof(uint32_t) * ring_words(P.lat, KC) * (size_t)jpw;
  switch (P.order) {
#define DSD_CASE(NN)                                                                          \
  case NN:                                                                                    \
    sdm_child_kernel<NN, KC, H, IM><<<grid, block, smem, stream>>>(P, d_jobs, njobs, d_ctxs,  \
                                                                   d_status);                 \
    break;
    DSD_CASE(2) DSD_CASE(3) DSD_CASE(4) DSD_CASE(5) DSD_CASE(6)
    DSD_CASE(7) DSD_CASE(8) DSD_CASE(9) DSD_CASE(10)
#undef DSD_CASE
    default: return -1;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace child

}  // namespace dsdgpu
