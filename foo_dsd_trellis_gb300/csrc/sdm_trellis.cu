// Launches of the trellis SDM: which kernel, at which width, for how many jobs.
// The warp kernels are in sdm_warp.h, the child-per-lane ones in sdm_child.h,
// the per-thread one in sdm_scalar.cu.
#include "sdm_warp.h"

#include <algorithm>
#include <cmath>
#include <cstdio>

namespace dsdgpu {

// Fixed rule (the batch plan sizes its job slots with it): a requested width,
// else a whole warp for K > 16 and a half-warp below.
int lanes_per_job(const SdmParams& P) {
  if (P.lat > 32 * kRegRingWords) return 32;   // the wide-ring kernel: one job per warp
  const int lo = min_lanes(P.cands);
  if (P.lanes > 0) return P.lanes > lo ? P.lanes : lo;
  return lo > 16 ? 32 : 16;
}

// Warp slots of the device: 16 one-warp CTAs per SM (128 registers a thread).
static int resident_warps() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 152 * 16;
  if (!cached[dev]) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cached[dev] = (sms > 0 ? sms : 152) * 16;
  }
  return cached[dev];
}

// Lanes and jobs per warp of a launch of njobs jobs with no block cap: the
// tightest width, and the fewest jobs a warp that still let every job start at
// once (warp slots: 16 one-warp CTAs per SM at 32 lanes, 12 below, whose builds
// take up to 168 registers; counted as 10, 1,700 jobs at K = 16 went two a warp,
// order 7 3.47 us a step against 2.63).  The selection's sort is as deep as the
// width asks (21 exchanges at 32 lanes, 15 at 16, 10 at 8), and an FP64
// instruction costs the same with 8 lanes active as with 32, so idle lanes
// beside a job cost nothing while a second job on them costs its FP64 time.
static int launch_lanes(const SdmParams& P, int njobs, int max_blocks, int* groups) {
  int lanes = lanes_per_job(P);
  *groups = 32 / lanes;
  if (P.lanes > 0 || max_blocks > 0 || P.lat > 32 * kRegRingWords) return lanes;
  lanes = min_lanes(P.cands);
  const long long slots = (long long)(resident_warps() / 16) * (lanes == 32 ? 16 : 12);
  *groups = (int)std::min<long long>(32 / lanes, std::max<long long>(1, (njobs + slots - 1) / slots));
  return lanes;
}

// Traceback latencies above 256 (the reference allows up to 2048,
// include/trellis.h:13): the whole 2048-bit ring in registers, one job per
// warp; 8 CTAs per SM leave 255 registers a thread.
template <int N>
__global__ void __launch_bounds__(32, 8)
sdm_jobs_wide_kernel(SdmParams P, const SdmJob* __restrict__ jobs, int njobs,
                     int* __restrict__ job_counter, SdmCtx* __restrict__ ctxs,
                     int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char sdm_smem_raw[];
  WarpSmem<32>& sm = reinterpret_cast<WarpSmem<32>*>(sdm_smem_raw)[0];
  for (;;) {
    int j = 0;
    if ((threadIdx.x & 31) == 0) j = atomicAdd(job_counter, 1);
    j = __shfl_sync(kFull, j, 0);
    if (j >= njobs) break;
    const SdmJob job = jobs[j];
    run_job<N, 32, kRingWords, false>(P, job, ctxs, sm, status);
    __syncwarp();
  }
}

// The kernel (with its template arguments) of this host thread's last SDM
// launch, for callers that report what ran.
static thread_local char g_last_kernel[64] = "";

const char* sdm_last_kernel() { return g_last_kernel; }

static void note_kernel(const char* name, int a, int b = -1, int c = -1) {
  if (c >= 0) snprintf(g_last_kernel, sizeof g_last_kernel, "%s<%d,%d,%d>", name, a, b, c);
  else if (b >= 0) snprintf(g_last_kernel, sizeof g_last_kernel, "%s<%d,%d>", name, a, b);
  else snprintf(g_last_kernel, sizeof g_last_kernel, "%s<%d>", name, a);
}

// The parameters with the coefficients' forms for products on the integer pipe.
static SdmParams with_int(const SdmParams& P) {
  SdmParams Q = P;
  bool ok = P.state_limit == 0.0 || (P.state_limit > 1e-200 && P.state_limit < 1e200);
  for (int i = 0; i < P.order; i++) {
    const bool ga = int_coef(P.a[i], &Q.ia[i]), gg = int_coef(P.g[i], &Q.ig[i]);
    ok = ok && ga;
    if (i <= P.order - 2 && (i & 1) != ((P.order & 1) ? 0 : 1)) ok = ok && gg;
  }
  Q.int_ok = ok ? 1 : 0;
  return Q;
}

__global__ void parts_queue_init_kernel(unsigned long long* queue, long long total, int njobs) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    queue[0] = 0ull;
    queue[1] = (unsigned long long)njobs;
  }
  if (i < total) queue[2 + i] = i < njobs ? (unsigned long long)i : ~0ull;
}

// Warps per sub-partition of a balanced launch of these jobs on `sms` SMs, or
// 0 when the plain launch is kept: K > 16 (a whole warp per job), no width
// or block cap requested, every job on its own context with its state kept,
// and the jobs only slightly above a whole number of warps per pipe (the
// parts of the extra jobs are shared out; a plain launch would give those
// pipes one warp more than the rest for the whole launch).
int sdm_balanced_warps(const SdmParams& P, const SdmJob* jobs, int njobs, int sms,
                       long long part_len) {
  if (P.lanes != 0 || lanes_per_job(P) != 32 || P.lat > 32 * kRegRingWords || sms <= 0) return 0;
  const long long pipes = 4ll * sms;
  if (njobs <= pipes) return 0;
  const long long w = (njobs + pipes - 1) / pipes;   // warps per pipe of the plain launch
  if (w < 2 || w > 4 || njobs % pipes == 0) return 0;
  if ((double)njobs > 1.10 * (double)((w - 1) * pipes)) return 0;
  long long samples = 0;
  for (int i = 0; i < njobs; i++) {
    if (jobs[i].ctx < 0 || (jobs[i].flags & kJobNoStore)) return 0;
    samples += jobs[i].n_in;
  }
  if (samples < 8 * part_len * (long long)njobs) return 0;   // parts too coarse to share out
  return (int)(w - 1);
}

long long sdm_parts_total(const SdmJob* jobs, int njobs, long long part_len) {
  long long total = 0;
  for (int i = 0; i < njobs; i++)
    total += jobs[i].n_in > 0 ? (jobs[i].n_in + part_len - 1) / part_len : 1;
  return total;
}

int launch_sdm_parts(const SdmParams& P0, const SdmJob* d_jobs, int njobs, long long part_len,
                     unsigned long long* d_queue, long long total, int warps_per_pipe, int sms,
                     SdmCtx* d_ctxs, int* d_status, cudaStream_t stream) {
  const SdmParams P = with_int(P0);
  parts_queue_init_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(d_queue, total, njobs);
  note_kernel("sdm_parts_kernel", P.order);
  const unsigned blocks = (unsigned)(4 * warps_per_pipe * sms);
  const int rc = P.int_ok ? launch_parts<true>(P, blocks, d_jobs, part_len, d_queue, total, d_ctxs, d_status, stream)
                          : launch_parts_fp64(P, blocks, d_jobs, part_len, d_queue, total, d_ctxs, d_status, stream);
  if (rc) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int sdm_jobs_per_cta(const SdmParams& P) { return 32 / lanes_per_job(P); }

static int launch_wide(const SdmParams& P, dim3 grid, const SdmJob* d_jobs, int njobs,
                       int* d_counter, SdmCtx* d_ctxs, int* d_status, cudaStream_t stream) {
  const size_t smem = sizeof(WarpSmem<32>);
  switch (P.order) {
#define DSD_CASE(NN)                                                                          \
  case NN:                                                                                    \
    sdm_jobs_wide_kernel<NN><<<grid, 32, smem, stream>>>(P, d_jobs, njobs, d_counter, d_ctxs, \
                                                         d_status);                           \
    break;
    DSD_CASE(2) DSD_CASE(3) DSD_CASE(4) DSD_CASE(5) DSD_CASE(6)
    DSD_CASE(7) DSD_CASE(8) DSD_CASE(9) DSD_CASE(10)
#undef DSD_CASE
    default: return -1;
  }
  return 0;
}

bool sdm_scalar_eligible(const SdmParams& P, int max_blocks);   // sdm_scalar.cu
int launch_sdm_scalar(const SdmParams& P, const SdmJob* d_jobs, int njobs, SdmCtx* d_ctxs,
                      cudaStream_t stream);
int launch_sdm_child_small(const SdmParams& P, int lanes, const SdmJob* d_jobs, int njobs,
                           SdmCtx* d_ctxs, int* d_status, cudaStream_t stream);   // sdm_child_small.cu
int launch_sdm_child_large(const SdmParams& P, int lanes, const SdmJob* d_jobs, int njobs,
                           SdmCtx* d_ctxs, int* d_status, cudaStream_t stream);   // sdm_child_large.cu

// FP64 instructions of a step of the child kernel with H lanes a child: per
// component of a lane the product with g (where a lane has one that is not
// structurally zero), the two sums and the product with a; v; and e, its
// square, the cost, s_0 and the cost's normalisation.
static int child_ops(int N, int H, bool im) {
  const int C = (N + H - 1) / H;
  int m = 0, d = 1;
  for (int j = 0; j < C; j++) {
    bool need = false;
    for (int q = 0; q < H; q++) {
      const int i = q * C + j;
      if (i <= N - 2 && (i & 1) != ((N & 1) ? 0 : 1)) need = true;
    }
    m += need;
    d += need && j > 0;
  }
  return (im ? 0 : m + C) + C + d + N + 5;
}

// Lanes of the child kernel (sdm_child.h) for a launch of njobs jobs without a
// block cap, or 0 for the other kernels.  With w warps a scheduler a step takes
// about 66 cycles an FP64 instruction and 640 to 1,300 more (by lanes a child
// and, at one, whether its products are formed on the integer pipe),
// or 76 w cycles an FP64 instruction (the FP64 unit is the SM's: 19 cycles a
// warp instruction) and 650 more; fewer lanes a job are more instructions a
// step over fewer warps.  Measured cycles a step at order 6, by lanes a job:
//   K = 2:  430 jobs 1,630 / 1,873 / 2,379 at 32 / 16 / 8 lanes,
//           1,722 jobs 4,241 / 2,300 / 2,463 / 2,186 at 32 / 16 / 8 / 4,
//           2,432 jobs 2,530 / 2,193 at 8 / 4, 4,864 jobs 2,252 at 4
//   K = 4:  608 jobs 1,879 / 2,607 at 32 / 16, 1,216 jobs 3,154 / 2,675 / 2,570
//           at 32 / 16 / 8, 4,000 jobs 3,189 at 8
//   K = 8:  1 job 2,396 / 2,507 at 32 / 16, 608 jobs 2,504 / 2,525, 1,216 jobs 4,414 / 2,567
// At K <= 2 the per-thread kernel (32 jobs a warp) is the alternative, from 5
// warps of eight jobs a scheduler on, at K = 1 from 3 (the second wave); us a
// step, child / per-thread kernel:
//   K = 2: order 4 12,000 jobs 1.56 / 3.25, 24,000 3.02 / 3.48, 32,000 4.45 / 4.00;
//          order 6 12,000 2.05 / 3.91, 24,000 3.95 / 4.25; order 8 24,000 4.88 / 5.08
//   K = 1: order 8 12,000 2.53 / 3.79, 18,000 4.86 / 4.05, 24,000 4.88 / 4.86
// At K = 3, 4 there is none: the warp kernel, eight jobs a warp, took 5.8 us at
// 8,000 jobs of order 6 and 12.2 at 20,000, this one 3.6 and 7.2.
// The warp kernel's step (one candidate a lane, its selection in sequence with
// its arithmetic) takes 5,500 cycles alone and 8,925 at order 8 with 2.47 warps
// a scheduler (the child kernel 5,700).
static int child_lanes(const SdmParams& P, int njobs) {
  const int K = P.cands, N = P.order;
  if (K > 16) return 0;
  const double pipes = 4.0 * (resident_warps() / 16);
  auto warps = [&](int jpw) { return (double)((njobs + jpw - 1) / jpw) / pipes; };
  const int KC = K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : 16;
  int best = 0;
  double cost = 1e300;
  for (int lanes = 32; lanes >= 2 * KC; lanes >>= 1) {
    const int H = lanes / (2 * KC);
    const bool im = H == 1 && P.int_ok;
    const double ops = child_ops(N, H, im), w = warps(32 / lanes);
    const double alone = H >= 8 ? 640.0 : H == 4 ? 760.0 : H == 2 ? 1080.0
                         : !im ? 1000.0 : KC == 2 ? 820.0 : 1300.0;
    const double c = std::max(66.0 * ops + alone, 76.0 * ops * w + 650.0);
    if (c < cost) { cost = c; best = lanes; }
  }
  if (K <= 2) return warps(8) > (K == 1 ? 3.0 : 5.0) && sdm_scalar_eligible(P, 0) ? 0 : best;
  double other = 1e300;
  if (K > 4 && P.lat <= 32 * kRegRingWords) {
    const int lanes = min_lanes(K);
    const double slots = pipes / 4.0 * 12.0;
    const int groups = (int)std::min(32.0 / lanes, std::max(1.0, std::ceil(njobs / slots)));
    other = std::max(5500.0, 89.0 * 5.0 * N * warps(groups));
  }
  return other < cost ? 0 : best;
}

// Host-side launcher: each warp-sized CTA of the warp kernel runs 32 / LPJ
// jobs side by side (lanes_per_job); max_blocks caps the CTAs.  Uncapped
// launches at K <= 16 take the child kernel by the rule above, and at K <= 2
// with more jobs than that serves the per-thread kernel (sdm_scalar.cu, the
// fewest FP64 instructions per job).
int launch_sdm_jobs(const SdmParams& P0, const SdmJob* d_jobs, int njobs, int* d_counter,
                    SdmCtx* d_ctxs, int* d_status, int max_blocks, cudaStream_t stream) {
  if (njobs <= 0) return 0;
  const SdmParams P = with_int(P0);
  // (a path-hash walk that gives up early, DSDGPU_FAIL_CHAIN_WALK, is the warp
  // kernel's above K = 4: the child kernel walks no chain)
  if (P.lanes == 0 && max_blocks == 0 && !(P.hop_limit > 0 && P.cands > 4)) {
    const int cl = child_lanes(P, njobs);
    if (cl > 0) {
      const int KC = P.cands <= 2 ? 2 : P.cands <= 4 ? 4 : P.cands <= 8 ? 8 : 16;
      note_kernel("sdm_child_kernel", P.order, KC, cl / (2 * KC));
      return KC <= 4 ? launch_sdm_child_small(P, cl, d_jobs, njobs, d_ctxs, d_status, stream)
                     : launch_sdm_child_large(P, cl, d_jobs, njobs, d_ctxs, d_status, stream);
    }
    if (P.lat <= 32 * kRegRingWords && sdm_scalar_eligible(P, max_blocks)) {
      note_kernel("sdm_scalar_kernel", P.order);
      return launch_sdm_scalar(P, d_jobs, njobs, d_ctxs, stream);
    }
  }
  int groups = 1;
  const int lanes = launch_lanes(P, njobs, max_blocks, &groups);
  const int jpc = groups;
  int blocks = (njobs + jpc - 1) / jpc;
  if (max_blocks > 0 && blocks > max_blocks) blocks = max_blocks;
  cudaMemsetAsync(d_counter, 0, sizeof(int), stream);
  const dim3 grid(blocks);
  int rc = -1;
  if (P.lat > 32 * kRegRingWords) {
    note_kernel("sdm_jobs_wide_kernel", P.order);
    rc = launch_wide(P, grid, d_jobs, njobs, d_counter, d_ctxs, d_status, stream);
    if (rc) return rc;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
  }
  note_kernel("sdm_jobs_kernel", P.order, lanes);
  // the build of 12 CTAs an SM: one job alone 4,986 cycles a step against 5,366;
  // a plan's classes share the SMs, 16 CTAs each (16 mixed streams: 928 ms with 12)
  const WarpLaunch W{lanes, groups, max_blocks == 0 && blocks <= 12 * (resident_warps() / 16), (unsigned)blocks};
  rc = P.int_ok ? launch_warp<true>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, stream)
                : launch_warp_fp64(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, stream);
  if (rc) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace dsdgpu
