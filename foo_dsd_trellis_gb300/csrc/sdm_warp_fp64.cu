// The warp trellis kernels (sdm_warp.h) with every product in FP64, for filters
// with a coefficient out of the integer products' range: a resonator at 0 where
// the others have one (the table's odd orders above DSD512 among them), a zero a.
// Formed on the integer pipe first and then in FP64 after all, a step at K = 32,
// order 7 with every g zero took 2.88 us with eight jobs, here 2.47.
#include "sdm_warp.h"

namespace dsdgpu {

int launch_warp_fp64(const SdmParams& P, const WarpLaunch& W, const SdmJob* d_jobs, int njobs, int* d_counter,
                     SdmCtx* d_ctxs, int* d_status, cudaStream_t stream) {
  return launch_warp<false>(P, W, d_jobs, njobs, d_counter, d_ctxs, d_status, stream);
}

int launch_parts_fp64(const SdmParams& P, unsigned blocks, const SdmJob* d_jobs, long long part_len,
                      unsigned long long* d_queue, long long total, SdmCtx* d_ctxs, int* d_status,
                      cudaStream_t stream) {
  return launch_parts<false>(P, blocks, d_jobs, part_len, d_queue, total, d_ctxs, d_status, stream);
}

}  // namespace dsdgpu
