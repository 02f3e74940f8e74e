// The child-per-lane trellis kernel at K = 5 .. 16 (sdm_child.h): K <= 8 on 32
// or 16 lanes a job, K <= 16 on 32.
#include "sdm_child.h"

namespace dsdgpu {

int launch_sdm_child_large(const SdmParams& P, int lanes, const SdmJob* d_jobs, int njobs,
                           SdmCtx* d_ctxs, int* d_status, cudaStream_t stream) {
  using namespace child;
  if (P.cands <= 8) {
    switch (lanes) {
      case 32: return launch<8, 2>(P, d_jobs, njobs, d_ctxs, d_status, stream);
      case 16: return launch<8, 1>(P, d_jobs, njobs, d_ctxs, d_status, stream);
    }
    return -1;
  }
  return lanes == 32 ? launch<16, 1>(P, d_jobs, njobs, d_ctxs, d_status, stream) : -1;
}

}  // namespace dsdgpu
