// The child-per-lane trellis kernel at K <= 4 (sdm_child.h): K <= 2 on 32, 16,
// 8 or 4 lanes a job, K = 3, 4 on 32, 16 or 8.
#include "sdm_child.h"

namespace dsdgpu {

int launch_sdm_child_small(const SdmParams& P, int lanes, const SdmJob* d_jobs, int njobs,
                           SdmCtx* d_ctxs, int* d_status, cudaStream_t stream) {
  using namespace child;
  if (P.cands <= 2) {
    switch (lanes) {
      case 32: return launch<2, 8>(P, d_jobs, njobs, d_ctxs, d_status, stream);
      case 16: return launch<2, 4>(P, d_jobs, njobs, d_ctxs, d_status, stream);
      case 8: return launch<2, 2>(P, d_jobs, njobs, d_ctxs, d_status, stream);
      case 4: return launch<2, 1>(P, d_jobs, njobs, d_ctxs, d_status, stream);
    }
    return -1;
  }
  switch (lanes) {
    case 32: return launch<4, 4>(P, d_jobs, njobs, d_ctxs, d_status, stream);
    case 16: return launch<4, 2>(P, d_jobs, njobs, d_ctxs, d_status, stream);
    case 8: return launch<4, 1>(P, d_jobs, njobs, d_ctxs, d_status, stream);
  }
  return -1;
}

}  // namespace dsdgpu
