// The batched solve in FP32 storage (sg_batch_solve.cuh).
#include "sg_batch_solve.cuh"

namespace sg {

cudaError_t launch_solve32(const BatchView& b, const ClusterPlan& p, int mode, cudaStream_t s) {
  return launch_solve<float>(b, p, mode, s);
}

bool solve32_fits(const ClusterPlan& p, int algorithm) {
  return solve_fits<float>(p, algorithm);
}

}  // namespace sg
