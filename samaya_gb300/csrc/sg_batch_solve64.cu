// The batched solve in FP64 storage (sg_batch_solve.cuh).
#include "sg_batch_solve.cuh"

namespace sg {

cudaError_t launch_solve64(const BatchView& b, const ClusterPlan& p, int mode, cudaStream_t s) {
  return launch_solve<double>(b, p, mode, s);
}

bool solve64_fits(const ClusterPlan& p, int algorithm) {
  return solve_fits<double>(p, algorithm);
}

}  // namespace sg
