/* eval_general.cu - evaluator kernels: several targets or affine statistics. */
#include "eval_kernel.cuh"

namespace sb {
cudaError_t launch_general(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                      const float* tables, cudaStream_t stream) {
    return launch_kind<KIND_GENERAL, false>(batch, prob, geom, plan, partial, tables, stream);
}
cudaError_t configure_general(int smem_limit) { return configure_kind<KIND_GENERAL, false>(smem_limit); }
}  // namespace sb
