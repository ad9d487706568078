/* eval_materialize.cu - evaluator kernels: predictions. */
#include "eval_kernel.cuh"

namespace sb {
cudaError_t launch_materialize(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                      const float* tables, cudaStream_t stream) {
    return launch_kind<KIND_MATERIALIZE, false>(batch, prob, geom, plan, partial, tables, stream);
}
cudaError_t configure_materialize(int smem_limit) { return configure_kind<KIND_MATERIALIZE, false>(smem_limit); }
}  // namespace sb
