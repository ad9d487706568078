/* eval_general_span.cu - evaluator kernels: the same with items that span toggle permutations. */
#include "eval_kernel.cuh"

namespace sb {
cudaError_t launch_general_span(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                      const float* tables, cudaStream_t stream) {
    return launch_kind<KIND_GENERAL, true>(batch, prob, geom, plan, partial, tables, stream);
}
cudaError_t configure_general_span(int smem_limit) { return configure_kind<KIND_GENERAL, true>(smem_limit); }
}  // namespace sb
