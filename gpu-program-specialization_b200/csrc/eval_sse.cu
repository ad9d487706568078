/* eval_sse.cu - evaluator kernels: one target, one permutation per item. */
#include "eval_kernel.cuh"

namespace sb {
cudaError_t launch_sse(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                      const float* tables, cudaStream_t stream) {
    return launch_kind<KIND_SSE, false>(batch, prob, geom, plan, partial, tables, stream);
}
cudaError_t configure_sse(int smem_limit) { return configure_kind<KIND_SSE, false>(smem_limit); }
}  // namespace sb
