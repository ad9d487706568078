/* eval_sse_span.cu - evaluator kernels: one target, items that span toggle permutations. */
#include "eval_kernel.cuh"

namespace sb {
cudaError_t launch_sse_span(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                      const float* tables, cudaStream_t stream) {
    return launch_kind<KIND_SSE, true>(batch, prob, geom, plan, partial, tables, stream);
}
cudaError_t configure_sse_span(int smem_limit) { return configure_kind<KIND_SSE, true>(smem_limit); }
}  // namespace sb
