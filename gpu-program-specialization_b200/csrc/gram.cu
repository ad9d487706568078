/*
 * gram.cu - cohort statistics of the static Gram shape.
 *
 * The reference's Gram-statistics kernels keep one cohort of up to 32 programs per kernel and
 * accumulate, over all rows, the programs' sums, their full Gram matrix and their cross sums with
 * the targets (projects/secant/secant.h:478-504, host form projects/secant/s_cpu.c:724-848).  Here
 * the runner materializes the predictions of a batch of cohorts for a range of rows with the
 * population evaluator and this kernel reduces them: lanes stride the rows, products rounded before
 * they are added (as the host evaluator does), a fixed-order reduction across the lanes, and one
 * read-modify-write of a statistic by one warp alone - so the result does not depend on scheduling.
 */
#include "evaluator.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace {

/* A warp sums a block of kLeft features x kRight columns, where the columns are the features and then the
 * targets: six loads of a row make eight products, and what the warps of a cohort share stays in the L1 of
 * their SM.  A lane's sums are serial chains over the rows (their order is fixed), so what bounds the
 * kernel is the wait for the loads: kAhead rows are loaded before the first is used.  Blocks wholly below
 * the diagonal are left out; their statistics are those of the mirrored ones, bit for bit.
 * 64 cohorts of eight programs, two targets, 16,384 rows, predictions in L2: 51 us with a warp per
 * statistic, 35 this way (64 with 2 x 4 blocks and six rows ahead). */
constexpr uint32_t kGramWarps = 4, kLeft = 2, kRight = 2, kAhead = 16;

__device__ __host__ __forceinline__ uint32_t first_right_block(uint32_t left_block) { return left_block * kLeft / kRight; }

/* statistics of cohort blockIdx.x: [0, A) sums, [A, A + A*A) Gram matrix row-major,
 * [A + A*A, A + A*A + A*T) cross sums [feature][target]; entries of inactive features stay untouched */
__global__ void __launch_bounds__(kGramWarps * 32)
gram_kernel(const float* __restrict__ predictions, size_t prediction_ld, uint32_t rows, const float* __restrict__ targets,
            size_t targets_ld, uint32_t T, uint32_t A, uint32_t batch_programs, float* statistics, size_t statistics_ld) {
    const uint32_t cohort = blockIdx.x, lane = threadIdx.x & 31u;
    const uint32_t left_blocks = (A + kLeft - 1) / kLeft, right_blocks = (A + T + kRight - 1) / kRight;
    uint32_t block = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), lb = 0;
    for (; lb < left_blocks && block >= right_blocks - first_right_block(lb); ++lb) block -= right_blocks - first_right_block(lb);
    if (lb >= left_blocks) return;
    const uint32_t rb = first_right_block(lb) + block;
    const uint32_t first = cohort * A;
    const uint32_t active = batch_programs - first < A ? batch_programs - first : A;
    if (lb * kLeft >= active) return;
    const float* left[kLeft];
    const float* right[kRight];
#pragma unroll
    for (uint32_t a = 0; a < kLeft; ++a) left[a] = predictions + (size_t)(first + min(lb * kLeft + a, active - 1u)) * prediction_ld;
#pragma unroll
    for (uint32_t b = 0; b < kRight; ++b) { /* a column that is not there repeats another and is not written */
        const uint32_t c = min(rb * kRight + b, A + T - 1u);
        right[b] = c < A ? predictions + (size_t)(first + min(c, active - 1u)) * prediction_ld : targets + (size_t)(c - A) * targets_ld;
    }
    float sum[kLeft] = {}, cross[kLeft][kRight] = {};
    const auto add_row = [&](const float (&x)[kLeft], const float (&y)[kRight]) {
#pragma unroll
        for (uint32_t a = 0; a < kLeft; ++a) {
            sum[a] = __fadd_rn(sum[a], x[a]);
#pragma unroll
            for (uint32_t b = 0; b < kRight; ++b) cross[a][b] = __fadd_rn(cross[a][b], __fmul_rn(x[a], y[b]));
        }
    };
    struct Rows { float x[kAhead][kLeft], y[kAhead][kRight]; };
    const auto load = [&](Rows& v, uint32_t batch) {
        const uint32_t at = batch * (kAhead * 32u) + lane;
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
#pragma unroll
            for (uint32_t a = 0; a < kLeft; ++a) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v.x[k][a]) : "l"(left[a] + at + k * 32u));
#pragma unroll
            for (uint32_t b = 0; b < kRight; ++b) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v.y[k][b]) : "l"(right[b] + at + k * 32u));
        }
    };
    const auto add = [&](const Rows& v) {
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) add_row(v.x[k], v.y[k]);
    };
    const uint32_t batches = rows / (kAhead * 32u);
    Rows even, odd;
    if (batches) load(even, 0);
#pragma unroll 1
    for (uint32_t b = 0; b < batches; b += 2) { /* one batch is on its way while the one before is summed */
        load(odd, min(b + 1u, batches - 1u));
        add(even);
        if (b + 1u >= batches) break;
        load(even, min(b + 2u, batches - 1u));
        add(odd);
    }
    uint32_t r = batches * (kAhead * 32u) + lane;
#pragma unroll 1
    for (; r < rows; r += 32u) {
        float x[kLeft], y[kRight];
#pragma unroll
        for (uint32_t a = 0; a < kLeft; ++a) x[a] = left[a][r];
#pragma unroll
        for (uint32_t b = 0; b < kRight; ++b) y[b] = right[b][r];
        add_row(x, y);
    }
    float* const out = statistics + (size_t)cohort * statistics_ld;
    const auto put = [&](uint32_t s, float v) { out[s] = __fadd_rn(out[s], v); };
#pragma unroll
    for (uint32_t a = 0; a < kLeft; ++a) {
#pragma unroll
        for (int d = 16; d; d >>= 1) {
            sum[a] = __fadd_rn(sum[a], __shfl_xor_sync(0xffffffffu, sum[a], d));
#pragma unroll
            for (uint32_t b = 0; b < kRight; ++b) cross[a][b] = __fadd_rn(cross[a][b], __shfl_xor_sync(0xffffffffu, cross[a][b], d));
        }
        const uint32_t i = lb * kLeft + a;
        if (lane || i >= active) continue;
        if (rb == first_right_block(lb)) put(i, sum[a]);
#pragma unroll
        for (uint32_t b = 0; b < kRight; ++b) {
            const uint32_t j = rb * kRight + b;
            if (j < A) {
                if (j < i || j >= active) continue;
                put(A + i * A + j, cross[a][b]);
                if (j > i) put(A + j * A + i, cross[a][b]);
            } else if (j < A + T) {
                put(A + A * A + i * T + (j - A), cross[a][b]);
            }
        }
    }
}

}  // namespace

namespace sb {

cudaError_t launch_gram(const float* predictions, size_t prediction_ld, uint32_t rows, const float* targets, size_t targets_ld,
                        uint32_t num_targets, uint32_t cohort_size, uint32_t batch_programs, float* statistics, size_t statistics_ld,
                        cudaStream_t stream) {
    const uint32_t cohorts = (batch_programs + cohort_size - 1) / cohort_size;
    uint32_t blocks = 0; /* warps of a cohort */
    for (uint32_t lb = 0; lb * kLeft < cohort_size; ++lb) blocks += (cohort_size + num_targets + kRight - 1) / kRight - first_right_block(lb);
    const uint32_t warps = std::min(blocks, kGramWarps);
    const dim3 grid(cohorts, (blocks + warps - 1) / warps);
    gram_kernel<<<grid, warps * 32, 0, stream>>>(predictions, prediction_ld, rows, targets, targets_ld, num_targets, cohort_size,
                                                 batch_programs, statistics, statistics_ld);
    note_kernel_launches(1);
    return cudaGetLastError();
}

}  // namespace sb
