/*
 * gram.cu - cohort statistics of the static Gram shape.
 *
 * The reference's Gram-statistics kernels keep one cohort of up to 32 programs per kernel and
 * accumulate, over all rows, the programs' sums, their full Gram matrix and their cross sums with
 * the targets (projects/secant/secant.h:478-504, host form projects/secant/s_cpu.c:724-848).  Here
 * the runner materializes the predictions of a batch of cohorts for a range of rows with the
 * population evaluator and these kernels reduce them: products rounded before they are added (as the host
 * evaluator does), fixed-order reductions across the threads and across the CTAs of a cluster, and one
 * read-modify-write of a statistic by one thread alone - so the result does not depend on scheduling.
 */
#include "evaluator.cuh"
#include "sbmath.cuh"

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

namespace {

namespace cg = cooperative_groups;
using sbm::f2;

/* A cluster of CTAs shares the rows of a task, which is a block of eight features of a cohort with all the
 * statistics among them and with up to two targets (gram_kernel), or the products of such a block with eight other
 * columns (gram_cross_kernel).  A thread keeps every sum of its task in registers, as pairs of two rows, and reads
 * each value once: eight features and two targets take 56 pair additions and 52 pair products for ten loads, and the
 * predictions come from L2.  The CTAs' sums meet in distributed shared memory, in the order of their ranks.
 * 64 cohorts of eight programs, two targets, 65,536 rows: 140 us for the statistics in four launches with a warp per
 * 2 x 2 block of them, whose lanes added their rows one after the other, 46 in two (predictions not in L2) this way; the
 * call 377 -> 308 us.  50 programs, three targets, 400,001 rows: 1,024 -> 275 us; 3,000 programs of 11,001 rows: no
 * difference, the host decides. */
constexpr uint32_t kThreads = 128, kSplit = 8, kBlock = 8, kTargets = 2, kSums = 64; /* kSplit: the portable cluster size */

/* Sums 64 values over the lanes of a warp in a fixed order: lanes trade halves of what they hold, so that lane l
 * ends with the totals of values 2 l' and 2 l' + 1, l' being l's bits from the highest down. */
__device__ __forceinline__ void warp_totals(float (&v)[kSums], uint32_t lane) {
#pragma unroll
    for (uint32_t d = 16, n = kSums / 2; d; d >>= 1, n >>= 1) {
        const bool upper = lane & d;
#pragma unroll
        for (uint32_t i = 0; i < kSums / 2; ++i)
            if (i < n) {
                const float keep = upper ? v[i + n] : v[i], give = upper ? v[i] : v[i + n];
                v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, d));
            }
    }
}

/* Adds the cluster's totals of `used` values; the CTA of rank 0 hands each to put(value, total) in one thread.  Every thread
 * of the cluster comes here. */
template <class Put>
__device__ __forceinline__ void cluster_totals(float (&v)[kSums], uint32_t used, const Put& put) {
    __shared__ float warps[kThreads / 32][kSums], cta[kSums];
    const uint32_t lane = threadIdx.x & 31u;
    warp_totals(v, lane);
    warps[threadIdx.x >> 5][2 * lane] = v[0];
    warps[threadIdx.x >> 5][2 * lane + 1] = v[1];
    __syncthreads();
    if (threadIdx.x < kSums) {
        float total = warps[0][threadIdx.x];
        for (uint32_t w = 1; w < kThreads / 32; ++w) total = __fadd_rn(total, warps[w][threadIdx.x]);
        cta[threadIdx.x] = total;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x < used) {
        float total = cta[threadIdx.x];
        for (uint32_t r = 1; r < kSplit; ++r) total = __fadd_rn(total, *cluster.map_shared_rank(cta + threadIdx.x, r));
        put(threadIdx.x, total);
    }
    cluster.sync(); /* no CTA leaves while its sums are read */
}

/* Where a column of a task is: predictions lie in columns aligned to four rows (16 bytes), targets anywhere. */
struct Column { const float* at; bool aligned; };

__device__ __forceinline__ void copy_16(uint32_t to, const float* from, uint32_t bytes) { /* what is missing of 16 bytes reads zero */
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_4(uint32_t to, const float* from, uint32_t bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(bytes) : "memory");
}

/* Calls add(x) for every two rows of this CTA's part, rows past its end as zeros.  A thread takes four rows at a time and
 * copies them into shared memory itself, kStages - 1 times ahead, so it waits for nobody else's copies: what bounds the
 * kernel otherwise is the wait for L2 (35 us per 32,768 rows of 64 cohorts with the next two rows in registers, 23 this way). */
constexpr uint32_t kStages = 3;
template <int N, class Add>
__device__ __forceinline__ void walk_rows(const Column (&column)[N], uint32_t rows, uint32_t rank, const Add& add) {
    extern __shared__ __align__(16) unsigned char stages[]; /* [stage][column][thread], 16 bytes each */
    const uint32_t step = 4u * kThreads, part = (rows + kSplit * step - 1) / (kSplit * step) * step;
    const uint32_t begin = rank * part, end = min(rows, begin + part), steps = begin < end ? (end - begin + step - 1) / step : 0u;
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(stages) + threadIdx.x * 16u;
    const auto fetch = [&](uint32_t k) {
        const uint32_t r = begin + k * step + 4u * threadIdx.x, left = r < end ? min(4u, end - r) : 0u, from = left ? r : 0u;
        if (k < steps) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const uint32_t to = mine + ((k % kStages) * N + i) * (kThreads * 16u);
                if (column[i].aligned) copy_16(to, column[i].at + from, left * 4u);
                else {
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) copy_4(to + q * 4u, column[i].at + (q < left ? r + q : 0u), q < left ? 4u : 0u);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory"); /* one group a step, empty ones too */
    };
#pragma unroll
    for (uint32_t k = 0; k + 1 < kStages; ++k) fetch(k);
#pragma unroll 1
    for (uint32_t k = 0; k < steps; ++k) {
        fetch(k + kStages - 1); /* into the place this thread read in the step before */
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        f2 x[N], y[N];
#pragma unroll
        for (int i = 0; i < N; ++i)
            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x[i]), "=l"(y[i]) : "r"(mine + ((k % kStages) * N + i) * (kThreads * 16u)) : "memory");
        add(x);
        add(y);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}
template <int N> constexpr uint32_t stage_bytes() { return kStages * N * kThreads * 16u; }

struct GramProblem {
    const float* predictions;
    size_t prediction_ld;
    const float* targets;
    size_t targets_ld;
    uint32_t rows, T, A, programs; /* of the batch */
    float* statistics;             /* of the batch's first cohort */
    size_t statistics_ld;
};

__device__ __forceinline__ void add_to(float* at, float v) { *at = __fadd_rn(*at, v); }

/* statistics of a cohort: [0, A) sums, [A, A + A*A) Gram matrix row-major, [A + A*A, A + A*A + A*T) cross sums
 * [feature][target]; entries of inactive features stay untouched */

/* feature block blockIdx.y of cohort blockIdx.x / kSplit: its sums, its part of the Gram matrix on the diagonal, its
 * cross sums with the first TT targets */
template <int TT>
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kThreads, 3) gram_kernel(const GramProblem prob) {
    const uint32_t first = blockIdx.x / kSplit * prob.A, active = min(prob.programs - first, prob.A), f0 = blockIdx.y * kBlock;
    if (f0 >= active) return; /* the whole cluster */
    constexpr int N = kBlock + TT;
    Column column[N]; /* one that is not there repeats another and is not written */
#pragma unroll
    for (int i = 0; i < (int)kBlock; ++i) column[i] = Column{prob.predictions + (size_t)(first + min(f0 + i, active - 1u)) * prob.prediction_ld, true};
#pragma unroll
    for (int t = 0; t < TT; ++t) column[kBlock + t] = Column{prob.targets + (size_t)t * prob.targets_ld, false};
    f2 sum[kBlock] = {}, gram[kBlock * (kBlock + 1) / 2] = {}, cross[kBlock * TT] = {};
    walk_rows<N>(column, prob.rows, blockIdx.x % kSplit,
        [&](const f2 (&x)[N]) {
            int k = 0;
#pragma unroll
            for (int i = 0; i < (int)kBlock; ++i) {
                sum[i] = sbm::add2(sum[i], x[i]);
#pragma unroll
                for (int j = i; j < (int)kBlock; ++j, ++k) gram[k] = sbm::add2(gram[k], sbm::mul2(x[i], x[j]));
#pragma unroll
                for (int t = 0; t < TT; ++t) cross[i * TT + t] = sbm::add2(cross[i * TT + t], sbm::mul2(x[i], x[kBlock + t]));
            }
        });
    constexpr int G = kBlock * (kBlock + 1) / 2;
    float v[kSums];
#pragma unroll
    for (int i = 0; i < (int)kSums; ++i) {
        const int g = i - (int)kBlock, c = g - G;
        const f2 p = g < 0 ? sum[i % kBlock] : c < 0 ? gram[g % G] : c < (int)kBlock * TT ? cross[c % (kBlock * TT)] : 0ull;
        v[i] = __fadd_rn(sbm::lo2(p), sbm::hi2(p));
    }
    float* const out = prob.statistics + (size_t)(blockIdx.x / kSplit) * prob.statistics_ld;
    const uint32_t A = prob.A;
    cluster_totals(v, kBlock + G + kBlock * TT, [&](uint32_t at, float total) {
        if (at < kBlock) {
            if (f0 + at < active) add_to(out + f0 + at, total);
            return;
        }
        at -= kBlock;
        if (at < (uint32_t)G) {
            uint32_t i = 0;
            for (; at >= kBlock - i; ++i) at -= kBlock - i;
            const uint32_t left = f0 + i, right = left + at;
            if (right >= active) return;
            add_to(out + A + left * A + right, total);
            if (left != right) add_to(out + A + right * A + left, total);
            return;
        }
        at -= G;
        const uint32_t i = f0 + at / TT;
        if (i < active) add_to(out + A + A * A + i * prob.T + at % TT, total);
    });
}

/* products of a feature block with eight columns it does not hold: a later feature block (the tasks before `pairs`, of
 * `blocks` blocks), or targets from kTargets on */
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kThreads, 2)
gram_cross_kernel(const GramProblem prob, uint32_t blocks, uint32_t pairs) {
    const uint32_t first = blockIdx.x / kSplit * prob.A, active = min(prob.programs - first, prob.A);
    uint32_t lb = 0, rb = blockIdx.y;
    const bool features = rb < pairs;
    if (features) {
        for (; rb >= blocks - 1u - lb; ++lb) rb -= blocks - 1u - lb;
        rb += lb + 1u;
    } else {
        lb = (rb - pairs) % blocks;
        rb = (rb - pairs) / blocks;
    }
    const uint32_t f0 = lb * kBlock, c0 = features ? rb * kBlock : kTargets + rb * kBlock, most = features ? active : prob.T;
    if (f0 >= active || c0 >= most) return;
    constexpr int N = 2 * kBlock;
    Column column[N];
#pragma unroll
    for (int i = 0; i < (int)kBlock; ++i) {
        column[i] = Column{prob.predictions + (size_t)(first + min(f0 + i, active - 1u)) * prob.prediction_ld, true};
        const uint32_t c = min(c0 + i, most - 1u);
        column[kBlock + i] = Column{features ? prob.predictions + (size_t)(first + c) * prob.prediction_ld : prob.targets + (size_t)c * prob.targets_ld, features};
    }
    f2 cross[kSums] = {};
    walk_rows<N>(column, prob.rows, blockIdx.x % kSplit,
        [&](const f2 (&x)[N]) {
#pragma unroll
            for (int i = 0; i < (int)kBlock; ++i)
#pragma unroll
                for (int j = 0; j < (int)kBlock; ++j) cross[i * kBlock + j] = sbm::add2(cross[i * kBlock + j], sbm::mul2(x[i], x[kBlock + j]));
        });
    float v[kSums];
#pragma unroll
    for (int i = 0; i < (int)kSums; ++i) v[i] = __fadd_rn(sbm::lo2(cross[i]), sbm::hi2(cross[i]));
    float* const out = prob.statistics + (size_t)(blockIdx.x / kSplit) * prob.statistics_ld;
    const uint32_t A = prob.A;
    cluster_totals(v, kSums, [&](uint32_t at, float total) {
        const uint32_t i = f0 + at / kBlock, c = c0 + at % kBlock;
        if (i >= active || c >= most) return;
        if (features) {
            add_to(out + A + i * A + c, total);
            add_to(out + A + c * A + i, total);
        } else {
            add_to(out + A + A * A + i * prob.T + c, total);
        }
    });
}

}  // namespace

namespace sb {

cudaError_t configure_gram() {
    cudaError_t e = cudaFuncSetAttribute(gram_kernel<kTargets>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stage_bytes<kBlock + kTargets>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gram_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stage_bytes<kBlock + 1>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gram_cross_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stage_bytes<2 * kBlock>());
    return e;
}

cudaError_t launch_gram(const float* predictions, size_t prediction_ld, uint32_t rows, const float* targets, size_t targets_ld,
                        uint32_t num_targets, uint32_t cohort_size, uint32_t batch_programs, float* statistics, size_t statistics_ld,
                        cudaStream_t stream) {
    const GramProblem prob{predictions, prediction_ld, targets, targets_ld, rows, num_targets, cohort_size, batch_programs, statistics, statistics_ld};
    const uint32_t cohorts = (batch_programs + cohort_size - 1) / cohort_size, blocks = (cohort_size + kBlock - 1) / kBlock;
    const dim3 grid(cohorts * kSplit, blocks);
    if (num_targets >= kTargets) gram_kernel<kTargets><<<grid, kThreads, stage_bytes<kBlock + kTargets>(), stream>>>(prob);
    else if (num_targets == 1) gram_kernel<1><<<grid, kThreads, stage_bytes<kBlock + 1>(), stream>>>(prob);
    else return cudaErrorInvalidValue;
    cudaError_t e = cudaGetLastError();
    const uint32_t pairs = blocks * (blocks - 1) / 2, others = num_targets > kTargets ? (num_targets - kTargets + kBlock - 1) / kBlock : 0u;
    unsigned launches = 1;
    if (e == cudaSuccess && pairs + others) {
        gram_cross_kernel<<<dim3(cohorts * kSplit, pairs + others * blocks), kThreads, stage_bytes<2 * kBlock>(), stream>>>(prob, blocks, pairs);
        e = cudaGetLastError();
        ++launches;
    }
    note_kernel_launches(launches);
    return e;
}

}  // namespace sb
