/*
 * evaluator.cuh - launch interface of the population evaluator kernels (evaluator.cu).
 */
#ifndef SECANT_B200_EVALUATOR_CUH
#define SECANT_B200_EVALUATOR_CUH

#include "../../include/secant_b200.h"
#include "record.h"

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

struct CUmemPoolHandle_st;

namespace sb {
/* adds to the process-wide count reported by secant_b200_kernel_launch_count() */
void note_kernel_launches(unsigned n);

/* The library's memory pool of a device, null when there is none to be had (rk4.cpp); what it keeps
 * goes back to the driver with secant_b200_release_cached_memory(). */
::CUmemPoolHandle_st* record_pool(int device); /* a cudaMemPool_t */

/* Grouped top-k of a [system][configuration] score grid (reduce.cu); scratch may be zero. */
SecantResult grouped_topk(uintptr_t scores, size_t num_systems, size_t num_banks, uint32_t toggle_bits, uint32_t grouping, uint32_t k,
                          uintptr_t winners, uintptr_t counts, uintptr_t scratch, size_t scratch_bytes, cudaStream_t stream);

/* Random pools and winner gathering of the ODE engine interface (pools.cu). */
cudaError_t fill_pool(float* out, unsigned long long size, unsigned long long seed, unsigned long long stream_id,
                      unsigned long long sample_base, bool normal, cudaStream_t stream);
struct GatherProblem {
    const SecantB200Winner* winners;
    const float* banks;                          /* [system][bank][constant], or null when sampled */
    const SecantB200SampledParameter* sampled;   /* [system][constant], or null */
    const float* uniform_pool;
    const float* normal_pool;
    unsigned long long pool_size, entries, configurations, bank_count, score_count;
    unsigned toggle_bits, constants;
    float* rows;                                 /* [entry][constant] */
};
cudaError_t gather_constants(const GatherProblem& problem, cudaStream_t stream);
}

namespace sb {

enum EvalMode : int {
    EVAL_SSE = 0,          /* sum over rows of (prediction - target)^2 per (program, target, configuration) */
    EVAL_MATERIALIZE = 1,  /* prediction per (program, row), one configuration */
    EVAL_AFFINE_STATS = 2  /* sum p, sum p*p, sum p*t per program */
};

/* Device-resident records of one program batch. */
struct DeviceBatch {
    const SbProgram* programs;
    const SbInsn* insns;
    const SbPatch* patches;
    const SbAffine* affines;
    const float* lits;
    uint32_t num_programs;
    uint32_t max_insn;    /* largest instruction count in the batch */
    uint32_t max_extra;   /* largest n_affine + n_lits (rollout records address source constants directly) */
    uint32_t max_slots;   /* largest spill-slot count */
    uint32_t max_hoisted; /* largest number of row-prelude values */
    uint32_t max_cst;     /* largest constant table */
    uint32_t max_btmp;    /* largest number of bank-part temporaries */
    uint32_t uses_scratch; /* some program needs the scratch spill slot */
    uint64_t total_cst;   /* constant-table entries of all programs (an upper bound will do) */
    uint64_t total_cost;  /* scheduling weights of all programs */
    uint64_t max_cost;    /* the largest of them */
    uint64_t main_cost, prelude_cost; /* of all programs: one pass of the main part, and of the row preludes */
    double total_perms;   /* permutations with values of their own, of all programs */
    uint32_t max_bits;    /* most toggle bits a program reads: a program has at most 1 << max_bits of them */
    uint32_t first;       /* the program CTAs begin with; those before it come last */
};

struct EvalProblem {
    int mode;
    const float* input;       /* [column][row] */
    size_t input_ld;
    uint32_t num_inputs;
    const float* targets;     /* [target][row] */
    size_t targets_ld;
    uint32_t num_targets;
    const float* banks;       /* [bank][slot] (+ program * program_bank_stride) */
    size_t bank_stride;
    size_t program_bank_stride;
    size_t first_program;     /* index of the batch's first program within the run */
    uint32_t num_constants;
    uint32_t num_banks;       /* >= 1 */
    uint32_t toggle_bits;
    uint32_t fast_math;       /* 1: approximate division and transcendental functions (see sbmath.cuh) */
    size_t num_rows;
    float* output;
    size_t out_program_stride; /* elements between consecutive programs */
    size_t out_target_stride;  /* elements between consecutive targets  */
};

/* How the planner's rules cut the rows of a launch into tiles and row splits, and with that the order in which rows are added:
 * the passes of a tile from zero, the tiles of a split, the splits. */
struct RowCut {
    uint32_t tile_rows;
    size_t rows_per_split;
};

/* Launch geometry chosen by plan_launch(). */
struct LaunchPlan {
    int variant;              /* rows x banks per thread: 0: 4x4, 1: 8x2, 2: 16x1 */
    uint32_t warps;           /* per CTA */
    uint32_t tile_rows;       /* rows staged per tile, multiple of the pass size */
    uint32_t tile_buffers;    /* 2 when a CTA walks more than one tile: the next tile is fetched while this one is used */
    uint32_t num_groups;      /* CTAs along the programs; group g owns programs g, g + num_groups, ... */
    uint32_t groups_per_item; /* bank groups of one permutation a warp handles per queue item */
    uint32_t perms_per_item;  /* consecutive permutations one item covers (a power of two; above 1 only when an item holds every bank group) */
    uint32_t parts;           /* items that share the rows of a tile, each with a range of its passes */
    uint32_t row_splits;      /* CTAs sharing one program group, each with a row range */
    size_t rows_per_split;
    RowCut rules[2];          /* of the programs before DeviceBatch::first, and of the others */
    bool pass_sums;           /* rows are not cut by the rules: the total of every pass is kept, and added in the rules' order afterwards */
    size_t smem_bytes;
    size_t partial_elements;  /* floats of partial sums over all row splits, or passes (0: materialize) */
    size_t table_elements;    /* floats of constant tables */
    size_t table_offset;      /* where they begin in the launch's scratch, 16-byte aligned: behind the partial sums, or
                                 at 0 when the rows are not split and the sums go straight to the output */
    uint32_t grid_x;
    bool ok;
    bool overflow;            /* !ok because a count does not fit the kernel's 32-bit indices */
};

/* Shared-memory layout and loop bounds of one launch, derived from the plan. */
struct Geom {
    uint32_t tile_rows;       /* floats between consecutive columns of a staged tile */
    uint32_t tile_buffers;
    uint32_t tile_bytes;      /* one buffer */
    uint32_t num_groups;
    uint32_t row_splits;
    uint32_t groups_per_item;
    uint32_t perms_per_item;
    uint32_t parts;
    uint32_t passes_per_part;
    uint32_t exec_bytes;      /* per-warp regions, each a multiple of 16 bytes */
    uint32_t table_bytes;
    uint32_t hoist_bytes;
    uint32_t slot_bytes;
    uint32_t psum_bytes;
    uint32_t warp_bytes;
    uint32_t scratch_slot;    /* spill slot reserved for the element-by-element FMA */
    unsigned long long rows_per_split;
    uint32_t direct;          /* rows are not split: sums go to the output, not to partial sums */
};

constexpr int kNumVariants = 3;
constexpr int kVariantRows[kNumVariants] = {4, 8, 16};
constexpr int kVariantBanks[kNumVariants] = {4, 2, 1};

Geom make_geom(const DeviceBatch& batch, const EvalProblem& problem, const LaunchPlan& plan);

/* scratch_limit: most floats of scratch a launch may use: the row splits are reduced until their partial sums
 * fit beside the constant tables (with one split there are none; the tables are not reduced here).
 * neighbour: what a small launch should know of another that runs beside it; it decides about time, never about the order in
 * which rows are added.
 * rules: of a batch of two kinds of programs (DeviceBatch::first), how each kind's rows are cut when it is launched by itself. */
struct Neighbour {
    enum Kind { NONE, SHARES, LEAVES, FILLS } kind; /* SHARES: it takes the rest of the machine.  LEAVES: it comes first and leaves some SMs, and
                                                       CTAs that do not fit those would hold up its own.  FILLS: it comes first and leaves SMs
                                                       one by one at its end */
    double share;                                   /* the part of the machine to count on */
};
LaunchPlan plan_launch(const DeviceBatch& batch, const EvalProblem& problem, int sm_count, size_t smem_limit,
                       size_t scratch_limit, Neighbour neighbour = Neighbour{Neighbour::NONE, 1.0}, const RowCut* rules = nullptr);
/* The same by the rules alone, without the cut of small launches: its register tile and rules[0] are what a launch adds by. */
LaunchPlan plan_rules(const DeviceBatch& batch, const EvalProblem& problem, int sm_count, size_t smem_limit, size_t scratch_limit);

/* Enqueues the evaluation of one batch on `stream`: the evaluator kernel writes per-split partial
 * sums into `partial` (plan.table_offset + plan.table_elements floats, private to the stream until the
 * launch has finished; the programs' constant tables are computed into its end first) and a second kernel
 * adds them in a fixed order into the output, so a result does not depend on the order CTAs ran in; with one
 * row split the sums are whole and go to the output at once.  With plan.pass_sums the partial sums are those of
 * every pass, and the second kernel adds them as the rules' cut would.  Returns the CUDA status of the launches. */
cudaError_t launch_eval(const DeviceBatch& batch, const EvalProblem& problem, const LaunchPlan& plan, float* partial,
                        cudaStream_t stream, unsigned* launches);

/* Fixed-step RK4 rollout scoring of S-state systems whose right-hand sides are programs. */
struct Rk4Problem {
    uint32_t num_systems, num_states, num_constants, num_banks, toggle_bits;
    const float* banks;            /* [system][bank][slot] */
    size_t bank_stride, system_bank_stride;
    const float* reference;        /* [state][total_points]; a trajectory starts at its first point */
    size_t reference_ld;
    uint32_t num_trajectories, points_per_trajectory, substeps;
    const float* times;            /* [points_per_trajectory], or [total_points] with offsets */
    const uint32_t* offsets;       /* [num_trajectories + 1] partition of total_points, or null */
    uint32_t total_points;         /* concatenated points (both forms) */
    uint32_t allow_missing;        /* NaN reference values after a first point are unobserved */
    int* invalid_flag;             /* device word the validation kernel raises */
    const SecantB200SampledParameter* sampled; /* [system][constant] descriptors, or null: explicit banks */
    const float* uniform_pool;
    const float* normal_pool;
    unsigned long long pool_size;
    float* output;                 /* [system][configuration] */
    size_t output_ld;
    unsigned long long* queue;      /* device counter, zero at launch: the next item to be taken */
    const uint32_t* order;          /* optional [num_systems]: the system whose items are taken k-th (costliest first) */
    unsigned long long* integrated; /* optional device counter: (trajectory, observation interval) pairs integrated */
};
/* Scans the times and reference values once per call and raises *problem.invalid_flag; every launch_rk4()
 * of the call has to come after it. */
cudaError_t launch_rk4_validation(const Rk4Problem& problem, cudaStream_t stream);
/* batch.programs holds num_systems * num_states records, system-major, encoded by
 * rollout_rules(). */
cudaError_t launch_rk4(const DeviceBatch& batch, const Rk4Problem& problem, size_t smem_limit, cudaStream_t stream);

/* Adds the statistics of the static Gram shape for a batch of cohorts over `rows` rows of
 * materialized predictions [program of the batch][prediction_ld] (gram.cu); statistics points at
 * the batch's first cohort. */
cudaError_t launch_gram(const float* predictions, size_t prediction_ld, uint32_t rows, const float* targets, size_t targets_ld,
                        uint32_t num_targets, uint32_t cohort_size, uint32_t batch_programs, float* statistics, size_t statistics_ld,
                        cudaStream_t stream);

/* One-time per-device kernel attribute setup (dynamic shared memory opt-in). */
cudaError_t configure_kernels();

#ifdef __CUDACC__
/* the low bits of v, in order, at the places of mask's bits */
__device__ __forceinline__ uint32_t deposit(uint32_t v, uint32_t mask) {
    uint32_t out = 0u;
#pragma unroll 1
    for (; mask; v >>= 1) {
        const uint32_t low = mask & (0u - mask);
        out |= v & 1u ? low : 0u;
        mask ^= low;
    }
    return out;
}
#endif

}  // namespace sb

#endif
