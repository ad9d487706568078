/*
 * evaluator.cu - population evaluator for sm_100a: the constant tables, the fold of the row splits and
 * the choice of kernel.  The evaluator kernel itself is in eval_kernel.cuh and instantiated in eval_*.cu.
 *
 * Replaces the reference's generated-and-patched kernels
 * (projects/secant/s_cubin_generate_toggle_sse.c:339-386, s_cubin_generate_sse.c:461-706,
 * s_cubin_generate_materialize.c:475-540) with one resident kernel family that interprets
 * the encoder's records (record.h).
 *
 * Work decomposition
 *   CTA    = one group of programs x one range of rows.  The CTA stages a tile of
 *            (inputs + targets) x tile_rows floats in shared memory once per chunk and all
 *            its warps read operands from that tile.
 *   warp   = one program at a time, taken from the CTA's queue, so long and short
 *            programs balance inside a CTA.  All 32 lanes execute the same instruction
 *            stream (no divergence); toggles are resolved per permutation by patching
 *            the warp's private copy of the program, not by per-thread selects.
 *   thread = a register tile acc[RR rows][RC banks]; one decoded instruction does
 *            RR*RC FP32 operations.  A column operand costs one 128-bit shared load per
 *            four rows and is reused for all RC coefficient banks; a bank constant is one
 *            broadcast load reused for all RR rows.
 * The squared error is accumulated in registers over the passes of a chunk, reduced
 * with warp shuffles, and added to the caller's output once per (program, configuration,
 * chunk): per-row predictions never reach HBM.
 *
 * Numerics follow the reference HOST evaluator (projects/secant/s_cpu.c:329-352): IEEE
 * add/sub/mul/div/sqrt, accurate sin/cos/exp/log, no flush-to-zero, and no contraction of
 * program-level multiplies and adds (only FMA_F32 fuses).
 */
#include "evaluator.cuh"
#include "sbmath.cuh"

#include <math_constants.h>

namespace sb {

namespace {

/* ---- the bank part: a scalar machine, one lane per coefficient bank ------------------------- */

struct BankSource {
    const float* banks;      /* this program's table, [bank][slot] */
    size_t bank_stride;
    uint32_t num_banks, K, n_affine;
    const SbAffine* affines; /* of this program */
    const float* lits;       /* of this program */
};

template <bool FAST>
__device__ __forceinline__ float scalar_unary(unsigned op, float a) {
    if (op == SB_UN_NEG) return -a;
    if (op == SB_UN_ABS) return fabsf(a);
    if (FAST) return sbm::fast_unary(op, a);
    return sbm::any1(a, op);
}
template <bool FAST>
__device__ __forceinline__ float scalar_binary(unsigned op, float a, float x) {
    switch (op) {
    case SB_BIN_ADD: return __fadd_rn(a, x);
    case SB_BIN_SUB: return __fsub_rn(a, x);
    case SB_BIN_RSUB: return __fsub_rn(x, a);
    case SB_BIN_MUL: return __fmul_rn(a, x);
    case SB_BIN_DIV: return FAST ? sbm::fast_div(a, x) : sbm::div1(a, x);
    case SB_BIN_RDIV: return FAST ? sbm::fast_div(x, a) : sbm::div1(x, a);
    case SB_BIN_MIN: return fminf(a, x);
    default: return fmaxf(a, x);
    }
}

/* The bank part of every program of a batch: what depends on the coefficient bank but not on the row,
 * once per (program, permutation, bank), into the program's constant tables in global memory, laid out
 * [program][permutation][bank group][entry][bank of the group] (cst_off entries before the program's).
 * The evaluator copies the tables of an item into shared memory.  It used to run the bank part itself,
 * for every tile of rows again: 15 % of its instructions on the 64-set population, and 6 KB of code.
 *
 * One warp per 32 (permutation, bank) pairs of a program, permutation-major.  Banks past the table's
 * end are padding and read zeros; temporaries live in shared memory, 32 floats apart.  A toggle site
 * of the bank part carries 1 + its index in the second instruction word; every lane takes the
 * alternative of its own permutation from the program's site list.  The same functions as the tile
 * machine are called, so a value computed here has the bits it would have had in the main part. */
constexpr int kTableWarps = 8;

template <int RC, bool FAST>
__global__ void __launch_bounds__(kTableWarps * 32)
bank_tables_kernel(const DeviceBatch batch, const EvalProblem prob, uint32_t padded_banks, uint32_t chunks, float* __restrict__ tables) {
    extern __shared__ float temporaries[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float* const tmp = temporaries + (size_t)warp * batch.max_btmp * 32;
    const unsigned long long work = (unsigned long long)batch.num_programs * chunks;
    const unsigned long long pairs = prob.mode == EVAL_MATERIALIZE ? padded_banks : (unsigned long long)padded_banks << batch.max_bits;
    const uint32_t first_cst = batch.programs[0].cst_off;
#pragma unroll 1
    for (unsigned long long id = (unsigned long long)blockIdx.x * kTableWarps + warp; id < work; id += (unsigned long long)gridDim.x * kTableWarps) {
        const uint32_t lp = (uint32_t)(id / chunks), chunk = (uint32_t)(id - (unsigned long long)lp * chunks);
        const SbProgram* const hp = batch.programs + lp;
        /* nothing to do without a bank part, or beyond the permutations the program tells apart */
        if (!hp->pre_off || (prob.mode != EVAL_MATERIALIZE && chunk * 32ull >= (unsigned long long)padded_banks << hp->bits)) continue;
        BankSource src;
        src.banks = prob.banks ? prob.banks + (prob.first_program + hp->index) * prob.program_bank_stride : nullptr;
        src.bank_stride = prob.bank_stride;
        src.num_banks = prob.banks ? prob.num_banks : 0u; /* without a table every bank constant reads zero */
        src.K = prob.num_constants;
        src.n_affine = hp->n_affine;
        src.affines = batch.affines + hp->affine_off;
        src.lits = batch.lits + hp->lit_off;
        const SbPatch* const sites = batch.patches + hp->patch_off;
        const uint32_t entries = hp->n_cst;
        const unsigned long long v = (unsigned long long)chunk * 32u + lane;
        const bool live = v < pairs;
        const uint32_t j = (uint32_t)(v / padded_banks), bank = (uint32_t)(v - (unsigned long long)j * padded_banks);
        const uint32_t perm = j; /* numbered by the bits the program reads */
        const bool real = live && bank < src.num_banks;
        float* const mine = tables + (size_t)(hp->cst_off - first_cst) * pairs + ((size_t)j * (padded_banks / RC) + bank / RC) * entries * RC + bank % RC;
        const float* const row = src.banks + (size_t)bank * src.bank_stride;
        auto operand = [&](unsigned kind, uint32_t idx) -> float {
            if (kind == SB_KIND_ROW) return live ? mine[(size_t)idx * RC] : 0.0f;
            if (kind == SB_KIND_SLOT) return tmp[idx * 32 + lane];
            if (idx < src.K) return real ? __ldg(row + idx) : 0.0f;
            if (idx < src.K + src.n_affine) {
                const SbAffine a = src.affines[idx - src.K];
                return real ? __fadd_rn(__fmul_rn(__ldg(row + a.slot), a.scale), a.offset) : 0.0f;
            }
            return __ldg(src.lits + (idx - src.K - src.n_affine));
        };
        const uint2* ip = reinterpret_cast<const uint2*>(batch.insns + hp->insn_off);
        float acc = 0.0f;
#pragma unroll 1
        for (;;) {
            uint2 ins = __ldg(ip++);
            const unsigned cs = ins.x & 0xffu; /* the operation is the same in every alternative of a site */
            if (cs == SB_CASE_END || cs > SB_CASE_FMA) break;
            const bool fma = cs == SB_CASE_FMA, bin = cs >= SB_CASE_BIN && cs < SB_CASE_UN;
            if (!fma && ins.y) { /* a toggle site: this lane's permutation selects the operand */
                const SbPatch* p = sites + (ins.y - 1u);
                unsigned choice = (perm >> p->bit0) & 1u;
                if (p->bit1 != 0xffu) choice |= ((perm >> p->bit1) & 1u) << 1;
                ins.x = p->alt[choice].w0;
            }
            const unsigned mine_cs = ins.x & 0xffu;
            /* operands first, at one site (the fetch is the bulky part): one for loads and binary
             * operations, three for the fused multiply-add, none otherwise */
            float v[3] = {acc, acc, acc};
            const unsigned count = fma ? 3u : (cs < SB_CASE_STORE || bin) ? 1u : 0u;
#pragma unroll 1
            for (unsigned i = 0; i < count; ++i) {
                const unsigned kind = fma ? (ins.x >> (8 + 2 * i)) & 3u : bin ? (mine_cs - SB_CASE_BIN) % SB_NUM_KINDS : mine_cs - SB_CASE_LOAD;
                const uint32_t idx = fma ? (ins.y >> (10 * i)) & 1023u : ins.x >> 16;
                if (kind != SB_FMA_ACC) v[i] = operand(kind, idx);
            }
            const uint32_t idx = ins.x >> 16;
            if (cs < SB_CASE_STORE) acc = v[0];
            else if (cs == SB_CASE_STORE) tmp[idx * 32 + lane] = acc;
            else if (cs == SB_CASE_STOREH) { if (live) mine[(size_t)idx * RC] = acc; }
            else if (bin) acc = scalar_binary<FAST>((cs - SB_CASE_BIN) / SB_NUM_KINDS, acc, v[0]);
            else if (fma) acc = __fmaf_rn(v[0], v[1], v[2]);
            else acc = scalar_unary<FAST>(cs - SB_CASE_UN, acc);
        }
    }
}

/* Adds the per-split partial sums of every (program, quantity, configuration) in split order and
 * writes the total to the caller's grid (only active bins are written: padding keeps its contents). */
__global__ void combine_kernel(const DeviceBatch batch, const EvalProblem prob, const float* __restrict__ partial, uint32_t splits,
                               uint32_t nq, unsigned long long configs) {
    const unsigned long long per_program = (unsigned long long)nq * configs;
    const unsigned long long total = per_program * batch.num_programs;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        float sum = partial[i];
        for (uint32_t s = 1; s < splits; ++s) sum = __fadd_rn(sum, partial[(unsigned long long)s * total + i]);
        const uint32_t lp = (uint32_t)(i / per_program);
        const unsigned long long rem = i % per_program, qn = rem / configs, cfg = rem % configs;
        const size_t gp = prob.first_program + batch.programs[lp].index;
        prob.output[gp * prob.out_program_stride + (size_t)qn * prob.out_target_stride + cfg] = sum;
    }
}

/* The same for a launch that kept the total of every pass ([pass][program][quantity][configuration]): adds them as the rules'
 * cut of the rows would have, the passes of a tile from zero, the tiles of a split, the splits, so the sum has the bits of a
 * launch cut by the rules.  `slots` threads share an output, each with a tile at a time; the thread of slot 0 folds the tiles in
 * order while the others fetch the next ones (two buffers of tile sums, one barrier for every `slots` tiles).  Bound by the
 * latency of its loads, of which a tile has up to eight: they are all started before the first is added, and there are as many
 * slots as the machine has room for threads (128,000 outputs x 157 passes, four slots: 36 us, 52 with loads that wait for
 * each other).  There are fewer totals than 2^32 (planner.cpp). */
struct PassNest { uint32_t tile, split; }; /* passes of a tile, tiles of a split */
constexpr uint32_t kFoldThreads = 256;

__global__ void __launch_bounds__(kFoldThreads)
combine_passes_kernel(const DeviceBatch batch, const EvalProblem prob, const float* __restrict__ partial, uint32_t passes, PassNest before,
                      PassNest others, uint32_t per_program, uint32_t slots) {
    __shared__ float sums[2][kFoldThreads];
    const uint32_t outputs = kFoldThreads / slots, slot = threadIdx.x / outputs;
    const uint32_t total = per_program * batch.num_programs, i = blockIdx.x * outputs + threadIdx.x % outputs;
    const bool live = i < total;
    const uint32_t lp = live ? i / per_program : 0u, within = i - lp * per_program;
    const uint32_t qn = within / prob.num_banks, cfg = within - qn * prob.num_banks;
    /* of a program that reads no coefficient only the first bank group is evaluated, and its first total is every bank's */
    const bool independent = (batch.programs[lp].flags & SB_PROG_BANK_INDEPENDENT) != 0;
    const PassNest nest = lp < batch.first ? before : others;
    const uint32_t tiles = (passes + nest.tile - 1) / nest.tile;
    const uint32_t most = max((passes + before.tile - 1) / before.tile, (passes + others.tile - 1) / others.tile);
    const float* const from = partial + (i - (independent ? cfg : 0u));
    float split = 0.0f, sum = 0.0f;
    uint32_t buffer = 0, in_split = 0;
#pragma unroll 1
    for (uint32_t first = 0; first < most; first += slots, buffer ^= 1u) {
        const uint32_t tile = first + slot;
        if (live && tile < tiles) {
            const uint32_t begin = tile * nest.tile, end = min(passes, begin + nest.tile);
            float v = 0.0f;
#pragma unroll 1
            for (uint32_t p = begin; p < end; p += 8u) {
                float x[8];
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j)
                    if (p + j < end) x[j] = __ldg(from + (size_t)(p + j) * total);
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j)
                    if (p + j < end) v = __fadd_rn(v, x[j]);
            }
            sums[buffer][threadIdx.x] = v;
        }
        __syncthreads();
        if (slot == 0 && live) {
            const uint32_t n = first < tiles ? min(slots, tiles - first) : 0u;
#pragma unroll 4
            for (uint32_t s = 0; s < n; ++s) {
                const float v = sums[buffer][s * outputs + threadIdx.x];
                split = in_split ? __fadd_rn(split, v) : v;
                if (++in_split == nest.split || first + s + 1 == tiles) {
                    sum = first + s < nest.split ? split : __fadd_rn(sum, split);
                    in_split = 0;
                }
            }
        }
    }
    if (slot == 0 && live) prob.output[(prob.first_program + batch.programs[lp].index) * prob.out_program_stride + (size_t)qn * prob.out_target_stride + cfg] = sum;
}

template <int RC>
void launch_tables(const DeviceBatch& batch, const EvalProblem& prob, uint32_t banks, float* tables, cudaStream_t stream) {
    const uint32_t padded = (banks + RC - 1) / RC * RC;
    const unsigned long long pairs = prob.mode == EVAL_MATERIALIZE ? padded : (unsigned long long)padded << batch.max_bits;
    const uint32_t chunks = (uint32_t)((pairs + 31) / 32);
    const unsigned long long work = (unsigned long long)batch.num_programs * chunks;
    const unsigned blocks = (unsigned)std::min<unsigned long long>((work + kTableWarps - 1) / kTableWarps, 148ull * 64ull);
    const size_t smem = (size_t)kTableWarps * batch.max_btmp * 32 * sizeof(float);
    if (prob.fast_math) bank_tables_kernel<RC, true><<<blocks, kTableWarps * 32, smem, stream>>>(batch, prob, padded, chunks, tables);
    else bank_tables_kernel<RC, false><<<blocks, kTableWarps * 32, smem, stream>>>(batch, prob, padded, chunks, tables);
}

}  // namespace

#define SB_FOR_KINDS(X) X(sse) X(sse_span) X(general) X(general_span) X(materialize)
#define SB_DECLARE(NAME) \
    cudaError_t launch_##NAME(const DeviceBatch&, const EvalProblem&, const Geom&, const LaunchPlan&, float*, const float*, cudaStream_t); \
    cudaError_t configure_##NAME(int smem_limit);
cudaError_t configure_gram(); /* gram.cu */
SB_FOR_KINDS(SB_DECLARE) /* eval_*.cu: one file per kind of kernel */

cudaError_t configure_kernels() {
    cudaError_t e;
    int dev = 0, limit = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
#define SB_CONFIGURE(NAME) if ((e = configure_##NAME(limit)) != cudaSuccess) return e;
    SB_FOR_KINDS(SB_CONFIGURE)
    return configure_gram();
}

cudaError_t launch_eval(const DeviceBatch& batch, const EvalProblem& prob, const LaunchPlan& plan, float* partial,
                        cudaStream_t stream, unsigned* launches) {
    Geom geom = make_geom(batch, prob, plan);
    const bool materialize = prob.mode == EVAL_MATERIALIZE;
    float* const tables = partial ? partial + plan.table_offset : nullptr; /* no table entry is used without a buffer for them */
    unsigned launched = 0;
    if (plan.table_elements) {
        const uint32_t banks = materialize ? 1u : prob.num_banks;
        if (plan.variant == 0) launch_tables<4>(batch, prob, banks, tables, stream);
        else if (plan.variant == 1) launch_tables<2>(batch, prob, banks, tables, stream);
        else launch_tables<1>(batch, prob, banks, tables, stream);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        ++launched;
    }
    /* a run whose rows are not split has whole sums: they go straight to the caller's grid */
    geom.direct = !materialize && !plan.pass_sums && plan.row_splits == 1 ? 1u : 0u;
    float* const sums = geom.direct ? prob.output : partial;
    /* runs without toggles have a kernel without the permutations' code: with it inside, the population of
     * 2,048 programs x 64 sets took 34.1 ms instead of 30.0 (registers, not instructions) */
    const bool span = prob.toggle_bits > 0, one_target = prob.mode == EVAL_SSE && prob.num_targets == 1;
    cudaError_t e = materialize ? launch_materialize(batch, prob, geom, plan, sums, tables, stream)
                    : one_target ? (span ? launch_sse_span : launch_sse)(batch, prob, geom, plan, sums, tables, stream)
                                 : (span ? launch_general_span : launch_general)(batch, prob, geom, plan, sums, tables, stream);
    if (e != cudaSuccess) return e;
    *launches = ++launched;
    if (materialize || geom.direct) return cudaSuccess;
    const uint32_t nq = prob.mode == EVAL_AFFINE_STATS ? prob.num_targets + 2u : prob.num_targets;
    const unsigned long long configs = (unsigned long long)prob.num_banks << prob.toggle_bits;
    const unsigned long long total = (unsigned long long)nq * configs * batch.num_programs;
    if (plan.pass_sums) {
        const uint32_t pass = 32u * (uint32_t)kVariantRows[plan.variant], passes = (uint32_t)((prob.num_rows + pass - 1) / pass);
        PassNest nest[2];
        uint32_t most = 1, slots = 1;
        for (int k = 0; k < 2; ++k) {
            nest[k] = PassNest{plan.rules[k].tile_rows / pass, (uint32_t)(plan.rules[k].rows_per_split / plan.rules[k].tile_rows)};
            most = std::max(most, (passes + nest[k].tile - 1) / nest[k].tile);
        }
        while (slots < most && slots < 32u && total * slots < 148ull * 2048ull) slots *= 2;
        const unsigned long long outputs = kFoldThreads / slots;
        combine_passes_kernel<<<(unsigned)((total + outputs - 1) / outputs), kFoldThreads, 0, stream>>>(batch, prob, partial, passes, nest[0], nest[1],
                                                                                                       nq * prob.num_banks, slots);
    } else {
        const unsigned blocks = (unsigned)std::min<unsigned long long>((total + 255) / 256, 148ull * 16ull);
        combine_kernel<<<blocks ? blocks : 1u, 256, 0, stream>>>(batch, prob, partial, plan.row_splits, nq, configs);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) *launches = ++launched;
    return e;
}

}  // namespace sb
