/*
 * eval_kernel.cuh - the population evaluator's kernel template (see evaluator.cu for the family).
 */
#ifndef SECANT_B200_EVAL_KERNEL_CUH
#define SECANT_B200_EVAL_KERNEL_CUH

#include "evaluator.cuh"
#include "pairs_ptx.cuh"
#include "sbmath.cuh"

#include <math_constants.h>

namespace sb {

namespace {

using sbm::f2;

/* FMA_F32 takes three arbitrary operands.  It is rare in scoring workloads, so it runs
 * element by element over shared memory (the caller parks the accumulator in the scratch
 * slot first and reloads it afterwards) instead of being unrolled for every combination of
 * operand kinds.  Nothing here touches the register tile, which therefore stays in
 * registers. */
template <int RR, int RC>
__device__ __noinline__ void fma_over_scratch(uint2 ins, const float* rowp, const float* hrowp, uint32_t tile_ld, const float* cst,
                                              float4* slots, uint32_t scratch_slot) {
    constexpr int V = RR * RC;
    const unsigned kinds = (ins.x >> 8) & 0x3fu;
    float* out = reinterpret_cast<float*>(slots + (size_t)scratch_slot * (V / 4) * 32);
#pragma unroll 1
    for (int k = 0; k < V; ++k) {
        float v[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const unsigned kind = (kinds >> (2 * i)) & 3u;
            const uint32_t index = (ins.y >> (10 * i)) & 1023u;
            const int r = 2 * (k / (2 * RC)) + (k & 1), c = (k >> 1) % RC; /* the tile's storage order: pairs of rows */
            if (kind == SB_KIND_ROW) {
                const float* q = (index & SB_FMA_ROW_HOISTED) ? hrowp + (size_t)(index & (SB_FMA_ROW_HOISTED - 1u)) * (32 * RR)
                                                              : rowp + (size_t)index * tile_ld;
                v[i] = q[(r / 4) * 128 + (r % 4)];
            } else if (kind == SB_KIND_CST) v[i] = cst[index * RC + c];
            else {
                const uint32_t slot = kind == SB_FMA_ACC ? scratch_slot : index;
                v[i] = reinterpret_cast<const float*>(slots + (size_t)slot * (V / 4) * 32)[(k >> 2) * 128 + (k & 3)];
            }
        }
        out[(k >> 2) * 128 + (k & 3)] = __fmaf_rn(v[0], v[1], v[2]);
    }
}

/* ---- the interpreter's core ------------------------------------------------------------------
 *
 * What a warp executes is its private copy of the program with every instruction of the row parts
 * rewritten once per item (rewrite() below): word 0 = the handler of the NEXT instruction (so that the
 * indexed branch's table is read while this one works), word 1 = the operand's byte offset from one of
 * four base addresses.  The handlers are PTX in one block so that three things hold
 * which the compiler does not give: the dispatch is one indexed branch that is known to be uniform (the
 * C++ switch became a tree of about ten compares and ten branches per instruction, with reconvergence
 * barriers around them), every handler leaves the tile in the registers the next one reads it from
 * (the calls of out-of-line functions cost 48 moves each), and the block with the functions is 19 KB,
 * which with what an item needs besides stays inside the instruction cache.  What is rare leaves the
 * block with its handler number and goes through memory (slow()).
 *
 * Measured on 2,048 programs x 64 sets x 131,072 rows, whole call: 58.6 ms with the scalar C++
 * interpreter; pairs in the C++ switch 69.8 (half the arithmetic, but the code no longer fitted the
 * cache); this core with the functions in C++ 46; with the functions in the block 43; with loops instead
 * of unrolled calls for unusual arguments 31.6; sine, cosine and exponential of any argument inside the
 * block 29.3 (sine and cosine had left it from 4,096 on and for NaN, the exponential beyond 86: 2 % of their tiles,
 * which took a sixth of the time; 256 programs x 33 sets x 10,007 rows, where such a program is the last to end,
 * 617 -> 455 us).  Before that, warp instructions 37.3e9 -> 18.4e9, cache hit rate of
 * the fetches 86 -> 98 %. */
enum Handler : uint32_t {
    H_END = 0,
    H_LOAD = 1,            /* + kind below: acc = X */
    H_STORE = 4,
    H_STOREH = 5,
    H_ADD = 6, H_SUB = 9, H_RSUB = 12, H_MUL = 15, /* + kind */
    H_NEG = 18, H_ABS = 19,
    H_DIV = 20, H_RDIV = 23,                       /* + kind: X is fetched, then the block is left */
    H_SIN = 26, H_COS, H_EXP, H_LOG, H_TANH,       /* unusual arguments leave the block; word 1 = SB_UN_* */
    H_UNARY,                                       /* any other function, word 1 = SB_UN_* */
    H_RARE,                                        /* word 1 = the record's word 0 */
    H_NARROW                                       /* + what follows H_DIV, up to H_TANH: the same for the first bank column only */
};
/* Operand kinds are the record's; the offset of a hoisted row value has this bit set, and the handlers
 * of row operands choose between the two bases by it (four handlers less each, one select more). */
constexpr uint32_t kHoistedOffset = 0x80000000u;

/* strides by kind, then of hoisted values: bytes between consecutive operands */
struct OperandStrides { uint32_t of[4]; };

/* by record case: handler in bits 0..7; bits 8..9 the operand's stride, bit 10: word 1 becomes an
 * operand offset (otherwise bits 16..: word 1 itself, or the record's word 0 for H_RARE) */
struct HandlerTable {
    uint32_t entry[SB_NUM_CASES];
    constexpr HandlerTable() : entry() {
        for (unsigned cs = 0; cs < SB_NUM_CASES; ++cs) {
            const bool bin = cs >= SB_CASE_BIN && cs < SB_CASE_UN, load = cs >= SB_CASE_LOAD && cs < SB_CASE_STORE;
            const unsigned rel = bin ? cs - SB_CASE_BIN : cs - SB_CASE_LOAD, kind = rel % SB_NUM_KINDS, op = rel / SB_NUM_KINDS;
            unsigned e = H_RARE;
            if (cs == SB_CASE_END) e = H_END;
            else if (load) e = (H_LOAD + kind) | kind << 8 | 1u << 10;
            else if (cs == SB_CASE_STORE) e = H_STORE | SB_KIND_SLOT << 8 | 1u << 10;
            else if (cs == SB_CASE_STOREH) e = H_STOREH | 3u << 8 | 1u << 10;
            else if (bin && op <= SB_BIN_MUL) e = (H_ADD + 3 * op + kind) | kind << 8 | 1u << 10;
            else if (bin && op <= SB_BIN_RDIV) e = (H_DIV + 3 * (op - SB_BIN_DIV) + kind) | kind << 8 | 1u << 10;
            else if (cs >= SB_CASE_UN && cs < SB_CASE_FMA) {
                const unsigned un = cs - SB_CASE_UN;
                const unsigned h = un == SB_UN_NEG ? H_NEG : un == SB_UN_ABS ? H_ABS : un == SB_UN_SIN ? H_SIN : un == SB_UN_COS ? H_COS
                                 : un == SB_UN_EXP ? H_EXP : un == SB_UN_LOG ? H_LOG : un == SB_UN_TANH ? H_TANH : H_UNARY;
                e = h | un << 16;
            }
            entry[cs] = e;
        }
    }
};
__constant__ HandlerTable kHandlers = HandlerTable();

/* `narrow`: the instruction's values are the same in all bank columns (it belongs to a row prelude, or to a program that
 * does not depend on the coefficients), and only the first column is read in the end: those that have such a form (`all`:
 * divisions and logarithms as well) leave the others as they are. */
__device__ __forceinline__ SbInsn rewrite(SbInsn ins, const OperandStrides& st, bool narrow, bool all) {
    const uint32_t e = kHandlers.entry[ins.w0 & 0xffu], idx = ins.w0 >> 16;
    uint32_t h = e & 0xffu;
    if (narrow && h >= H_DIV && h <= H_TANH && (all || (h >= H_SIN && h <= H_EXP))) h += H_NARROW - H_DIV;
    if (!(e & 1u << 10)) return SbInsn{h, h == H_RARE ? ins.w0 : e >> 16};
    const uint32_t kind = (e >> 8) & 3u;
    if (kind == SB_KIND_ROW && (idx & SB_ROW_HOISTED)) return SbInsn{h, kHoistedOffset | (idx - SB_ROW_HOISTED) * st.of[3]};
    const uint32_t stride = kind == SB_KIND_ROW ? st.of[0] : kind == SB_KIND_CST ? st.of[1] : kind == SB_KIND_SLOT ? st.of[2] : st.of[3];
    return SbInsn{h, idx * stride};
}

/* into a warp's program copy, where an instruction's handler stands in the entry before it */
__device__ __forceinline__ void put_insn(SbInsn* at, SbInsn ins) {
    at[-1].w0 = ins.w0;
    at->w1 = ins.w1;
}

/* asm operands: 0..7 the tile, 8..15 the operand, 16 the address of the next instruction, 17 the
 * next handler and 18 word 1 of this instruction (at the end 17 says whether the run is over, 0, or an
 * instruction was left, 1); 19..22 the bases of dataset columns, hoisted
 * values (less kHoistedOffset), constants and slots for this lane; 23 the pair (-1, -1), 24 the pair (-0, -0),
 * 25 the turns of large arguments (sbmath.cuh). */
#define SB_NEXT "mov.u32 hb, %17;\n ld.shared.v2.u32 {%17, %18}, [%16];\n add.u32 %16, %16, 8;\n"
#define SB_GO "brx.idx.uni hb, targets;\n"
#define SB_AT(BASE) "add.u32 ad, %18, " BASE ";\n"
#define SB_AT_ROW "setp.lt.s32 p, %18, 0;\n selp.b32 ad, %20, %19, p;\n add.u32 ad, ad, %18;\n"
#define SB_ADD8(M0, M1, M2, M3, M4, M5, M6, M7) SB_TWO8("add.rn.f32x2", M0, M1, M2, M3, M4, M5, M6, M7)
#define SB_MUL8(M0, M1, M2, M3, M4, M5, M6, M7) SB_TWO8("mul.rn.f32x2", M0, M1, M2, M3, M4, M5, M6, M7)
#define SB_TWO8(OP, M0, M1, M2, M3, M4, M5, M6, M7)                                                     \
    OP " %0, %0, " M0 ";\n" OP " %1, %1, " M1 ";\n" OP " %2, %2, " M2 ";\n" OP " %3, %3, " M3 ";\n"      \
    OP " %4, %4, " M4 ";\n" OP " %5, %5, " M5 ";\n" OP " %6, %6, " M6 ";\n" OP " %7, %7, " M7 ";\n"
#define SB_SUB8(M0, M1, M2, M3, M4, M5, M6, M7) /* acc - x = x * -1 + acc */                             \
    "fma.rn.f32x2 %0, " M0 ", %23, %0;\n fma.rn.f32x2 %1, " M1 ", %23, %1;\n"                           \
    "fma.rn.f32x2 %2, " M2 ", %23, %2;\n fma.rn.f32x2 %3, " M3 ", %23, %3;\n"                           \
    "fma.rn.f32x2 %4, " M4 ", %23, %4;\n fma.rn.f32x2 %5, " M5 ", %23, %5;\n"                           \
    "fma.rn.f32x2 %6, " M6 ", %23, %6;\n fma.rn.f32x2 %7, " M7 ", %23, %7;\n"
#define SB_RSUB8(M0, M1, M2, M3, M4, M5, M6, M7)                                                         \
    "fma.rn.f32x2 %0, %0, %23, " M0 ";\n fma.rn.f32x2 %1, %1, %23, " M1 ";\n"                           \
    "fma.rn.f32x2 %2, %2, %23, " M2 ";\n fma.rn.f32x2 %3, %3, %23, " M3 ";\n"                           \
    "fma.rn.f32x2 %4, %4, %23, " M4 ";\n fma.rn.f32x2 %5, %5, %23, " M5 ";\n"                           \
    "fma.rn.f32x2 %6, %6, %23, " M6 ";\n fma.rn.f32x2 %7, %7, %23, " M7 ";\n"
/* a pair is copied by adding (-0, -0), which changes no value: one issue slot instead of two moves */
#define SB_COPY(D, S) "add.rn.f32x2 " D ", " S ", %24;\n"
#define SB_MOV8(M0, M1, M2, M3, M4, M5, M6, M7)                                                          \
    SB_COPY("%0", M0) SB_COPY("%1", M1) SB_COPY("%2", M2) SB_COPY("%3", M3) SB_COPY("%4", M4) SB_COPY("%5", M5) SB_COPY("%6", M6) SB_COPY("%7", M7)
/* which register of the fetched operand meets tile pair 0..7, by tile shape and operand kind */
#define SB_MAP_ROW_4(F) F("%8", "%8", "%8", "%8", "%9", "%9", "%9", "%9")
#define SB_MAP_ROW_8(F) F("%8", "%8", "%9", "%9", "%10", "%10", "%11", "%11")
#define SB_MAP_ROW_16(F) F("%8", "%9", "%10", "%11", "%12", "%13", "%14", "%15")
#define SB_MAP_CST_4(F) F("%8", "%9", "%10", "%11", "%8", "%9", "%10", "%11")
#define SB_MAP_CST_8(F) F("%8", "%9", "%8", "%9", "%8", "%9", "%8", "%9")
#define SB_MAP_CST_16(F) F("%8", "%8", "%8", "%8", "%8", "%8", "%8", "%8")
#define SB_MAP_SLOT(F) SB_MAP_ROW_16(F)
#define SB_LD2(A, B, OFF) "ld.shared.v2.b64 {" A ", " B "}, [ad+" OFF "];\n"
#define SB_FETCH_ROW_4 SB_LD2("%8", "%9", "0")
#define SB_FETCH_ROW_8 SB_LD2("%8", "%9", "0") SB_LD2("%10", "%11", "512")
#define SB_FETCH_ROW_16 SB_FETCH_ROW_8 SB_LD2("%12", "%13", "1024") SB_LD2("%14", "%15", "1536")
#define SB_FETCH_CST_4 "ld.shared.v4.b32 {c0, c1, c2, c3}, [ad];\n mov.b64 %8, {c0, c0};\n mov.b64 %9, {c1, c1};\n mov.b64 %10, {c2, c2};\n mov.b64 %11, {c3, c3};\n"
#define SB_FETCH_CST_8 "ld.shared.v2.b32 {c0, c1}, [ad];\n mov.b64 %8, {c0, c0};\n mov.b64 %9, {c1, c1};\n"
#define SB_FETCH_CST_16 "ld.shared.b32 c0, [ad];\n mov.b64 %8, {c0, c0};\n"
#define SB_FETCH_SLOT SB_FETCH_ROW_16
#define SB_STOREH_4 "st.shared.v2.b64 [ad], {%0, %4};\n"
#define SB_STOREH_8 "st.shared.v2.b64 [ad], {%0, %2};\n st.shared.v2.b64 [ad+512], {%4, %6};\n"
#define SB_STOREH_16 "st.shared.v2.b64 [ad], {%0, %1};\n st.shared.v2.b64 [ad+512], {%2, %3};\n st.shared.v2.b64 [ad+1024], {%4, %5};\n st.shared.v2.b64 [ad+1536], {%6, %7};\n"
#define SB_NEG8 SB_TWO8("xor.b64", "m", "m", "m", "m", "m", "m", "m", "m")
#define SB_ABS8 SB_TWO8("and.b64", "m", "m", "m", "m", "m", "m", "m", "m")
/* one operation for the three operand kinds: labels NAME R, C, S */
#define SB_THREE(N, NAME, F)                                                                            \
    NAME "R:\n" SB_AT_ROW SB_FETCH_ROW_##N SB_NEXT SB_MAP_ROW_##N(F) SB_GO                               \
    NAME "C:\n" SB_AT("%21") SB_FETCH_CST_##N SB_NEXT SB_MAP_CST_##N(F) SB_GO                            \
    NAME "S:\n" SB_AT("%22") SB_FETCH_SLOT SB_NEXT SB_MAP_SLOT(F) SB_GO
/* a division fetches its operand over the whole tile first */
#define SB_OVER8_4R SB_COPY("%12", "%9") SB_COPY("%13", "%9") SB_COPY("%14", "%9") SB_COPY("%15", "%9") SB_COPY("%9", "%8") SB_COPY("%10", "%8") SB_COPY("%11", "%8")
#define SB_OVER8_8R SB_COPY("%15", "%11") SB_COPY("%14", "%11") SB_COPY("%13", "%10") SB_COPY("%12", "%10") SB_COPY("%11", "%9") SB_COPY("%10", "%9") SB_COPY("%9", "%8")
#define SB_OVER8_16R ""
#define SB_OVER8_4C SB_COPY("%12", "%8") SB_COPY("%13", "%9") SB_COPY("%14", "%10") SB_COPY("%15", "%11")
#define SB_OVER8_8C SB_COPY("%10", "%8") SB_COPY("%11", "%9") SB_COPY("%12", "%8") SB_COPY("%13", "%9") SB_COPY("%14", "%8") SB_COPY("%15", "%9")
#define SB_OVER8_16C SB_COPY("%9", "%8") SB_COPY("%10", "%8") SB_COPY("%11", "%8") SB_COPY("%12", "%8") SB_COPY("%13", "%8") SB_COPY("%14", "%8") SB_COPY("%15", "%8")
#define SB_DIVISIONS(N)                                                                                 \
    "DR:\n" SB_AT_ROW SB_FETCH_ROW_##N SB_OVER8_##N##R "bra.uni DV;\n"                               \
    "DC:\n" SB_AT("%21") SB_FETCH_CST_##N SB_OVER8_##N##C "bra.uni DV;\n"                            \
    "DS:\n" SB_AT("%22") SB_FETCH_SLOT "bra.uni DV;\n"                                              \
    /* operand / acc: the tile goes to the divisors' place first */                                     \
    "QR:\n" SB_AT_ROW SB_KEEP8 SB_LOADQ_##N SB_MAPQ_ROW_##N "bra.uni DV;\n"                          \
    "QC:\n" SB_AT("%21") SB_KEEP8 SB_LOADQC_##N SB_MAPQ_CST_##N "bra.uni DV;\n"                      \
    "QS:\n" SB_AT("%22") SB_KEEP8 "ld.shared.v2.b64 {%0, %1}, [ad];\n ld.shared.v2.b64 {%2, %3}, [ad+512];\n ld.shared.v2.b64 {%4, %5}, [ad+1024];\n ld.shared.v2.b64 {%6, %7}, [ad+1536];\n bra.uni DV;\n"
#define SB_KEEP8 SB_COPY("%8", "%0") SB_COPY("%9", "%1") SB_COPY("%10", "%2") SB_COPY("%11", "%3") SB_COPY("%12", "%4") SB_COPY("%13", "%5") SB_COPY("%14", "%6") SB_COPY("%15", "%7")
#define SB_LOADQ_4 SB_LD2("%0", "%4", "0")
#define SB_MAPQ_ROW_4 SB_COPY("%1", "%0") SB_COPY("%2", "%0") SB_COPY("%3", "%0") SB_COPY("%5", "%4") SB_COPY("%6", "%4") SB_COPY("%7", "%4")
#define SB_LOADQ_8 SB_LD2("%0", "%2", "0") SB_LD2("%4", "%6", "512")
#define SB_MAPQ_ROW_8 SB_COPY("%1", "%0") SB_COPY("%3", "%2") SB_COPY("%5", "%4") SB_COPY("%7", "%6")
#define SB_LOADQ_16 SB_LD2("%0", "%1", "0") SB_LD2("%2", "%3", "512") SB_LD2("%4", "%5", "1024") SB_LD2("%6", "%7", "1536")
#define SB_MAPQ_ROW_16 ""
#define SB_LOADQC_4 "ld.shared.v4.b32 {c0, c1, c2, c3}, [ad];\n mov.b64 %0, {c0, c0};\n mov.b64 %1, {c1, c1};\n mov.b64 %2, {c2, c2};\n mov.b64 %3, {c3, c3};\n"
#define SB_MAPQ_CST_4 SB_COPY("%4", "%0") SB_COPY("%5", "%1") SB_COPY("%6", "%2") SB_COPY("%7", "%3")
#define SB_LOADQC_8 "ld.shared.v2.b32 {c0, c1}, [ad];\n mov.b64 %0, {c0, c0};\n mov.b64 %1, {c1, c1};\n"
#define SB_MAPQ_CST_8 SB_COPY("%2", "%0") SB_COPY("%4", "%0") SB_COPY("%6", "%0") SB_COPY("%3", "%1") SB_COPY("%5", "%1") SB_COPY("%7", "%1")
#define SB_LOADQC_16 "ld.shared.b32 c0, [ad];\n mov.b64 %0, {c0, c0};\n"
#define SB_MAPQ_CST_16 SB_COPY("%1", "%0") SB_COPY("%2", "%0") SB_COPY("%3", "%0") SB_COPY("%4", "%0") SB_COPY("%5", "%0") SB_COPY("%6", "%0") SB_COPY("%7", "%0")
/* The accurate functions on all eight pairs (pairs_ptx.cuh). */
/* What any argument takes is there once, for the pair in the first place: the pairs go round, c5 of them, or (top bit of c5,
 * only in the 4 x 4 tile) those of its first column change places. */
#define SB_ROTATE "mov.b64 m, %0;\n mov.b64 %0, %1;\n mov.b64 %1, %2;\n mov.b64 %2, %3;\n mov.b64 %3, %4;\n mov.b64 %4, %5;\n mov.b64 %5, %6;\n mov.b64 %6, %7;\n mov.b64 %7, m;\n"
#define SB_AROUND(NAME) SB_ROTATE "sub.u32 c5, c5, 1;\n setp.ne.u32 p, c5, 0;\n @p bra.uni " NAME "L;\n" SB_GO
#define SB_AROUND_4(NAME)                                                                               \
    "setp.lt.s32 p, c5, 0;\n @p bra.uni " NAME "WAP;\n" SB_ROTATE "bra.uni " NAME "ROUND;\n"            \
    NAME "WAP:\n mov.b64 m, %0;\n mov.b64 %0, %4;\n mov.b64 %4, m;\n" NAME "ROUND:\n sub.u32 c5, c5, 1;\n and.b32 c4, c5, 15;\n" \
    "setp.ne.u32 p, c4, 0;\n @p bra.uni " NAME "L;\n" SB_GO
#define SB_EACH(F) F("%0") F("%1") F("%2") F("%3") F("%4") F("%5") F("%6") F("%7")
#define SB_FUNCTIONS(AROUND)                                                                                    \
    "CO:\n" SB_COS_SHIFT "bra.uni SC0;\n SI:\n" SB_SIN_SHIFT                                            \
    "SC0:\n mov.f32 top, 0f00000000;\n" SB_EACH(SB_TOP_NUMBER) "setp.lt.f32 p, top, 0f45800000;\n" SB_VOTE SB_NEXT \
    SB_SIN_CONSTANTS "@!p bra.uni SA;\n" SB_EACH(SB_SIN_PAIR) SB_GO                                     \
    "SA:\n mov.u32 c5, 8;\n SL:\n" SB_SIN_ANY("%0", "%25", "SN") AROUND("S")                           \
    "EX:\n mov.f32 top, 0f00000000;\n" SB_EACH(SB_TOP) "setp.le.f32 p, top, 0f42AC0000;\n" SB_VOTE SB_NEXT \
    SB_EXP_CONSTANTS SB_MINUS_ONE "@!p bra.uni EA;\n" SB_EACH(SB_EXP_PAIR) SB_GO                        \
    "EA:\n mov.u32 c5, 8;\n EL:\n" SB_EXP_ANY("%0") AROUND("E")                                       \
    "TH:\n" SB_NEXT SB_TANH_CONSTANTS SB_MINUS_ONE SB_EACH(SB_TANH_PAIR) SB_GO                          \
    "LG:\n mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n" SB_EACH(SB_TOP) SB_EACH(SB_LOW)       \
    "setp.lt.f32 p, top, 0f7F800000;\n setp.ge.and.f32 p, low, 0f00800000, p;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_LOG_CONSTANTS SB_MINUS_ONE SB_EACH(SB_LOG_PAIR) SB_GO                                            \
    "DV:\n mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n"                                      \
    SB_EACH(SB_TOP_NUMBER) SB_TOP_NUMBER("%8") SB_TOP_NUMBER("%9") SB_TOP_NUMBER("%10") SB_TOP_NUMBER("%11") SB_TOP_NUMBER("%12") SB_TOP_NUMBER("%13") SB_TOP_NUMBER("%14") SB_TOP_NUMBER("%15") \
    SB_EACH(SB_LOW_NUMBER) SB_LOW_NUMBER("%8") SB_LOW_NUMBER("%9") SB_LOW_NUMBER("%10") SB_LOW_NUMBER("%11") SB_LOW_NUMBER("%12") SB_LOW_NUMBER("%13") SB_LOW_NUMBER("%14") SB_LOW_NUMBER("%15") \
    SB_DIV_USUAL "@p bra.uni DW;\n"                                                                     \
    "mov.u32 c2, 0xffffffff;\n" SB_EACH(SB_LEAST) "mov.f32 low, 0f7F800000;\n"                          \
    SB_LOW_NUMBER("%8") SB_LOW_NUMBER("%9") SB_LOW_NUMBER("%10") SB_LOW_NUMBER("%11") SB_LOW_NUMBER("%12") SB_LOW_NUMBER("%13") SB_LOW_NUMBER("%14") SB_LOW_NUMBER("%15") \
    SB_DIV_RANGE SB_ALL_OR_LEAVE "DW:\n" SB_NEXT                                                       \
    SB_DIV_CONSTANTS SB_DIV_PAIR("%0", "%8") SB_DIV_PAIR("%1", "%9") SB_DIV_PAIR("%2", "%10") SB_DIV_PAIR("%3", "%11") \
    SB_DIV_PAIR("%4", "%12") SB_DIV_PAIR("%5", "%13") SB_DIV_PAIR("%6", "%14") SB_DIV_PAIR("%7", "%15") SB_GO

/* The approximate functions: the hardware's, in the forms that flush subnormal numbers where the
 * arguments show that there are none to flush (the other forms scale before and after: 5 to 8
 * instructions per element instead of 1 or 2; both forms give the same bits there, tried for every
 * argument).  The rest leaves the block as above.  1,024 programs x 16 sets x 1,048,583 rows: 27.6 ms with
 * these functions outside the block, 22.2 inside it. */
#define SB_FAST_TWO(OP, A) "mov.b64 {f0, f1}, " A ";\n " OP " f0, f0;\n " OP " f1, f1;\n mov.b64 " A ", {f0, f1};\n"
#define SB_FAST_SIN(A) SB_FAST_TWO("sin.approx.f32", A)
#define SB_FAST_COS(A) SB_FAST_TWO("cos.approx.f32", A)
#define SB_FAST_TANH(A) SB_FAST_TWO("tanh.approx.f32", A)
#define SB_FAST_EXP(A) "mul.rn.f32x2 " A ", " A ", k0;\n" SB_FAST_TWO("ex2.approx.ftz.f32", A)
#define SB_FAST_LOG(A) SB_FAST_TWO("lg2.approx.ftz.f32", A) "mul.rn.f32x2 " A ", " A ", k0;\n"
#define SB_FAST_DIV(A, B) SB_FAST_TWO("rcp.approx.ftz.f32", B) "mul.rn.f32x2 " A ", " A ", " B ";\n"
#define SB_FAST_FUNCTIONS                                                                               \
    "CO:\n" SB_NEXT SB_EACH(SB_FAST_COS) SB_GO                                                          \
    "TH:\n" SB_NEXT SB_EACH(SB_FAST_TANH) SB_GO                                                         \
    "SI:\n" SB_NEXT SB_EACH(SB_FAST_SIN) SB_GO                                                          \
    "EX:\n mov.f32 top, 0f00000000;\n" SB_EACH(SB_TOP) "setp.le.f32 p, top, 0f42AE0000;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_PAIR_CONST("k0", "0x3FB8AA3B3FB8AA3B") SB_EACH(SB_FAST_EXP) SB_GO                                \
    "LG:\n mov.f32 low, 0f7F800000;\n" SB_EACH(SB_LOW) "setp.ge.f32 p, low, 0f00800000;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_PAIR_CONST("k0", "0x3F3172183F317218") SB_EACH(SB_FAST_LOG) SB_GO                                \
    "DV:\n mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n" \
    SB_TOP_NUMBER("%8") SB_TOP_NUMBER("%9") SB_TOP_NUMBER("%10") SB_TOP_NUMBER("%11") SB_TOP_NUMBER("%12") SB_TOP_NUMBER("%13") SB_TOP_NUMBER("%14") SB_TOP_NUMBER("%15") \
    SB_LOW_NUMBER("%8") SB_LOW_NUMBER("%9") SB_LOW_NUMBER("%10") SB_LOW_NUMBER("%11") SB_LOW_NUMBER("%12") SB_LOW_NUMBER("%13") SB_LOW_NUMBER("%14") SB_LOW_NUMBER("%15") \
    "setp.le.f32 p, top, 0f7E800000;\n setp.ge.and.f32 p, low, 0f00800000, p;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_FAST_DIV("%0", "%8") SB_FAST_DIV("%1", "%9") SB_FAST_DIV("%2", "%10") SB_FAST_DIV("%3", "%11")   \
    SB_FAST_DIV("%4", "%12") SB_FAST_DIV("%5", "%13") SB_FAST_DIV("%6", "%14") SB_FAST_DIV("%7", "%15") SB_GO

/* Functions (and, approximate, divisions) of the first bank column of the 4 x 4 tile, pairs 0 and 4: a quarter of the
 * arithmetic for what is the same in all columns.  Of 64 sets' work the row preludes and the programs without
 * coefficients are a tenth, of 16 sets' almost a third: 169 programs x 20 sets x 1,042,866 rows 4.38 -> 4.29 ms, 1,024 x 16
 * x 1,048,583 with approximate functions 21.9 -> 21.3, 470 x 8 x 18,277 168 -> 163 us.  What bounds it is the
 * instruction cache, which the accurate functions fill: with narrow forms of all of them the first took 10 % fewer
 * instructions and 4.62 ms, so sine, cosine and exponential go through the loops that arguments of any size take, and
 * the others stay as they are.  Launches with toggles, whose kernel is the largest, go without (2.77 ms against 2.84). */
#define SB_FIRST(F) F("%0") F("%4")
#define SB_NARROW_TARGETS_4 ", NDR, NDC, NDS, NQR, NQC, NQS, NSI, NCO, NEX, NLG, NTH"
#define SB_NARROW_TARGETS_8 ""
#define SB_NARROW_TARGETS_16 ""
#define SB_NARROW_DIVISIONS                                                                             \
    "NDR:\n" SB_AT_ROW SB_LD2("%8", "%12", "0") "bra.uni NDV;\n"                                       \
    "NDC:\n" SB_AT("%21") "ld.shared.b32 c0, [ad];\n mov.b64 %8, {c0, c0};\n mov.b64 %12, {c0, c0};\n bra.uni NDV;\n" \
    "NDS:\n" SB_AT("%22") "ld.shared.b64 %8, [ad];\n ld.shared.b64 %12, [ad+1024];\n bra.uni NDV;\n"   \
    "NQR:\n" SB_AT_ROW SB_COPY("%8", "%0") SB_COPY("%12", "%4") SB_LD2("%0", "%4", "0") "bra.uni NDV;\n" \
    "NQC:\n" SB_AT("%21") SB_COPY("%8", "%0") SB_COPY("%12", "%4") "ld.shared.b32 c0, [ad];\n mov.b64 %0, {c0, c0};\n mov.b64 %4, {c0, c0};\n bra.uni NDV;\n" \
    "NQS:\n" SB_AT("%22") SB_COPY("%8", "%0") SB_COPY("%12", "%4") "ld.shared.b64 %0, [ad];\n ld.shared.b64 %4, [ad+1024];\n bra.uni NDV;\n"
#define SB_NARROW_ACCURATE                                                                              \
    "NCO:\n" SB_COS_SHIFT "bra.uni NS0;\n NSI:\n" SB_SIN_SHIFT "NS0:\n" SB_NEXT SB_SIN_CONSTANTS "mov.u32 c5, 0x80000002;\n bra.uni SL;\n" \
    "NEX:\n" SB_NEXT SB_EXP_CONSTANTS SB_MINUS_ONE "mov.u32 c5, 0x80000002;\n bra.uni EL;\n"            \
    "NDR: NDC: NDS: NQR: NQC: NQS: NLG: NTH: bra.uni LEAVE;\n"
#define SB_NARROW_FAST                                                                                  \
    SB_NARROW_DIVISIONS                                                                                 \
    "NCO:\n" SB_NEXT SB_FIRST(SB_FAST_COS) SB_GO "NTH:\n" SB_NEXT SB_FIRST(SB_FAST_TANH) SB_GO "NSI:\n" SB_NEXT SB_FIRST(SB_FAST_SIN) SB_GO \
    "NEX:\n mov.f32 top, 0f00000000;\n" SB_FIRST(SB_TOP) "setp.le.f32 p, top, 0f42AE0000;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_PAIR_CONST("k0", "0x3FB8AA3B3FB8AA3B") SB_FIRST(SB_FAST_EXP) SB_GO                               \
    "NLG:\n mov.f32 low, 0f7F800000;\n" SB_FIRST(SB_LOW) "setp.ge.f32 p, low, 0f00800000;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_PAIR_CONST("k0", "0x3F3172183F317218") SB_FIRST(SB_FAST_LOG) SB_GO                               \
    "NDV:\n mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n" SB_TOP_NUMBER("%8") SB_TOP_NUMBER("%12") SB_LOW_NUMBER("%8") SB_LOW_NUMBER("%12") \
    "setp.le.f32 p, top, 0f7E800000;\n setp.ge.and.f32 p, low, 0f00800000, p;\n" SB_ALL_OR_LEAVE SB_NEXT \
    SB_FAST_DIV("%0", "%8") SB_FAST_DIV("%4", "%12") SB_GO

#define SB_CORE(N, FUNCTIONS)                                                                           \
    "{\n" SB_PTX_REGISTERS SB_PTX_REGISTERS_ANY                                                        \
    ".reg .u32 hb;\n targets: .branchtargets EN, LR, LC, LS, ST, SH, AR, AC, AS, SR, SC, SS, RR, RC, RS, MR, MC, MS, NG, AB, " \
    "DR, DC, DS, QR, QC, QS, SI, CO, EX, LG, TH, LEAVE, LEAVE" SB_NARROW_TARGETS_##N ";\n"                                           \
    "ld.shared.u32 %17, [%16+-8];\n" SB_NEXT SB_GO                                                       \
    SB_THREE(N, "L", SB_MOV8) SB_THREE(N, "A", SB_ADD8) SB_THREE(N, "S", SB_SUB8) SB_THREE(N, "R", SB_RSUB8) \
    SB_THREE(N, "M", SB_MUL8) SB_DIVISIONS(N)                                                           \
    "ST:\n" SB_AT("%22") SB_NEXT "st.shared.v2.b64 [ad], {%0, %1};\n st.shared.v2.b64 [ad+512], {%2, %3};\n st.shared.v2.b64 [ad+1024], {%4, %5};\n st.shared.v2.b64 [ad+1536], {%6, %7};\n" SB_GO \
    "SH:\n add.u32 ad, %18, %20;\n xor.b32 ad, ad, 0x80000000;\n" SB_NEXT SB_STOREH_##N SB_GO           \
    "NG:\n mov.b64 m, 0x8000000080000000;\n" SB_NEXT SB_NEG8 SB_GO                                       \
    "AB:\n mov.b64 m, 0x7fffffff7fffffff;\n" SB_NEXT SB_ABS8 SB_GO                                       \
    FUNCTIONS "EN:\n mov.u32 %17, 0;\n bra.uni OUT;\n LEAVE:\n mov.u32 %17, 1;\n OUT:\n }"

/* The tile is kept as pairs of rows (sbmath.cuh, f2): acc[h][c] holds rows 2h and 2h + 1 of bank column
 * c.  A ROW operand arrives as pairs straight from its 128-bit loads; a CST operand is doubled in
 * registers. */
template <int RR, int RC, bool FAST = false>
struct Machine {
    static constexpr int V = RR * RC;
    static constexpr int HR = RR / 2;         /* row pairs */
    static constexpr int PASS = 32 * RR;      /* rows one warp covers per pass */
    static constexpr int GROUPS = RR / 4;     /* float4 row groups per thread */

    f2 acc[HR][RC];

    static __device__ __forceinline__ f2 load2(uint32_t address, f2& second) {
        f2 first;
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(first), "=l"(second) : "r"(address) : "memory");
        return first;
    }

    /* one float per row of a column, from a shared-memory address */
    __device__ __forceinline__ void fetch_column(uint32_t address, f2 (&x)[HR]) const {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) x[2 * g] = load2(address + g * 512, x[2 * g + 1]);
    }
    /* one float per row, starting at the thread's first row of a column laid out [row of the pass] */
    __device__ __forceinline__ void fetch_column(const float* q, f2 (&x)[HR]) const {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(q + g * 128);
            x[2 * g] = v.x;
            x[2 * g + 1] = v.y;
        }
    }
    /* ROW operand: a dataset column of the staged tile, or (SB_ROW_HOISTED) a value the row prelude
     * left in the warp's hoist buffer, which holds PASS floats per value */
    __device__ __forceinline__ void fetch_row(const float* rowp, const float* hrowp, uint32_t tile_ld, uint32_t col,
                                              f2 (&x)[HR]) const {
        const float* q = (col & SB_ROW_HOISTED) ? hrowp + (size_t)(col & (SB_ROW_HOISTED - 1u)) * PASS : rowp + (size_t)col * tile_ld;
        fetch_column(q, x);
    }
    __device__ __forceinline__ void fetch_cst(const float* cst, uint32_t entry, f2 (&x)[RC]) const {
        const float* q = cst + entry * RC;
        if (RC == 4) {
            const float4 v = *reinterpret_cast<const float4*>(q);
            x[0] = sbm::both2(v.x); x[1 % RC] = sbm::both2(v.y); x[2 % RC] = sbm::both2(v.z); x[3 % RC] = sbm::both2(v.w);
        } else if (RC == 2) {
            const float2 v = *reinterpret_cast<const float2*>(q);
            x[0] = sbm::both2(v.x); x[1 % RC] = sbm::both2(v.y);
        } else {
            x[0] = sbm::both2(q[0]);
        }
    }
    /* Slot s of this warp: V/4 16-byte vectors per lane, lane-interleaved (conflict free). */
    __device__ __forceinline__ void fetch_slot(const float4* slots, uint32_t s, f2 (&x)[HR][RC]) const {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(slots + (size_t)s * (V / 4) * 32);
        f2* flat = &x[0][0];
#pragma unroll
        for (int j = 0; j < V / 4; ++j) {
            const ulonglong2 v = q[j * 32];
            flat[2 * j] = v.x;
            flat[2 * j + 1] = v.y;
        }
    }
    __device__ __forceinline__ void store_slot(float4* slots, uint32_t s) const {
        ulonglong2* q = reinterpret_cast<ulonglong2*>(slots + (size_t)s * (V / 4) * 32);
        const f2* flat = &acc[0][0];
#pragma unroll
        for (int j = 0; j < V / 4; ++j) q[j * 32] = make_ulonglong2(flat[2 * j], flat[2 * j + 1]);
    }

    /* approximate functions of what the core leaves (sine, cosine and tanh it never does): a few
     * instructions per element, unrolled in place */
    __device__ __forceinline__ void fast_unary(unsigned op, f2 (&v)[8]) {
        switch (op) {
        case SB_UN_EXP: fast_tile<SB_UN_EXP>(v); break;
        case SB_UN_LOG: fast_tile<SB_UN_LOG>(v); break;
        case SB_UN_EX2: fast_tile<SB_UN_EX2>(v); break;
        default:
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = sbm::pack2(sbm::fast_unary(op, sbm::lo2(v[i])), sbm::fast_unary(op, sbm::hi2(v[i])));
        }
    }
    template <unsigned OP>
    static __device__ __forceinline__ void fast_tile(f2 (&v)[8]) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) v[i] = sbm::pack2(sbm::fast_unary(OP, sbm::lo2(v[i])), sbm::fast_unary(OP, sbm::hi2(v[i])));
    }

    /* Shared-memory addresses of a warp's working set, as the core takes them (32 bits, this lane's part
     * added where lanes differ) and what the rare operations need besides. */
    struct Place {
        uint32_t exec, row, hoist, table, slots; /* program copy; first row of the pass; hoisted values; an item's tables; spill slots */
        uint32_t tile_ld, scratch_slot;
        const SbInsn* code;                      /* the program as the host made it */
    };
    template <class T> static __device__ __forceinline__ T* generic(uint32_t address) {
        return reinterpret_cast<T*>(__cvta_shared_to_generic(address));
    }

    /* What the core leaves to others, through memory, so that the call costs the common path no register
     * moves: e[0..15] is the tile and receives the result, e[16..31] the divisors of a division. */
    __device__ __noinline__ static void slow(float* e, const Place& place, uint32_t h, uint32_t w, uint32_t ip, uint32_t cst) {
        if (h < H_UNARY) { sbm::mend_tile(reinterpret_cast<f2*>(e), h < H_SIN ? sbm::kDivide : w); return; }
        if (h == H_UNARY) { sbm::rare_tile(e, w); return; }
        Machine m;
        f2 (&a)[8] = reinterpret_cast<f2(&)[8]>(m.acc);
        f2* const t = reinterpret_cast<f2*>(e);
        const float *rowp = generic<float>(place.row), *hrowp = generic<float>(place.hoist), *table = generic<float>(cst);
        float4* const slots = generic<float4>(place.slots);
        const uint32_t cs = w & 0xffu, idx = w >> 16;
        if (cs == SB_CASE_FMA) {
            const SbInsn ins = place.code[(ip - place.exec) / sizeof(SbInsn) - 1u];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = t[i];
            m.store_slot(slots, place.scratch_slot);
            fma_over_scratch<RR, RC>(make_uint2(ins.w0, ins.w1), rowp, hrowp, place.tile_ld, table, slots, place.scratch_slot);
            m.fetch_slot(slots, place.scratch_slot, m.acc);
        } else { /* minimum or maximum */
            const uint32_t rel = cs - SB_CASE_BIN, kind = rel % SB_NUM_KINDS;
            const bool low = rel / SB_NUM_KINDS == SB_BIN_MIN;
            if (kind == SB_KIND_ROW) {
                f2 r[HR];
                m.fetch_row(rowp, hrowp, place.tile_ld, idx, r);
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = r[i / RC];
            } else if (kind == SB_KIND_CST) {
                f2 k[RC];
                m.fetch_cst(table, idx, k);
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = k[i % RC];
            } else {
                m.fetch_slot(slots, idx, m.acc);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                a[i] = low ? sbm::pack2(fminf(sbm::lo2(t[i]), sbm::lo2(a[i])), fminf(sbm::hi2(t[i]), sbm::hi2(a[i])))
                           : sbm::pack2(fmaxf(sbm::lo2(t[i]), sbm::lo2(a[i])), fmaxf(sbm::hi2(t[i]), sbm::hi2(a[i])));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = a[i];
    }

    static __device__ __forceinline__ void put(float* e, const f2 (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<ulonglong2*>(e)[i] = make_ulonglong2(v[2 * i], v[2 * i + 1]);
    }
    static __device__ __forceinline__ void take(const float* e, f2 (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const ulonglong2 w = reinterpret_cast<const ulonglong2*>(e)[i];
            v[2 * i] = w.x;
            v[2 * i + 1] = w.y;
        }
    }

    /* Runs one instruction run of the warp's rewritten program: the instructions from `start` on, over
     * the rows at place.row and the constants at `cst`. */
    __device__ __forceinline__ void run(const Place& place, uint32_t start, uint32_t cst) {
        f2 (&a)[V / 2] = reinterpret_cast<f2(&)[V / 2]>(acc);
        uint32_t ip = start;
        const f2 minus_one = sbm::both2(-1.0f), minus_zero = 0x8000000080000000ull;
        f2 x[8];
        uint32_t h, w;
        __align__(16) float unusual[32]; /* the tile and its arguments, when they have to go through memory */
#define SB_RUN_CORE(N, FUNCTIONS)                                                                                                               \
        asm volatile(SB_CORE(N, FUNCTIONS)                                                                                            \
                     : "+l"(a[0]), "+l"(a[1]), "+l"(a[2]), "+l"(a[3]), "+l"(a[4]), "+l"(a[5]), "+l"(a[6]), "+l"(a[7]), "=&l"(x[0]),    \
                       "=&l"(x[1]), "=&l"(x[2]), "=&l"(x[3]), "=&l"(x[4]), "=&l"(x[5]), "=&l"(x[6]), "=&l"(x[7]), "+r"(ip), "=&r"(h),  \
                       "=&r"(w)                                                                                                       \
                     : "r"(place.row), "r"(place.hoist - kHoistedOffset), "r"(cst), "r"(place.slots), "l"(minus_one), "l"(minus_zero),                                  \
                       "l"(__cvta_generic_to_global(&sbm::kTurns))                                                                         \
                     : "memory")
#pragma unroll 1
        for (;;) {
            if constexpr (RR == 4 && FAST) SB_RUN_CORE(4, SB_FAST_FUNCTIONS SB_NARROW_FAST);
            else if constexpr (RR == 4) SB_RUN_CORE(4, SB_FUNCTIONS(SB_AROUND_4) SB_NARROW_ACCURATE);
            else if constexpr (RR == 8 && FAST) SB_RUN_CORE(8, SB_FAST_FUNCTIONS);
            else if constexpr (RR == 8) SB_RUN_CORE(8, SB_FUNCTIONS(SB_AROUND));
            else if constexpr (FAST) SB_RUN_CORE(16, SB_FAST_FUNCTIONS);
            else SB_RUN_CORE(16, SB_FUNCTIONS(SB_AROUND));
            if (h == 0u) return;
            asm volatile("ld.shared.u32 %0, [%1+-16];" : "=r"(h) : "r"(ip) : "memory"); /* of the instruction the core stopped at */
            if (RR == 4 && h >= H_NARROW) h -= H_NARROW - H_DIV; /* in all columns: what the others hold is not read */
            if (FAST && h < H_SIN) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    a[i] = sbm::pack2(sbm::fast_div(sbm::lo2(a[i]), sbm::lo2(x[i])), sbm::fast_div(sbm::hi2(a[i]), sbm::hi2(x[i])));
                continue;
            }
            if (FAST && h != H_RARE) {
                fast_unary(w, a);
                continue;
            }
            put(unusual, a);
            if (h < H_SIN) put(unusual + 16, x);
            slow(unusual, place, h, w, ip, cst);
            take(unusual, a);
        }
#undef SB_RUN_CORE
    }
};

/* Sums RC per-lane values over the warp, one total per value, in a fixed order: halves of the warp
 * trade values so that every step adds pairs, and value c ends in lane c * (32 / RC). */
template <int RC>
__device__ __forceinline__ float column_totals(const float (&p)[RC], int lane) {
    float k;
    if (RC == 4) {
        const bool hi = lane & 16, hi8 = lane & 8;
        float k0 = hi ? p[2 % RC] : p[0], k1 = hi ? p[3 % RC] : p[1 % RC];
        const float s0 = hi ? p[0] : p[2 % RC], s1 = hi ? p[1 % RC] : p[3 % RC];
        k0 = __fadd_rn(k0, __shfl_xor_sync(0xffffffffu, s0, 16));
        k1 = __fadd_rn(k1, __shfl_xor_sync(0xffffffffu, s1, 16));
        k = hi8 ? k1 : k0;
        k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, hi8 ? k0 : k1, 8));
    } else if (RC == 2) {
        const bool hi = lane & 16;
        k = hi ? p[1 % RC] : p[0];
        k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, hi ? p[0] : p[1 % RC], 16));
        k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, k, 8));
    } else {
        k = __fadd_rn(p[0], __shfl_xor_sync(0xffffffffu, p[0], 16));
        k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, k, 8));
    }
    k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, k, 4));
    k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, k, 2));
    k = __fadd_rn(k, __shfl_xor_sync(0xffffffffu, k, 1));
    return k;
}

/* ---- tile staging ----------------------------------------------------------------------- */

__device__ __forceinline__ void cp_async_16(float* dst, const float* src, uint32_t src_bytes) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

/* Starts the asynchronous copy of rows [c0, c0 + rows) of every column into a tile buffer laid out
 * [column][tile_ld]; rows up to `padded` are zero-filled.  A column whose first row is 16-byte
 * aligned moves as 16-byte copies, any other as 4-byte copies (callers only promise 4-byte
 * alignment of their matrices).  Completion: cp_async_wait_all() by every thread, then a barrier. */
__device__ __noinline__ void stage_tile(float* tile, uint32_t tile_ld, const EvalProblem& prob, uint32_t ncols, size_t c0,
                                           uint32_t rows, uint32_t padded) {
#pragma unroll 1
    for (uint32_t col = 0; col < ncols; ++col) {
        const float* src = (col < prob.num_inputs ? prob.input + (size_t)col * prob.input_ld
                                                  : prob.targets + (size_t)(col - prob.num_inputs) * prob.targets_ld) + c0;
        float* dst = tile + (size_t)col * tile_ld;
        if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll 1
            for (uint32_t i = threadIdx.x * 4; i < padded; i += blockDim.x * 4) {
                if (i < rows) cp_async_16(dst + i, src + i, min(16u, (rows - i) * 4u)); /* short copies zero-fill their tail */
                else *reinterpret_cast<float4*>(dst + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        } else {
#pragma unroll 1
            for (uint32_t i = threadIdx.x; i < padded; i += blockDim.x) {
                if (i < rows) cp_async_4(dst + i, src + i);
                else dst[i] = 0.0f;
            }
        }
    }
    cp_async_commit();
}

__device__ __forceinline__ void add_shared(uint32_t address, float v, bool mine) {
    if (!mine) return;
    float s;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(s) : "r"(address) : "memory");
    s = __fadd_rn(s, v);
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(address), "f"(s) : "memory");
}

/* What a launch evaluates.  One kernel each, because the instruction cache decides the speed: with the
 * three epilogues, the rarer functions and the bank part in one kernel the population took 77 ms, with
 * the cold parts taken out 58 (see sbmath.cuh for the size of the cache). */
enum { KIND_SSE = 0, KIND_GENERAL = 1, KIND_MATERIALIZE = 2 }; /* one target; several targets or affine statistics; predictions */

template <int RC> struct TableWord { typedef float type; };
template <> struct TableWord<2> { typedef float2 type; };
template <> struct TableWord<4> { typedef float4 type; };

/* 16 values per thread: 20 warps per CTA within 96 registers (32-value tiles were measured
 * slower at the 12 warps their 168 registers allow). */
template <int RR, int RC, bool FAST, bool SPAN, bool PARTS, int KIND>
__global__ void __launch_bounds__(640, 1)
eval_kernel(const DeviceBatch batch, const EvalProblem prob, const Geom geom, float* __restrict__ partial,
            const float* __restrict__ tables) {
    using M = Machine<RR, RC, FAST>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* const tiles = reinterpret_cast<float*>(smem);
    unsigned int* const queue = reinterpret_cast<unsigned int*>(smem + (size_t)geom.tile_bytes * geom.tile_buffers);
    unsigned char* const warea = smem + (size_t)geom.tile_bytes * geom.tile_buffers + 16 + (size_t)warp * geom.warp_bytes;
    SbInsn* const exec = reinterpret_cast<SbInsn*>(warea) + 1; /* the entry before the first holds the first handler */
    float* const table = reinterpret_cast<float*>(warea + geom.exec_bytes);
    float* const psum = reinterpret_cast<float*>(warea + geom.exec_bytes + geom.table_bytes + geom.hoist_bytes + geom.slot_bytes);

    typename M::Place place;
    place.exec = (uint32_t)__cvta_generic_to_shared(exec);
    place.table = place.exec - 8u + geom.exec_bytes;
    place.hoist = place.table + geom.table_bytes + lane * 16u;
    place.slots = place.table + geom.table_bytes + geom.hoist_bytes + lane * 16u;
    place.tile_ld = geom.tile_rows;
    place.scratch_slot = geom.scratch_slot;
    const uint32_t psum32 = place.table + geom.table_bytes + geom.hoist_bytes + geom.slot_bytes + (lane / (32 / RC)) * 4u;
    const bool lane_sums = (lane & (32 / RC - 1)) == 0; /* the lanes in which column_totals() leaves a total */
    const uint32_t group = blockIdx.x / geom.row_splits, split = blockIdx.x % geom.row_splits;
    /* this CTA's programs: group, group + num_groups, ... (the batch is sorted by cost) */
    const uint32_t prog_count = (batch.num_programs - group + geom.num_groups - 1) / geom.num_groups;
    const size_t row_begin = (size_t)split * geom.rows_per_split;
    const size_t row_end = min(prob.num_rows, row_begin + (size_t)geom.rows_per_split);
    constexpr bool materialize = KIND == KIND_MATERIALIZE;
    const uint32_t ncols = prob.num_inputs + (materialize ? 0u : prob.num_targets);
    const uint32_t tile_ld = geom.tile_rows;
    const uint32_t T = prob.num_targets;
    const uint32_t nq = KIND == KIND_SSE ? 1u : prob.mode == EVAL_AFFINE_STATS ? T + 2 : T;
    const uint32_t gpi = geom.groups_per_item;
    const uint32_t ppi = SPAN ? geom.perms_per_item : 1u; /* SPAN: the run has toggles, and items may cover several permutations */
    const uint32_t wide = ppi * gpi; /* (permutation, bank group) pairs of an item: the partial sums' middle dimension */
    /* configuration groups of one program: permutation-major, RC banks per group */
    const uint32_t bank_groups = materialize ? 1u : (prob.num_banks + RC - 1) / RC;
    /* items of one program: permutation-major, `chunks` items of gpi bank groups per permutation, or
     * (when one item holds every bank group) one item per block of ppi permutations; the planner keeps
     * items_per_program * prog_count below 2^32 - 256, so item arithmetic is 32-bit */
    const uint32_t chunks = materialize ? 1u : bank_groups / gpi;
    const uint32_t items_per_program = PARTS ? chunks * geom.parts : !SPAN ? chunks : (uint32_t)(((unsigned long long)chunks << batch.max_bits) / ppi);
    const unsigned int num_items = items_per_program * prog_count;
    const unsigned long long configs = (unsigned long long)prob.num_banks << prob.toggle_bits;
    const size_t quantity_stride = geom.direct ? prob.out_target_stride : (size_t)configs;
    const size_t padded_configs = materialize ? (size_t)RC : ((size_t)bank_groups * RC) << batch.max_bits; /* per table entry */
    const size_t tile_floats = geom.tile_bytes / 4;
    const OperandStrides strides{{tile_ld * 4u, RC * 4u, M::V * 128u, M::PASS * 4u}};
    const uint32_t num_tiles = (uint32_t)((row_end - row_begin + geom.tile_rows - 1) / geom.tile_rows);

    /* Tiles: with two buffers tile t + 1 is fetched while tile t is used; with one (a tile so large
     * that only one fits beside the warps' working sets) the fetch follows a barrier after the tile. */
    const bool overlapped = geom.tile_buffers > 1;
    if (threadIdx.x == 0) queue[0] = 0u;
#pragma unroll 1
    for (uint32_t t = 0; t < num_tiles; ++t) {
        const size_t c0 = row_begin + (size_t)t * geom.tile_rows;
        const uint32_t chunk_rows = (uint32_t)min((size_t)geom.tile_rows, row_end - c0);
        const uint32_t npass = (chunk_rows + M::PASS - 1) / M::PASS;
        const uint32_t tile32 = (uint32_t)__cvta_generic_to_shared(tiles + (overlapped ? (size_t)(t & 1u) * tile_floats : 0));
        unsigned int* const q = queue + (t & 1u);
        if (t == 0 || !overlapped) {
            if (t) __syncthreads(); /* every warp has left the buffer */
            stage_tile(tiles, tile_ld, prob, ncols, c0, chunk_rows, npass * M::PASS);
        }
        cp_async_wait_all();
        __syncthreads(); /* tile t has landed; every warp has left tile t - 1 */
        if (threadIdx.x == 0) queue[(t + 1) & 1u] = 0u;
        if (overlapped && t + 1 < num_tiles) {
            const size_t n0 = c0 + geom.tile_rows;
            const uint32_t nrows = (uint32_t)min((size_t)geom.tile_rows, row_end - n0);
            stage_tile(tiles + (size_t)((t + 1) & 1u) * tile_floats, tile_ld, prob, ncols, n0, nrows, (nrows + M::PASS - 1) / M::PASS * M::PASS);
        }

#pragma unroll 1
        for (;;) {
            unsigned int item = 0;
            if (lane == 0) item = atomicAdd(q, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= num_items) break;
            /* with toggles (SPAN) the programs' first items come first: a program that reads fewer bits than the
             * batch's most has no more than those, and the rest of its numbers are passed over */
            uint32_t pi = item / items_per_program, within = item - pi * items_per_program;
            if (SPAN) {
                within = item / prog_count;
                pi = item - within * prog_count;
            }
            uint32_t pass = 0, end_pass = npass; /* the item's part of the tile */
            uint32_t lp = group + pi * geom.num_groups; /* index inside the batch */
            if constexpr (PARTS) {
                const uint32_t chunk = within / geom.parts;
                pass = (within - chunk * geom.parts) * geom.passes_per_part;
                end_pass = min(npass, pass + geom.passes_per_part);
                within = chunk;
                lp += batch.first;
                if (lp >= batch.num_programs) lp -= batch.num_programs;
            }
            const SbProgram* const hp = batch.programs + lp;
            const uint32_t pre_off = hp->pre_off, n_insn = hp->n_insn - pre_off, mid_off = hp->mid_off - pre_off, main_off = hp->main_off - pre_off;
            const uint32_t n_cst = hp->n_cst, n_patch = hp->n_patch, flags = hp->flags;
            /* the item's permutations perm0 .. perm0 + perms - 1, numbered by the bits the program reads */
            const uint32_t block = SPAN ? within / chunks : 0u;
            const uint32_t perm0 = SPAN ? block * ppi : 0u;
            if (SPAN && perm0 >= 1ull << hp->bits) continue;
            const uint32_t perms = !SPAN ? 1u : (uint32_t)min((unsigned long long)ppi, (1ull << hp->bits) - perm0);
            const auto narrow = [&](uint32_t i) { return RR == 4 && !SPAN && (i < main_off || (flags & SB_PROG_BANK_INDEPENDENT)); };
            __syncwarp(); /* the previous item's reads of exec, table and psum are done */
            const SbInsn* const code = batch.insns + hp->insn_off + pre_off; /* the row parts; the bank part has run (bank_tables_kernel) */
#pragma unroll 1
            for (uint32_t i = lane; i < n_insn; i += 32) put_insn(exec + i, rewrite(code[i], strides, narrow(i), FAST));
            const uint32_t first_bg = materialize ? 0u : (within - block * chunks) * gpi;
            const uint32_t ngroups = materialize ? 1u : min(gpi, bank_groups - first_bg);
            const SbPatch* const patches = batch.patches + hp->patch_off;
            /* rewrites the toggle sites of the warp's copy for one permutation */
            auto patch_for = [&](uint32_t perm) {
                __syncwarp(); /* earlier reads and writes of the copy by other lanes are done */
#pragma unroll 1
                for (uint32_t i = lane; i < n_patch; i += 32) {
                    const SbPatch* p = patches + i;
                    unsigned choice = (perm >> p->bit0) & 1u;
                    if (p->bit1 != 0xffu) choice |= ((perm >> p->bit1) & 1u) << 1;
                    if (p->insn >= pre_off) put_insn(exec + (p->insn - pre_off), rewrite(p->alt[choice], strides, narrow(p->insn - pre_off), FAST));
                }
                __syncwarp();
            };
            if (!materialize && !PARTS) {
#pragma unroll 1
                for (uint32_t e = lane; e < nq * wide * RC; e += 32) psum[e] = 0.0f;
            }
            const size_t gp = prob.first_program + hp->index; /* position in the run: output row, bank table */
            const uint32_t table_stride = n_cst * RC;
            { /* the item's constant tables: contiguous, since an item of several permutations holds every bank group of each */
                const float* src = tables + (size_t)(hp->cst_off - batch.programs[0].cst_off) * padded_configs +
                                   ((size_t)perm0 * bank_groups + first_bg) * table_stride;
                const uint32_t n = perms * ngroups * table_stride / RC;
                typedef typename TableWord<RC>::type Word;
#pragma unroll 1
                for (uint32_t i = lane; i < n; i += 32) reinterpret_cast<Word*>(table)[i] = __ldg(reinterpret_cast<const Word*>(src) + i);
            }
            if (SPAN && ppi == 1u && n_patch) patch_for(perm0);
            __syncwarp();
            const bool has_shared = mid_off > 0u, has_prelude = main_off > mid_off;
            const uint32_t eval_groups = (flags & SB_PROG_BANK_INDEPENDENT) ? 1u : ngroups;

            /* PARTS: where this lane's totals of a pass go, [pass][program][quantity][bank]; of the last group's
             * columns only those below `banks` are banks */
            const uint32_t my_bank = first_bg * RC + lane / (32 / RC), banks = lane_sums ? prob.num_banks : 0u;
            float* totals = partial;
            if constexpr (PARTS && !materialize) totals += ((c0 / M::PASS + pass) * batch.num_programs + lp) * nq * configs + my_bank;

            M m;
            place.code = code;
#pragma unroll 1
            for (; pass < end_pass; ++pass) {
                place.row = tile32 + (pass * M::PASS + lane * 4) * 4u;
                const uint32_t row0 = pass * M::PASS + lane * 4; /* first row of this thread in the tile */
                const bool full = (pass + 1) * M::PASS <= chunk_rows;
                /* One loop over the steps of a pass, so that the interpreter has one call site (a second
                 * inlined copy would not fit the instruction caches).  First (only when the program has
                 * one) the shared row prelude: the row-only sub-expressions no toggle reaches, once for the
                 * pass.  Then, for every permutation of the item: the row-only sub-expressions that depend
                 * on it (only when the program has any), and the main part once per bank group.  Without
                 * SPAN an item has one permutation and the steps are -2 (shared prelude), -1 (prelude),
                 * 0.. (bank groups); with it they are -1 (shared prelude) and then per_perm steps per
                 * permutation. */
                const int per_perm = (has_prelude ? 1 : 0) + (int)eval_groups;
                const int first = SPAN ? (has_shared ? -1 : 0) : (has_shared ? -2 : has_prelude ? -1 : 0);
                const int last = SPAN ? (int)perms * per_perm : (int)eval_groups;
#pragma unroll 1
                for (int s = first, permutation = 0, step = 0; s < last; ++s) {
                    /* SPAN: step `step` of permutation `permutation`, counted on: a division per step cost 384 gated programs
                     * 3.15 ms instead of 2.99 */
                    if (SPAN && s > 0 && ++step == per_perm) { step = 0; ++permutation; }
                    int j = 0, g = s < 0 ? 0 : s;
                    bool prelude = s < 0;
                    uint32_t start = s == first && has_shared ? 0u : s < 0 ? mid_off : main_off;
                    if (SPAN) {
                        j = permutation;
                        const int w = step;
                        prelude = s < 0 || (has_prelude && w == 0);
                        g = prelude ? 0 : w - (has_prelude ? 1 : 0);
                        start = prelude ? (s < 0 ? 0u : mid_off) : main_off;
                        if (s >= 0 && w == 0 && ppi > 1u && n_patch) patch_for(perm0 + (uint32_t)j);
                    } else if (s == -1 && !has_prelude) continue;
                    const uint32_t gi = (uint32_t)j * ngroups + (uint32_t)g; /* this permutation's table, this group's */
                    m.run(place, place.exec + start * (uint32_t)sizeof(SbInsn), place.table + gi * table_stride * 4u);
                    if (prelude) continue;
                    if (!full && !materialize) { /* rows past the data score nothing: their staged targets are zero, and so is their prediction now */
#pragma unroll
                        for (int h = 0; h < M::HR; ++h) {
                            const uint32_t row = row0 + (h / 2) * 128 + (h % 2) * 2;
                            const f2 keep = (row < chunk_rows ? 0xffffffffull : 0ull) | (row + 1 < chunk_rows ? 0xffffffff00000000ull : 0ull);
#pragma unroll
                            for (int c = 0; c < RC; ++c) m.acc[h][c] &= keep;
                        }
                    }
                    if constexpr (materialize) {
                        float* out = prob.output + gp * prob.out_program_stride + c0;
#pragma unroll
                        for (int r = 0; r < RR; ++r) {
                            const uint32_t row = row0 + (r / 4) * 128 + (r % 4);
                            if (row < chunk_rows) out[row] = r & 1 ? sbm::hi2(m.acc[r / 2][0]) : sbm::lo2(m.acc[r / 2][0]);
                        }
                    } else if constexpr (KIND == KIND_SSE) {
                        f2 tv[M::HR];
                        float part[RC]; /* row after row */
                        m.fetch_column(place.row + prob.num_inputs * tile_ld * 4u, tv);
#pragma unroll
                        for (int c = 0; c < RC; ++c) {
                            part[c] = 0.0f;
#pragma unroll
                            for (int h = 0; h < M::HR; ++h) {
                                const f2 e = sbm::sub2(m.acc[h][c], tv[h]);
                                part[c] = __fmaf_rn(sbm::lo2(e), sbm::lo2(e), part[c]);
                                part[c] = __fmaf_rn(sbm::hi2(e), sbm::hi2(e), part[c]);
                            }
                        }
                        const float total = column_totals<RC>(part, lane);
                        if constexpr (!PARTS) add_shared(psum32 + gi * (RC * 4u), total, lane_sums);
                        else if (my_bank + g * RC < banks) totals[g * RC] = total;
                    } else {
                        /* several targets, or affine statistics: quantity q of pair gi lives in psum[(q * wide + gi) * RC + c] */
#pragma unroll 1
                        for (uint32_t qn = 0; qn < nq; ++qn) {
                            f2 tv[M::HR];
                            const bool is_target = prob.mode == EVAL_SSE || qn >= 2;
                            const uint32_t tcol = prob.num_inputs + (prob.mode == EVAL_SSE ? qn : qn - 2);
                            if (is_target) m.fetch_column(place.row + tcol * tile_ld * 4u, tv);
                            float s[RC];
#pragma unroll
                            for (int c = 0; c < RC; ++c) {
                                s[c] = 0.0f;
#pragma unroll
                                for (int h = 0; h < M::HR; ++h) {
                                    const f2 p = m.acc[h][c];
                                    f2 term;
                                    if (prob.mode == EVAL_SSE) { const f2 e = sbm::sub2(p, tv[h]); term = sbm::mul2(e, e); }
                                    else if (qn == 0) term = p;
                                    else if (qn == 1) term = sbm::mul2(p, p);
                                    else term = sbm::mul2(p, tv[h]);
                                    s[c] = __fadd_rn(__fadd_rn(s[c], sbm::lo2(term)), sbm::hi2(term));
                                }
                            }
                            const float total = column_totals<RC>(s, lane);
                            if constexpr (!PARTS) add_shared(psum32 + (qn * wide + gi) * (RC * 4u), total, lane_sums);
                            else if (my_bank + g * RC < banks) totals[qn * configs + g * RC] = total;
                        }
                    }
                }
                if constexpr (PARTS && !materialize) totals += (size_t)batch.num_programs * nq * configs;
            }
            if (materialize || PARTS) continue;
            __syncwarp();
            /* this CTA's partial sums of the item: stored on its first tile, added to afterwards (only this
             * CTA touches them, and a barrier separates its tiles) */
            {
                const bool independent = (flags & SB_PROG_BANK_INDEPENDENT) != 0;
                const uint32_t width = ngroups * RC, bank0 = first_bg * RC; /* banks of the item, padding included */
                const uint32_t real = min(width, prob.num_banks - bank0);
                float* mine = partial + (geom.direct ? gp * prob.out_program_stride : ((size_t)split * batch.num_programs + lp) * nq * configs) +
                              ((size_t)bank0 << prob.toggle_bits);
                float* sums = psum; /* psum is [quantity][permutation][group][bank of the group] */
                if constexpr (!SPAN) {
#pragma unroll 1
                    for (uint32_t qn = 0; qn < nq; ++qn, mine += quantity_stride, sums += wide * RC)
#pragma unroll 1
                        for (uint32_t e = lane; e < real; e += 32) {
                            const float v = sums[independent ? 0u : e];
                            mine[e] = t == 0 ? v : __fadd_rn(mine[e], v);
                        }
                } else {
                    const uint32_t apart = independent ? 1u : real; /* banks with a sum of their own */
                    /* A program has one value for all permutations that differ only in bits it does not read, so only
                     * those it tells apart were evaluated (384 gated programs, 256 permutations x 4 sets, 32,768 rows:
                     * 33.2 -> 4.3 ms; 1,000 programs, 256 permutations, 2,001 rows: 2.9 -> 1.0 ms). */
                    /* between tiles a sum waits where the bits the program does not read are 0; after the last
                     * one every permutation that differs only in those bits receives it */
                    const uint32_t used = batch.programs[lp].bit_mask, unused = (uint32_t)((1ull << prob.toggle_bits) - 1ull) & ~used;
                    const uint32_t free_bits = prob.toggle_bits - (uint32_t)__popc(used);
#pragma unroll 1
                    for (uint32_t qn = 0; qn < nq; ++qn, mine += quantity_stride, sums += wide * RC)
#pragma unroll 1
                        for (uint32_t j = 0; j < perms; ++j) {
                            float* const dst = mine + deposit(perm0 + j, used);
                            float* const s = sums + j * width;
                            if (t) {
#pragma unroll 1
                                for (uint32_t e = lane; e < apart; e += 32) s[e] = __fadd_rn(dst[(size_t)e << prob.toggle_bits], s[e]);
                                __syncwarp();
                            }
                            if (t + 1 < num_tiles) {
#pragma unroll 1
                                for (uint32_t e = lane; e < apart; e += 32) dst[(size_t)e << prob.toggle_bits] = s[e];
                            } else {
#pragma unroll 1
                                for (unsigned long long x = lane; x < (unsigned long long)real << free_bits; x += 32) {
                                    const uint32_t e = (uint32_t)(x >> free_bits);
                                    dst[((size_t)e << prob.toggle_bits) + deposit((uint32_t)x & (uint32_t)((1ull << free_bits) - 1ull), unused)] =
                                        s[independent ? 0u : e];
                                }
                            }
                        }
                }
            }
        }
    }
    cp_async_wait_all();
}


/* the launches of one kind of kernel, over the tile shapes; PARTS: the launch keeps the totals of passes (in place of sums in
 * shared memory), cuts tiles into parts or does not begin with its first program (small launches without toggles; what it
 * takes made large ones 1 % slower) */
template <int KIND, int RR, int RC, bool SPAN, bool PARTS>
void launch_parts(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                  const float* tables, cudaStream_t stream) {
    if (prob.fast_math) eval_kernel<RR, RC, true, SPAN, PARTS, KIND><<<plan.grid_x, plan.warps * 32, plan.smem_bytes, stream>>>(batch, prob, geom, partial, tables);
    else eval_kernel<RR, RC, false, SPAN, PARTS, KIND><<<plan.grid_x, plan.warps * 32, plan.smem_bytes, stream>>>(batch, prob, geom, partial, tables);
}
template <int KIND, int RR, int RC, bool SPAN>
cudaError_t launch_shape(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                         const float* tables, cudaStream_t stream) {
    if (!SPAN && (plan.pass_sums || geom.parts > 1u || batch.first)) launch_parts<KIND, RR, RC, SPAN, !SPAN>(batch, prob, geom, plan, partial, tables, stream);
    else launch_parts<KIND, RR, RC, SPAN, false>(batch, prob, geom, plan, partial, tables, stream);
    return cudaGetLastError();
}
template <int KIND, bool SPAN>
cudaError_t launch_kind(const DeviceBatch& batch, const EvalProblem& prob, const Geom& geom, const LaunchPlan& plan, float* partial,
                        const float* tables, cudaStream_t stream) {
    switch (plan.variant) {
    case 0: return launch_shape<KIND, 4, 4, SPAN>(batch, prob, geom, plan, partial, tables, stream);
    case 1: return launch_shape<KIND, 8, 2, SPAN>(batch, prob, geom, plan, partial, tables, stream);
    default: return launch_shape<KIND, 16, 1, SPAN>(batch, prob, geom, plan, partial, tables, stream);
    }
}
template <int KIND, bool SPAN, bool PARTS>
cudaError_t configure_parts(int smem_limit) {
    const void* kernels[] = {(const void*)eval_kernel<4, 4, false, SPAN, PARTS, KIND>,  (const void*)eval_kernel<4, 4, true, SPAN, PARTS, KIND>,
                             (const void*)eval_kernel<8, 2, false, SPAN, PARTS, KIND>,  (const void*)eval_kernel<8, 2, true, SPAN, PARTS, KIND>,
                             (const void*)eval_kernel<16, 1, false, SPAN, PARTS, KIND>, (const void*)eval_kernel<16, 1, true, SPAN, PARTS, KIND>};
    for (const void* f : kernels) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_limit);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
template <int KIND, bool SPAN>
cudaError_t configure_kind(int smem_limit) {
    const cudaError_t e = configure_parts<KIND, SPAN, false>(smem_limit);
    return e == cudaSuccess && !SPAN ? configure_parts<KIND, SPAN, !SPAN>(smem_limit) : e;
}

}  // namespace

}  // namespace sb

#endif
