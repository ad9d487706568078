/*
 * rollout.cu - RK4 rollout scoring: candidate right-hand sides interpreted inside the integrator.
 *
 * Restates the integration loop of the reference engine's generated scoring kernel
 * (projects/odezza/core/o_generate_scoring_cuda.c:494-588): per observation interval
 * h = interval / substeps; per substep base = stage = state, sum = 0, four stages with
 * sum = fma(w, rhs, sum) (w = 1,2,2,1), stage = fma(h/2 or h, rhs, base), then
 * state = fma(h/6, sum, base); after every interval all states must be finite and
 * sq = fma(err, err, sq).  Score = sq / residuals, or FLT_MAX when anything was not finite.
 *
 * Mapping (different from the reference, which gives a thread one configuration and loops all
 * trajectories inside it): one warp per (system, configuration, state), lanes = trajectories, RR per
 * lane.  RR is chosen from the trajectory count so that a pass of 32 * RR trajectories keeps all
 * lanes busy: 1 up to 32 trajectories, 2 up to 64, 4 beyond.  A right-hand side is a flat record
 * (record.h) whose operands are constants of the program, stage values (what COLUMN s reads) and
 * temporaries of the warp.
 */
#include "evaluator.cuh"
#include "pairs_ptx.cuh"
#include "sbmath.cuh"

#include <algorithm>

namespace sb {

namespace {

using sbm::f2;

constexpr int kRolloutMaxWarps = 16;
constexpr float kFltMax = 3.402823466e+38f;

/* Two elements behind one call, any argument: what the core leaves to others.  The whole warp is here. */
__device__ __noinline__ f2 unary_pair(f2 v, unsigned op) {
    switch (op) {
    case SB_UN_SIN: case SB_UN_COS: return sbm::sincos_pair(v, op == SB_UN_COS ? 1 : 0);
    case SB_UN_EXP: return sbm::exp_pair(v);
    case SB_UN_LOG: return sbm::log_pair(v);
    default: return sbm::pack2(sbm::any1(sbm::lo2(v), op), sbm::any1(sbm::hi2(v), op));
    }
}
__device__ __noinline__ f2 div_pair(f2 a, f2 b) { return sbm::pack2(sbm::div1(sbm::lo2(a), sbm::lo2(b)), sbm::div1(sbm::hi2(a), sbm::hi2(b))); }

/* ---- shared memory by 32-bit shared-window address ------------------------------------------
 * The interpreter's operands, the integrator's vectors and the instruction stream itself are read
 * through these, so address arithmetic stays 32 bits wide and an operand's address can be stored
 * ready-made in the instruction word. */
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int RR>
__device__ __forceinline__ void lds(uint32_t a, float (&x)[RR]) {
    if constexpr (RR == 4) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(a));
    else if constexpr (RR == 2) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x[0]), "=f"(x[1]) : "r"(a));
    else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x[0]) : "r"(a));
}
__device__ __forceinline__ uint32_t lds_word(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
template <int RR>
__device__ __forceinline__ void sts(uint32_t a, const float (&x)[RR]) {
    if constexpr (RR == 4) asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]) : "memory");
    else if constexpr (RR == 2) asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x[0]), "f"(x[1]) : "memory");
    else asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x[0]) : "memory");
}

/* Handlers of the rollout machine.  A warp rewrites the main part of its private copy of a record
 * once per item into this form: word 0 = the handler of the NEXT instruction (so that the indexed branch's
 * table is read while this one works), word 1 = where the operand is (C: the shared address of a
 * constant-table entry, one for all lanes; V: the offset of a state in the vector of stage values; T: the
 * offset of one of the warp's temporaries) or, for the functions, SB_UN_*.  H_STLOAD (temporary = acc,
 * then acc = operand) keeps the temporary's offset, in units of 128 bytes, above the operand's 18 bits.
 * One item runs its right-hand sides 4 stages x steps times, so the rewrite is free.
 *
 * The machine is one block of PTX for the reasons given in eval_kernel.cuh, and here for one more: an
 * item is one chain of dependent instructions, so what an interpreted instruction costs decides how long
 * a call takes (two values per lane share it, where the population evaluator's sixteen do).  With the
 * C++ machine it cost 50 issued instructions, of which dispatch was half; here it costs 20, the
 * integrator's part included.  In a chain of them one takes 75 cycles for an addition with any operand,
 * 110 for an exponential, 200 for a sine or a division (one warp alone on its SM). */
enum { H_END = 0, H_LOAD = 1, H_STORE = 4, H_STLOAD = 5, H_ADD = 8, H_SUB = 11, H_RSUB = 14, H_MUL = 17, H_DIV = 20, H_RDIV = 23, /* + kind */
       H_MIN = 26, H_MAX = 29, H_NEG = 32, H_ABS = 33, H_SIN = 34, H_COS, H_EXP, H_LOG, H_TANH, H_UNARY, H_FMA };
enum { RK_CST = 0, RK_STATE = 1, RK_TEMP = 2 };
constexpr uint32_t kStoredShift = 18, kStoredUnit = 128;

/* the constants of the functions by pairs, read two at a time: moves would cost as much as the
 * arithmetic of a single pair */
__constant__ __align__(16) unsigned long long kPairConstants[] = {
    SB_SIN_LIST(SB_PAIR_WORD) 0ull, /* 0: eleven and one to fill the last pair of words, as RK_K2's offsets count them */
    SB_EXP_LIST(SB_PAIR_WORD) 0ull, /* 96 */
    SB_LOG_LIST(SB_PAIR_WORD)       /* 128 */
    SB_TANH_LIST(SB_PAIR_WORD)};    /* 224 */
static_assert(sizeof(kPairConstants) == 320, "the offsets RK_K2 is given count on this layout");

/* The block carries a whole observation interval: the instruction that ends a right-hand side goes on with
 * the integrator's part of the stage (EN, and E3 for the last: sum += weight * rhs, the next stage's value of this
 * warp's state from the step's base), meets the other warps of the item at their barrier and starts the
 * next stage, until the interval's steps are done.  A right-hand side begins by loading a constant or a state in
 * nearly all cases: the end of the stage does that itself (MEET), with one branch for both kinds, and only what
 * begins otherwise (REST: a fused multiply-add) starts from its first instruction.  That, and a stage chosen by
 * selects instead of an indexed branch, is two indexed branches less per stage: 1,846 systems of one state, 130
 * trajectories, 527 steps 16.6 -> 16.3 ms (three populations); 600 engine systems of two states, 184 stages 1.05 -> 1.00 ms a
 * call; of 4,096 of three states, 1,000 steps, whose stages wait for the longest right-hand side, it does not show (six
 * populations: 23.9 -> 23.8, which differ by 0.1 between runs).
 * (The functions on a copy while the warp votes on their arguments, so that the vote is no link of the chain, and
 * the copy taken over behind it: 23.2 -> 24.7 ms.  It is instructions that cost here as well.)
 *
 * asm operands: 0 the address of the next instruction, 1 the next handler and 2 word 1 of this
 * instruction (at the end 1 says whether the interval is done, 0, or an instruction was left, 1), 3 and 4
 * the accumulator (RR = 1: both halves of 3 hold the value), 5 and 6 the stage sum, 7 and 8 the state (base of the step), 9 and 10 the addresses of this stage's values and of the next
 * stage's for this lane, 11 the stage, 12 the steps left; 13 the address of the temporaries for this lane,
 * 14 the pair (-1, -1), 15 the constants, 16 to 21 h / 2, h and h / 6, 22 the first instruction, 23 the
 * offset of this warp's state, 24 and 25 the barrier and its threads (0: no barrier), 26 the first handler. */
#define RK_NEXT "mov.u32 hb, %1;\n ld.shared.v2.u32 {%1, %2}, [%0];\n add.u32 %0, %0, 8;\n"
#define RK_GO "brx.idx.uni hb, targets;\n"
#define RK_FETCH_1(A) "ld.shared.b32 c0, [" A "];\n mov.b64 x0, {c0, c0};\n"
#define RK_FETCH_2(A) "ld.shared.b64 x0, [" A "];\n"
#define RK_FETCH_4(A) "ld.shared.v2.b64 {x0, x1}, [" A "];\n"
#define RK_KEEP_1(A, P, Q) "mov.b64 {c0, c1}, " P ";\n st.shared.b32 [" A "], c0;\n"
#define RK_KEEP_2(A, P, Q) "st.shared.b64 [" A "], " P ";\n"
#define RK_KEEP_4(A, P, Q) "st.shared.v2.b64 [" A "], {" P ", " Q "};\n"
#define RK_BOTH_1(F) F("%3", "x0")
#define RK_BOTH_2(F) F("%3", "x0")
#define RK_BOTH_4(F) F("%3", "x0") F("%4", "x1")
#define RK_EACH_1(F) F("%3")
#define RK_EACH_2(F) F("%3")
#define RK_EACH_4(F) F("%3") F("%4")
#define RK_EACHX_1(F) F("x0")
#define RK_EACHX_2(F) F("x0")
#define RK_EACHX_4(F) F("x0") F("x1")
#define RK_MOV(A, X) "mov.b64 " A ", " X ";\n"
#define RK_ADD(A, X) "add.rn.f32x2 " A ", " A ", " X ";\n"
#define RK_SUB(A, X) "fma.rn.f32x2 " A ", " X ", mone, " A ";\n"
#define RK_RSUB(A, X) "fma.rn.f32x2 " A ", " A ", mone, " X ";\n"
#define RK_MUL(A, X) "mul.rn.f32x2 " A ", " A ", " X ";\n"
#define RK_MIN(A, X) "mov.b64 {f0, f1}, " A ";\n mov.b64 {top, low}, " X ";\n min.f32 f0, f0, top;\n min.f32 f1, f1, low;\n mov.b64 " A ", {f0, f1};\n"
#define RK_MAX(A, X) "mov.b64 {f0, f1}, " A ";\n mov.b64 {top, low}, " X ";\n max.f32 f0, f0, top;\n max.f32 f1, f1, low;\n mov.b64 " A ", {f0, f1};\n"
#define RK_NEG(A) "xor.b64 " A ", " A ", 0x8000000080000000;\n"
#define RK_ABS(A) "and.b64 " A ", " A ", 0x7fffffff7fffffff;\n"
#define RK_SWAP(A, X) "mov.b64 m, " A ";\n mov.b64 " A ", " X ";\n mov.b64 " X ", m;\n"
/* an operation with a constant (label NAME C), a state (NAME V) and a temporary (NAME T) */
#define RK_THREE(N, NAME, F)                                                                            \
    NAME "C:\n" RK_FETCH_##N("%2") RK_NEXT RK_BOTH_##N(F) RK_GO                                          \
    NAME "V:\n add.u32 ad, %2, %9;\n" RK_FETCH_##N("ad") RK_NEXT RK_BOTH_##N(F) RK_GO                    \
    NAME "T:\n add.u32 ad, %2, %13;\n" RK_FETCH_##N("ad") RK_NEXT RK_BOTH_##N(F) RK_GO
#define RK_STLOAD(N, NAME, BASE)                                                                        \
    NAME ":\n shr.u32 c2, %2, 18;\n shl.b32 c2, c2, 7;\n add.u32 c2, c2, %13;\n" RK_KEEP_##N("c2", "%3", "%4")       \
    "and.b32 ad, %2, 0x3ffff;\n" BASE RK_FETCH_##N("ad") RK_NEXT RK_BOTH_##N(RK_MOV) RK_GO
#define RK_FETCH_THEN(N, NAME, WHERE)                                                                   \
    NAME "C:\n" RK_FETCH_##N("%2") "bra.uni " WHERE ";\n"                                               \
    NAME "V:\n add.u32 ad, %2, %9;\n" RK_FETCH_##N("ad") "bra.uni " WHERE ";\n"                         \
    NAME "T:\n add.u32 ad, %2, %13;\n" RK_FETCH_##N("ad") "bra.uni " WHERE ";\n"
#define RK_K2(A, B, OFF) "ld.const.v2.u64 {" A ", " B "}, [%15+" OFF "];\n"
#define RK_CORE(N)                                                                                      \
    "{\n" SB_PTX_REGISTERS ".reg .b64 x0, x1;\n .reg .pred meet;\n .reg .u32 hb;\n"                                                        \
    "targets: .branchtargets EN, LC, LV, LT, ST, KC, KV, KT, AC, AV, AT, SC, SV, STT, RC, RV, RT, MC, MV, MT, DC, DV, DT, QC, QV, QT, " \
    "NC, NV, NT, XC, XV, XT, NG, AB, SI, CO, EX, LG, TH, LEAVE, LEAVE;\n mov.b64 mone, %14;\n setp.ne.u32 meet, %25, 0;\n"               \
    "ld.shared.u32 %1, [%0+-8];\n" RK_NEXT RK_GO                                                         \
    RK_THREE(N, "L", RK_MOV) RK_THREE(N, "A", RK_ADD) RK_THREE(N, "R", RK_RSUB)                         \
    "SC:\n" RK_FETCH_##N("%2") RK_NEXT RK_BOTH_##N(RK_SUB) RK_GO                                         \
    "SV:\n add.u32 ad, %2, %9;\n" RK_FETCH_##N("ad") RK_NEXT RK_BOTH_##N(RK_SUB) RK_GO                   \
    "STT:\n add.u32 ad, %2, %13;\n" RK_FETCH_##N("ad") RK_NEXT RK_BOTH_##N(RK_SUB) RK_GO                  \
    RK_THREE(N, "M", RK_MUL) RK_THREE(N, "N", RK_MIN) RK_THREE(N, "X", RK_MAX)                          \
    "ST:\n add.u32 ad, %2, %13;\n" RK_NEXT RK_KEEP_##N("ad", "%3", "%4") RK_GO                                       \
    RK_STLOAD(N, "KC", "") RK_STLOAD(N, "KV", "add.u32 ad, ad, %9;\n") RK_STLOAD(N, "KT", "add.u32 ad, ad, %13;\n") \
    "NG:\n" RK_NEXT RK_EACH_##N(RK_NEG) RK_GO "AB:\n" RK_NEXT RK_EACH_##N(RK_ABS) RK_GO                  \
    "CO:\n" SB_COS_SHIFT "bra.uni SC0;\n SI:\n" SB_SIN_SHIFT                                            \
    "SC0:\n" RK_K2("k0", "k1", "0") RK_K2("k2", "k3", "16") RK_K2("k4", "k5", "32") RK_K2("k6", "k7", "48") RK_K2("k8", "k9", "64") \
    RK_K2("k10", "m", "80") "mov.f32 top, 0f00000000;\n" RK_EACH_##N(SB_TOP) "setp.lt.f32 p, top, 0f45800000;\n" SB_ALL_OR_LEAVE RK_NEXT \
    RK_EACH_##N(SB_SIN_PAIR) RK_GO                                                                      \
    "EX:\n" RK_K2("k0", "k1", "96") RK_K2("k2", "m", "112") "mov.f32 top, 0f00000000;\n" RK_EACH_##N(SB_TOP) \
    "setp.le.f32 p, top, 0f42AC0000;\n" SB_ALL_OR_LEAVE RK_NEXT RK_EACH_##N(SB_EXP_PAIR) RK_GO          \
    "LG:\n" RK_K2("k0", "k1", "128") RK_K2("k2", "k3", "144") RK_K2("k4", "k5", "160") RK_K2("k6", "k7", "176") RK_K2("k8", "k9", "192") \
    RK_K2("k10", "k11", "208") "mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n" RK_EACH_##N(SB_TOP) RK_EACH_##N(SB_LOW) \
    "setp.lt.f32 p, top, 0f7F800000;\n setp.ge.and.f32 p, low, 0f00800000, p;\n" SB_ALL_OR_LEAVE RK_NEXT RK_EACH_##N(SB_LOG_PAIR) RK_GO \
    "TH:\n" RK_K2("k0", "k1", "224") RK_K2("k2", "k3", "240") RK_K2("k4", "k5", "256") RK_K2("k6", "k7", "272") RK_K2("k8", "k9", "288") \
    RK_K2("k10", "k11", "304") RK_NEXT RK_EACH_##N(SB_TANH_PAIR) RK_GO                                   \
    RK_FETCH_THEN(N, "D", "DIV") RK_FETCH_THEN(N, "Q", "RDIV")                                          \
    /* operand / acc; what leaves for an unusual argument takes the accumulator along as it was */      \
    "RDIV:\n mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n" RK_EACH_##N(SB_TOP) RK_EACHX_##N(SB_TOP) \
    RK_EACH_##N(SB_LOW_NUMBER) RK_EACHX_##N(SB_LOW_NUMBER) SB_DIV_USUAL "@p bra.uni RS;\n"                    \
    "mov.u32 c2, 0xffffffff;\n mov.f32 low, 0f7F800000;\n" RK_EACHX_##N(SB_LEAST) RK_EACH_##N(SB_LOW_NUMBER) SB_DIV_RANGE SB_ALL_OR_LEAVE \
    "RS:\n" RK_BOTH_##N(RK_SWAP) "bra.uni DW;\n"                                                       \
    "DIV:\n mov.f32 top, 0f00000000;\n mov.f32 low, 0f7F800000;\n" RK_EACH_##N(SB_TOP) RK_EACHX_##N(SB_TOP) \
    RK_EACH_##N(SB_LOW_NUMBER) RK_EACHX_##N(SB_LOW_NUMBER) SB_DIV_USUAL "@p bra.uni DW;\n"                    \
    "mov.u32 c2, 0xffffffff;\n mov.f32 low, 0f7F800000;\n" RK_EACH_##N(SB_LEAST) RK_EACHX_##N(SB_LOW_NUMBER) SB_DIV_RANGE SB_ALL_OR_LEAVE \
    "DW:\n" RK_NEXT SB_DIV_CONSTANTS RK_BOTH_##N(SB_DIV_PAIR) RK_GO                                      \
    "EN:\n setp.eq.u32 p, %11, 3;\n @p bra.uni E3;\n"                                                    \
    "setp.eq.u32 p, %11, 0;\n selp.b64 k0, 0x3f8000003f800000, 0x4000000040000000, p;\n"               \
    "setp.eq.u32 p, %11, 2;\n" RK_STAGE_##N                                                             \
    "add.u32 ad, %10, %23;\n" RK_KEEP_##N("ad", "x0", "x1")                                             \
    "mov.u32 c0, %9;\n mov.u32 %9, %10;\n mov.u32 %10, c0;\n add.u32 %11, %11, 1;\n bra.uni MEET;\n"    \
    "E3:\n" RK_LAST_##N "add.u32 ad, %10, %23;\n" RK_KEEP_##N("ad", "%7", "%8")                         \
    "mov.u32 c0, %9;\n mov.u32 %9, %10;\n mov.u32 %10, c0;\n mov.u32 %11, 0;\n"                        \
    "sub.u32 %12, %12, 1;\n setp.eq.u32 p, %12, 0;\n mov.u32 %0, %22;\n @p bra.uni DONE;\n"            \
    "MEET:\n mov.u32 %0, %22;\n mov.u32 %1, %26;\n" RK_NEXT                                              \
    "sub.u32 c0, hb, 1;\n setp.gt.u32 p, c0, 1;\n @p bra.uni REST;\n"                                   \
    "setp.eq.u32 p, hb, 2;\n selp.u32 c0, %9, 0, p;\n add.u32 ad, %2, c0;\n" RK_NEXT                    \
    "@meet barrier.cta.sync %24, %25;\n" RK_FETCH_##N("ad") RK_BOTH_##N(RK_MOV) RK_GO                   \
    "REST:\n @meet barrier.cta.sync %24, %25;\n" RK_GO                                                  \
    "DONE:\n mov.u32 %1, 0;\n bra.uni OUT;\n LEAVE:\n mov.u32 %1, 1;\n OUT:\n }"
/* the weights of the stages are 1, 2, 2, 1 (a multiplication by 1 is exact, and the sum starts at 0) */
#define RK_STAGE_1 "fma.rn.f32x2 %5, %3, k0, %5;\n selp.b64 k1, %18, %16, p;\n fma.rn.f32x2 x0, k1, %3, %7;\n"
#define RK_STAGE_2 RK_STAGE_1
#define RK_STAGE_4 RK_STAGE_1 "fma.rn.f32x2 %6, %4, k0, %6;\n selp.b64 k2, %19, %17, p;\n fma.rn.f32x2 x1, k2, %4, %8;\n"
#define RK_LAST_1 "add.rn.f32x2 %5, %3, %5;\n fma.rn.f32x2 %7, %20, %5, %7;\n mov.b64 %5, 0;\n"
#define RK_LAST_2 RK_LAST_1
#define RK_LAST_4 RK_LAST_1 "add.rn.f32x2 %6, %4, %6;\n fma.rn.f32x2 %8, %21, %6, %8;\n mov.b64 %6, 0;\n"

template <int RR>
struct Rollout {
    uint32_t temps; /* shared address of this lane's part of the warp's first temporary; the next lie 32 * RR floats further each */

    /* What stays the same for a warp while it integrates an item. */
    struct Item {
        uint32_t start, first;     /* shared address of the rewritten main part; its first handler */
        uint32_t own;              /* offset of this warp's state in the vector of stage values */
        uint32_t barrier, threads; /* of the item's warps; threads = 0: one warp, no barrier */
        uint32_t program, first_temp, table; /* the record's number; its first temporary slot; its constant table (RR copies of every entry) */
    };
    static __device__ __forceinline__ f2 pair(const float (&v)[RR], int i) { return sbm::pack2(v[RR > 2 ? 2 * i : 0], v[RR > 2 ? 2 * i + 1 : RR - 1]); }

    /* Integrates `steps` steps of this warp's state, whose base is `state`; now and other are the shared
     * addresses of the two vectors of stage values for this lane, and at the end `now` holds the new states
     * of all warps that have come this far. */
    __device__ __forceinline__ void interval(const Item& item, const DeviceBatch& batch, uint32_t steps, float (&state)[RR], const float (&half)[RR],
                                             const float (&h)[RR], const float (&sixth)[RR], uint32_t& now, uint32_t& other) {
        constexpr int W = RR > 2 ? 1 : 0; /* the second pair, where there is one */
        f2 a0 = 0ull, a1 = 0ull, sum0 = 0ull, sum1 = 0ull, st0 = pair(state, 0), st1 = pair(state, W);
        uint32_t ip = item.start, stage = 0u, handler, w;
#define RK_RUN(N)                                                                                                          \
        asm volatile(RK_CORE(N)                                                                                            \
                     : "+r"(ip), "=&r"(handler), "=&r"(w), "+l"(a0), "+l"(a1), "+l"(sum0), "+l"(sum1), "+l"(st0), "+l"(st1), "+r"(now), "+r"(other), \
                       "+r"(stage), "+r"(steps)                                                                             \
                     : "r"(temps), "l"(sbm::both2(-1.0f)), "l"(__cvta_generic_to_constant(kPairConstants)), "l"(pair(half, 0)), "l"(pair(half, W)), \
                       "l"(pair(h, 0)), "l"(pair(h, W)), "l"(pair(sixth, 0)), "l"(pair(sixth, W)), "r"(item.start), "r"(item.own),         \
                       "r"(item.barrier), "r"(item.threads), "r"(item.first)                                                                 \
                     : "memory")
#pragma unroll 1
        for (;;) {
            if constexpr (RR == 1) RK_RUN(1);
            else if constexpr (RR == 2) RK_RUN(2);
            else RK_RUN(4);
            if (handler == 0u) break;
            handler = lds_word(ip - 16u); /* of the instruction the core stopped at */
            slow(a0, a1, handler, w, now, batch, item.program, item.first_temp, (ip - item.start) / (uint32_t)sizeof(SbInsn) - 1u, item.table);
        }
#undef RK_RUN
        state[0] = sbm::lo2(st0);
        if constexpr (RR > 1) state[1] = sbm::hi2(st0);
        if constexpr (RR > 2) { state[2] = sbm::lo2(st1); state[3] = sbm::hi2(st1); }
    }
    /* what the core leaves to others: unusual arguments, the rarer functions, fused multiply-adds */
    __device__ __forceinline__ void slow(f2& a0, f2& a1, uint32_t h, uint32_t w, uint32_t states, const DeviceBatch& batch, uint32_t program,
                                         uint32_t first_temp, uint32_t at, uint32_t table) {
        if (h == H_FMA) { /* its three operands need the record's own words */
            const SbProgram* const pr = batch.programs + program;
            const SbInsn ins = batch.insns[pr->insn_off + pr->main_off + at];
            float acc[RR];
            acc[0] = sbm::lo2(a0);
            if constexpr (RR > 1) acc[1] = sbm::hi2(a0);
            if constexpr (RR > 2) { acc[2] = sbm::lo2(a1); acc[3] = sbm::hi2(a1); }
            fused(acc, ins.w0, ins.w1, states, first_temp, table);
            a0 = pair(acc, 0);
            a1 = pair(acc, RR > 2 ? 1 : 0);
            return;
        }
        if (h >= H_SIN) {
            a0 = unary_pair(a0, w);
            if constexpr (RR > 2) a1 = unary_pair(a1, w);
            return;
        }
        const uint32_t kind = (h - H_DIV) % 3u;
        float x[RR];
        lds<RR>(w + (kind == RK_STATE ? states : kind == RK_TEMP ? temps : 0u), x);
        const f2 x0 = pair(x, 0), x1 = pair(x, RR > 2 ? 1 : 0);
        const bool reverse = h >= H_RDIV;
        a0 = reverse ? div_pair(x0, a0) : div_pair(a0, x0);
        if constexpr (RR > 2) a1 = reverse ? div_pair(x1, a1) : div_pair(a1, x1);
    }

    /* FMA_F32 over three operands of any kind (table entry, slot, or the accumulator) */
    __device__ __forceinline__ void fused(float (&acc)[RR], uint32_t w0, uint32_t w1, uint32_t states, uint32_t first_temp, uint32_t table) {
        const unsigned kinds = (w0 >> 8) & 0x3fu;
        float v[3][RR];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const unsigned kind = (kinds >> (2 * i)) & 3u;
            const uint32_t index = (w1 >> (10 * i)) & 1023u;
            if (kind == SB_FMA_ACC) {
#pragma unroll
                for (int q = 0; q < RR; ++q) v[i][q] = acc[q];
            } else if (kind == SB_KIND_CST) lds<RR>(table + index * (uint32_t)(RR * 4), v[i]);
            else lds<RR>(index < first_temp ? states + index * (uint32_t)(RR * 128) : temps + (index - first_temp) * (uint32_t)(RR * 128), v[i]);
        }
#pragma unroll
        for (int q = 0; q < RR; ++q) acc[q] = __fmaf_rn(v[0][q], v[1][q], v[2][q]);
    }
};

/* Rewrites instruction `in` of a record's main part for the machine above; `table` is the shared address
 * of the record's constant table, `first_temp` the first slot that is a temporary (the ones before it are
 * the states). */
template <int RR>
__device__ __forceinline__ SbInsn rewritten(SbInsn in, uint32_t table, uint32_t first_temp) {
    const unsigned cs = in.w0 & 0xffu;
    const uint32_t idx = in.w0 >> 16;
    const auto made = [&](unsigned handler, unsigned kind, uint32_t i) {
        if (kind == SB_KIND_CST) return SbInsn{handler + RK_CST, table + i * (uint32_t)(RR * 4)};
        if (i < first_temp) return SbInsn{handler + RK_STATE, i * (uint32_t)(RR * 128)};
        return SbInsn{handler + RK_TEMP, (i - first_temp) * (uint32_t)(RR * 128)};
    };
    if (cs >= SB_CASE_LOAD && cs < SB_CASE_STORE) return made(H_LOAD, cs - SB_CASE_LOAD, idx);
    if (cs == SB_CASE_STORE && (in.w1 & SB_STORE_THEN_LOAD)) {
        SbInsn both = made(H_STLOAD, (in.w1 >> 16) & 3u, in.w1 & 0xffffu);
        both.w1 |= ((idx - first_temp) * (RR * 128u / kStoredUnit)) << kStoredShift;
        return both;
    }
    if (cs == SB_CASE_STORE) return SbInsn{H_STORE, (idx - first_temp) * (uint32_t)(RR * 128)};
    if (cs >= SB_CASE_BIN && cs < SB_CASE_UN) /* in the record's order of operations */
        return made(H_ADD + 3u * ((cs - SB_CASE_BIN) / SB_NUM_KINDS), (cs - SB_CASE_BIN) % SB_NUM_KINDS, idx);
    if (cs >= SB_CASE_UN && cs < SB_CASE_FMA) {
        const unsigned un = cs - SB_CASE_UN;
        const unsigned h = un == SB_UN_NEG ? H_NEG : un == SB_UN_ABS ? H_ABS : un == SB_UN_SIN ? H_SIN : un == SB_UN_COS ? H_COS
                         : un == SB_UN_EXP ? H_EXP : un == SB_UN_LOG ? H_LOG : un == SB_UN_TANH ? H_TANH : H_UNARY;
        return SbInsn{h, un};
    }
    if (cs == SB_CASE_FMA) return SbInsn{H_FMA, 0u};
    return SbInsn{H_END, 0u};
}

/* The bank part of a record (record.h): sub-expressions that depend on the candidate's constants
 * only, computed once per item instead of once per stage.  Every lane runs it on the same values
 * (no divergence, no exchange) and stores the same results: table entry e as RR adjacent copies, so
 * the main part reads a constant with the load it uses for a lane's slot values.  Operand kinds of
 * the bank part: CST = source constant (bank slots, affine entries, literals), ROW = table entry
 * written earlier, SLOT = scalar temporary.  The functions are the scalar pieces the wider
 * machines use, so a value has the bits it would have had in the main part. */
__device__ __noinline__ void rollout_bank_part(const SbInsn* code, const float* source, float* tmp, float* table, int copies) {
    float acc = 0.0f;
    auto operand = [&](unsigned kind, uint32_t idx) -> float {
        return kind == SB_KIND_ROW ? table[idx * copies] : kind == SB_KIND_SLOT ? tmp[idx] : source[idx];
    };
#pragma unroll 1
    for (;; ++code) {
        const SbInsn ins = *code;
        const unsigned cs = ins.w0 & 0xffu;
        const uint32_t idx = ins.w0 >> 16;
        if (cs == SB_CASE_END || cs > SB_CASE_FMA) return;
        if (cs < SB_CASE_STORE) acc = operand(cs - SB_CASE_LOAD, idx);
        else if (cs == SB_CASE_STORE) tmp[idx] = acc;
        else if (cs == SB_CASE_STOREH) {
            for (int q = 0; q < copies; ++q) table[idx * copies + q] = acc;
        } else if (cs < SB_CASE_UN) {
            const float x = operand((cs - SB_CASE_BIN) % SB_NUM_KINDS, idx);
            switch ((cs - SB_CASE_BIN) / SB_NUM_KINDS) {
            case SB_BIN_ADD: acc = __fadd_rn(acc, x); break;
            case SB_BIN_SUB: acc = __fsub_rn(acc, x); break;
            case SB_BIN_RSUB: acc = __fsub_rn(x, acc); break;
            case SB_BIN_MUL: acc = __fmul_rn(acc, x); break;
            case SB_BIN_DIV: acc = __fdiv_rn(acc, x); break;
            case SB_BIN_RDIV: acc = __fdiv_rn(x, acc); break;
            case SB_BIN_MIN: acc = fminf(acc, x); break;
            default: acc = fmaxf(acc, x); break;
            }
        } else if (cs < SB_CASE_FMA) {
            const unsigned op = cs - SB_CASE_UN;
            acc = op == SB_UN_NEG ? -acc : op == SB_UN_ABS ? fabsf(acc) : sbm::any1(acc, op);
        } else {
            const unsigned kinds = (ins.w0 >> 8) & 0x3fu;
            float v[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const unsigned kind = (kinds >> (2 * i)) & 3u;
                v[i] = kind == SB_FMA_ACC ? acc : operand(kind, (ins.w1 >> (10 * i)) & 1023u);
            }
            acc = __fmaf_rn(v[0], v[1], v[2]);
        }
    }
}

/* projects/odezza/core/o_sampled_constants_source.h:32-44 */
__device__ __forceinline__ float sampled_constant(const Rk4Problem& prob, unsigned long long index, uint32_t bank) {
    const SecantB200SampledParameter p = prob.sampled[index];
    if (!p.distribution) return p.shift;
    const unsigned long long delta = (unsigned long long)bank * p.stride;
    if (p.offset >= prob.pool_size || delta >= prob.pool_size - p.offset) return __int_as_float(0x7fc00000);
    const float* pool = p.distribution == 1 ? prob.uniform_pool : p.distribution == 2 ? prob.normal_pool : nullptr;
    if (!pool) return __int_as_float(0x7fc00000);
    const float value = __fadd_rn(__fmul_rn(pool[p.offset + delta], p.scale), p.shift);
    return fminf(p.upper, fmaxf(p.lower, value));
}

/* h / 6 rounded to nearest, for h >= 0: the quotient's estimate and one correction (Markstein) give the
 * rounded quotient for every significand (checked for all 2^24), as long as nothing underflows. */
__device__ __forceinline__ float sixth_of(float h) {
    if (h != 0.0f && !(h > 1e-30f)) return h / 6.0f;
    const float c = 1.0f / 6.0f, q = __fmul_rn(h, c);
    return __fmaf_rn(__fmaf_rn(-6.0f, q, h), c, q);
}

/* Shared memory of one group (the S warps of an item): the two vectors of stage values, S states each,
 * and one word for the item's number; then per warp the record of its right-hand side (exec_bytes), its
 * constant table (table_bytes), its source constants and bank-part temporaries (source_bytes), its
 * temporaries (temp_bytes). */
struct RolloutLayout {
    uint32_t exec_bytes, table_bytes, source_bytes, temp_bytes, warp_bytes, group_bytes;
};

/* The S warps of a group meet at a named barrier of their own; a group of one warp needs none. */
__device__ __forceinline__ void group_sync(uint32_t barrier, uint32_t threads) {
    if (threads == 32u) __syncwarp();
    else asm volatile("barrier.cta.sync %0, %1;" ::"r"(barrier), "r"(threads) : "memory");
}
__device__ __forceinline__ bool group_all(uint32_t barrier, uint32_t threads, bool ok) { /* also a barrier */
    if (threads == 32u) return __all_sync(0xffffffffu, ok);
    uint32_t all;
    asm volatile("{ .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.and.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n }"
                 : "=r"(all) : "r"((uint32_t)ok), "r"(barrier), "r"(threads) : "memory");
    return all != 0u;
}

/* An item (system, configuration) is integrated by S warps, one per state: the right-hand sides of a stage
 * are independent, so the chain of dependent instructions that decides how long an item takes is that of
 * the longest right-hand side and not that of all of them.  A warp keeps its own state, stage sum and step
 * sizes in registers; the stage values are in shared memory twice, so one barrier per stage is enough
 * (a warp writes the next stage's value of its state while others still read this stage's).
 * 4,096 systems of three states, 64 trajectories, 1,000 steps: 71.8 ms with one warp per item and the
 * machine in C++, 23.8 now; the warps that are resident (30 of an SM's 64, by their registers) issue in
 * 45 % of the cycles, and wait for one another at the barriers for a third of their time. */
template <int RR>
__global__ void __launch_bounds__(kRolloutMaxWarps * 32, RR == 4 ? 1 : 2)
rk4_kernel(const DeviceBatch batch, const Rk4Problem prob, const RolloutLayout lay) {
    constexpr uint32_t PASS = 32 * RR; /* trajectories of one pass */
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t S = prob.num_states, K = prob.num_constants;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, group = warp / S, s = warp - group * S;
    const uint32_t barrier = group + 1u, threads = S * 32u;
    unsigned char* const garea = smem + (size_t)group * lay.group_bytes;
    const uint32_t stage_bytes = S * (uint32_t)(RR * 128);
    const uint32_t stage0 = shared_address(garea) + lane * (uint32_t)(RR * 4); /* this lane's part of the first vector; the second follows it */
    volatile unsigned long long* const item_word = reinterpret_cast<volatile unsigned long long*>(garea + 2u * stage_bytes);
    unsigned char* const warea = garea + 2u * stage_bytes + 16u + (size_t)s * lay.warp_bytes;
    SbInsn* const exec = reinterpret_cast<SbInsn*>(warea) + 1; /* the entry before the first holds the first handler */
    float* const table = reinterpret_cast<float*>(warea + lay.exec_bytes);
    float* const source = reinterpret_cast<float*>(warea + lay.exec_bytes + lay.table_bytes);
    float* const tmp = source + K + batch.max_extra;
    const uint32_t table_address = shared_address(table), first_temp = S; /* the states' slots come first */
    Rollout<RR> m;
    m.temps = shared_address(warea + lay.exec_bytes + lay.table_bytes + lay.source_bytes) + lane * (uint32_t)(RR * 4);
    const unsigned long long configs = (unsigned long long)prob.num_banks << prob.toggle_bits;
    const unsigned long long num_items = configs * prob.num_systems;
    /* Items are drawn from a device-wide counter: a group whose candidate went invalid early takes
     * the next one at once, and no warp slot idles behind the longest item of its CTA. */
#pragma unroll 1
    for (;;) {
    unsigned long long item = 0;
    if (s == 0 && lane == 0) item = atomicAdd(prob.queue, 1ull);
    if (S > 1) {
        if (s == 0 && lane == 0) *item_word = item;
        group_sync(barrier, threads);
        item = *item_word;
    } else {
        item = __shfl_sync(0xffffffffu, item, 0);
    }
    if (item >= num_items) break;
    const uint32_t turn = (uint32_t)(item / configs);
    const uint32_t sys = prob.order ? prob.order[turn] : turn;
    const unsigned long long cfg = item - turn * configs;
    const unsigned long long perm = cfg & ((1ull << prob.toggle_bits) - 1ull);
    const uint32_t bank = (uint32_t)(cfg >> prob.toggle_bits);
    /* configurations that differ only in toggle bits the system does not read have one score: the one
     * where those bits are 0 is integrated, and its group writes the others (600 systems of two states,
     * two bits, three sets: two thirds of the items, 1.31 -> 1.09 ms a call) */
    uint32_t unread = (uint32_t)((1ull << prob.toggle_bits) - 1ull);
    for (uint32_t c = 0; c < S; ++c) unread &= ~batch.programs[sys * S + c].bit_mask;
    if (perm & unread) {
        group_sync(barrier, threads); /* the item's number has been read */
        continue;
    }
    unsigned int integrated = 0; /* (trajectory, observation interval) pairs this lane carries out */
    const float* bank_ptr = prob.banks ? prob.banks + (size_t)sys * prob.system_bank_stride + (size_t)bank * prob.bank_stride : nullptr;

    /* private copy of the right-hand side: toggles resolved, the bank part run once, the main part
     * rewritten for the machine */
    const SbProgram* const pr = batch.programs + sys * S + s;
    const uint32_t n_insn = pr->n_insn, main_off = pr->main_off;
    {
        const uint32_t n_patch = pr->n_patch, n_affine = pr->n_affine, n_source = K + n_affine + pr->n_lits;
#pragma unroll 1
        for (uint32_t i = lane; i < n_insn; i += 32) exec[i] = batch.insns[pr->insn_off + i];
        __syncwarp();
#pragma unroll 1
        for (uint32_t i = lane; i < n_patch; i += 32) {
            const SbPatch* p = batch.patches + pr->patch_off + i;
            unsigned choice = (unsigned)(perm >> p->bit0) & 1u;
            if (p->bit1 != 0xffu) choice |= ((unsigned)(perm >> p->bit1) & 1u) << 1;
            exec[p->insn] = p->alt[choice];
        }
#pragma unroll 1
        for (uint32_t e = lane; e < n_source; e += 32) {
            float v;
            if (e < K) v = prob.sampled ? sampled_constant(prob, (unsigned long long)sys * K + e, bank) : bank_ptr[e];
            else if (e < K + n_affine) {
                const SbAffine a = batch.affines[pr->affine_off + e - K];
                const float slot = prob.sampled ? sampled_constant(prob, (unsigned long long)sys * K + a.slot, bank) : bank_ptr[a.slot];
                v = __fadd_rn(__fmul_rn(slot, a.scale), a.offset);
            } else v = batch.lits[pr->lit_off + e - K - n_affine];
            source[e] = v;
        }
        __syncwarp();
        if (main_off) rollout_bank_part(exec, source, tmp, table, RR);
        __syncwarp();
#pragma unroll 1
        for (uint32_t i0 = main_off; i0 < n_insn; i0 += 32) { /* in place: every lane reads before any writes */
            const uint32_t i = i0 + lane;
            const SbInsn made = i < n_insn ? rewritten<RR>(exec[i], table_address, first_temp) : SbInsn{H_END, 0u};
            __syncwarp();
            if (i < n_insn) {
                (exec + i)[-1].w0 = made.w0;
                exec[i].w1 = made.w1;
            }
            __syncwarp();
        }
    }
    const typename Rollout<RR>::Item place{shared_address(exec + main_off), lds_word(shared_address(exec + main_off) - 8u), s * (uint32_t)(RR * 128), barrier, S > 1 ? threads : 0u,
                                           sys * S + s, first_temp, table_address};

    const bool ragged = prob.offsets != nullptr;
    float sq = 0.0f;
    unsigned long long residuals = 0;
    /* any non-finite time or reference value (NaN excepted where it means "unobserved"), found
     * by the validation kernel, invalidates every score; so do offsets that do not span the data */
    bool ok = *prob.invalid_flag == 0;
    if (ragged) ok = ok && prob.offsets[0] == 0u && prob.offsets[prob.num_trajectories] == prob.total_points;
    /* a candidate that is already invalid scores FLT_MAX whatever follows: the group stops integrating it */
    bool alive = group_all(barrier, threads, ok);
    uint32_t now = stage0, other = stage0 + stage_bytes; /* the vectors of this stage's values and of the next stage's */
#pragma unroll 1
    for (uint32_t t0 = 0; t0 < prob.num_trajectories && alive; t0 += PASS) {
        uint32_t at[RR], npts[RR], longest = 0; /* the point a trajectory has reached; its number of points */
        float state[RR], reached[RR], next[RR]; /* the times of that point and of the one after it */
        const float* const reference = prob.reference + (size_t)s * prob.reference_ld; /* of this warp's state */
#pragma unroll
        for (int q = 0; q < RR; ++q) {
            const uint32_t traj = t0 + lane * RR + q;
            const bool live = traj < prob.num_trajectories;
            at[q] = 0; npts[q] = 0;
            if (live && ragged) {
                const uint32_t b = prob.offsets[traj], e = prob.offsets[traj + 1];
                const bool sane = e > b && e <= prob.total_points;
                ok = ok && sane;
                if (sane) { at[q] = b; npts[q] = e - b; }
            } else if (live) {
                at[q] = traj * prob.points_per_trajectory; npts[q] = prob.points_per_trajectory;
            }
            longest = max(longest, npts[q]);
            state[q] = npts[q] ? reference[at[q]] : 0.0f;
            reached[q] = npts[q] ? prob.times[ragged ? at[q] : 0u] : 0.0f;
            next[q] = npts[q] > 1u ? prob.times[ragged ? at[q] + 1u : 1u] : 0.0f;
            ok = ok && (fabsf(state[q]) <= kFltMax); /* initial states must be complete and finite */
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
        sts<RR>(now + s * (uint32_t)(RR * 128), state);
        alive = group_all(barrier, threads, ok);
#pragma unroll 1
        for (uint32_t k = 1; k < longest && alive; ++k) {
            /* per trajectory step size; a trajectory that has ended keeps integrating with h = 0
             * and is left out of every check and sum.  What memory holds for the end of this interval
             * and for the next one is asked for here and used after the interval's stages. */
            float h[RR], half[RR], sixth[RR], expected[RR];
#pragma unroll
            for (int q = 0; q < RR; ++q) {
                const bool act = k < npts[q];
                const float interval = act ? next[q] - reached[q] : 0.0f;
                const float step = prob.substeps == 1u ? interval : interval / (float)prob.substeps;
                ok = ok && (!act || ((fabsf(interval) <= kFltMax) && interval > 0.0f && step > 0.0f));
                h[q] = act ? step : 0.0f;
                half[q] = __fmul_rn(0.5f, h[q]);
                sixth[q] = sixth_of(h[q]);
                integrated += act ? 1u : 0u;
                reached[q] = next[q];
                ++at[q];
                expected[q] = act ? reference[at[q]] : 0.0f;
                if (k + 1u < npts[q]) next[q] = prob.times[ragged ? at[q] + 1u : k + 1u];
            }
            m.interval(place, batch, prob.substeps, state, half, h, sixth, now, other);
#pragma unroll
            for (int q = 0; q < RR; ++q)
                if (k < npts[q]) {
                    ok = ok && fabsf(state[q]) <= kFltMax; /* one state that is not finite and no residual counts */
                    if (prob.allow_missing && expected[q] != expected[q]) continue; /* unobserved */
                    const float err = __fsub_rn(state[q], expected[q]);
                    sq = __fmaf_rn(err, err, sq);
                    ++residuals;
                }
            alive = group_all(barrier, threads, ok);
        }
    }
    /* the warps' sums meet in their source areas, which the next item fills only after another barrier */
#pragma unroll
    for (int d = 16; d; d >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
    {
        uint32_t lo = (uint32_t)residuals, hi = (uint32_t)(residuals >> 32);
#pragma unroll
        for (int d = 16; d; d >>= 1) {
            residuals += ((unsigned long long)__shfl_xor_sync(0xffffffffu, hi, d) << 32) | __shfl_xor_sync(0xffffffffu, lo, d);
            lo = (uint32_t)residuals; hi = (uint32_t)(residuals >> 32);
        }
    }
    if (lane == 0) {
        source[0] = sq;
        source[1] = __uint_as_float((uint32_t)residuals);
        source[2] = __uint_as_float((uint32_t)(residuals >> 32));
    }
    group_sync(barrier, threads);
    if (s == 0 && lane == 0) {
        float total = sq;
        for (uint32_t c = 1; c < S; ++c) {
            const float* other_source = source + (size_t)c * (lay.warp_bytes / 4u);
            total += other_source[0];
            residuals += ((unsigned long long)__float_as_uint(other_source[2]) << 32) | __float_as_uint(other_source[1]);
        }
        const bool finite = fabsf(total) <= kFltMax;
        sq = (alive && residuals && finite) ? total / (float)residuals : kFltMax;
    }
    if (s == 0) {
        sq = __shfl_sync(0xffffffffu, sq, 0);
        const unsigned long long copies = 1ull << __popc(unread);
        float* const out = prob.output + (size_t)sys * prob.output_ld + cfg;
#pragma unroll 1
        for (unsigned long long x = lane; x < copies; x += 32u) out[deposit((uint32_t)x, unread)] = sq;
        if (prob.integrated) { /* counted for every configuration that has the score */
#pragma unroll
            for (int d = 16; d; d >>= 1) integrated += __shfl_xor_sync(0xffffffffu, integrated, d);
            if (lane == 0) atomicAdd(prob.integrated, (unsigned long long)integrated * copies);
        }
    }
    if (S == 1) __syncwarp(); /* a group of several meets again before anything is overwritten */
    }
}

/* Raises *flag when a time or a reference value of an active state is not finite; NaN reference
 * values are tolerated when they mean "unobserved" (initial points are checked by the scorer). */
__global__ void rk4_validate_kernel(const Rk4Problem prob) {
    const size_t n = (size_t)prob.total_points * (prob.num_states + 1);
    bool bad = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i / prob.total_points, col = i % prob.total_points;
        if (row == prob.num_states) {
            if (!prob.offsets && col >= prob.points_per_trajectory) continue; /* uniform form: one shared time axis */
            bad = bad || !(fabsf(prob.times[col]) <= kFltMax);
        } else {
            const float v = prob.reference[row * prob.reference_ld + col];
            bad = bad || !((fabsf(v) <= kFltMax) || (prob.allow_missing && v != v));
        }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(prob.invalid_flag, 1);
}

uint32_t round16(size_t v) { return (uint32_t)((v + 15) / 16 * 16); }

template <int RR>
cudaError_t launch_width(const DeviceBatch& batch, const Rk4Problem& prob, size_t smem_limit, cudaStream_t stream) {
    RolloutLayout lay;
    const uint32_t S = prob.num_states;
    lay.exec_bytes = round16(((size_t)batch.max_insn + 1) * sizeof(SbInsn));
    lay.table_bytes = round16(((size_t)batch.max_cst + 1) * RR * 4);
    lay.source_bytes = round16(((size_t)prob.num_constants + batch.max_extra + batch.max_btmp) * 4 + 16);
    /* max_slots counts the states' slots, which the records leave before their temporaries */
    lay.temp_bytes = (batch.max_slots > S ? batch.max_slots - S : 0u) * (uint32_t)RR * 128u;
    lay.warp_bytes = lay.exec_bytes + lay.table_bytes + lay.source_bytes + lay.temp_bytes;
    lay.group_bytes = 2u * S * (uint32_t)(RR * 128) + 16u + S * lay.warp_bytes;
    /* groups per CTA: the count that puts most warps on an SM (shared memory per SM is the CTA limit
     * plus 1 KB reserved per resident CTA; the register file holds 64 K registers, allocated per warp
     * in units of 256; a CTA has fifteen barriers to give to groups) */
    cudaFuncAttributes attributes;
    cudaError_t e = cudaFuncGetAttributes(&attributes, rk4_kernel<RR>);
    if (e != cudaSuccess) return e;
    const int warp_registers = (attributes.numRegs * 32 + 255) / 256 * 256;
    const int register_warps = std::min(64, 65536 / std::max(256, warp_registers));
    int groups = 0, best = 0;
    for (int g = 1; g <= 15 && g * (int)S <= kRolloutMaxWarps; ++g) {
        const size_t cta = (size_t)lay.group_bytes * g;
        if (cta > smem_limit) break;
        const int ctas = std::min((int)((smem_limit + 1024) / (cta + 1024)), register_warps / (g * (int)S));
        if (ctas && ctas * g >= best) { best = ctas * g; groups = g; }
    }
    const int warps = groups * (int)S;
    /* a parked temporary's offset has 14 bits, a state's 18 with the rest of the word */
    if (!groups || batch.max_slots * (uint32_t)RR > 16383u) return cudaErrorInvalidConfiguration;
    const size_t smem = (size_t)lay.group_bytes * groups;
    e = cudaFuncSetAttribute(rk4_kernel<RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit);
    if (e != cudaSuccess) return e;
    /* the largest shared-memory carve-out, always: left to itself the driver gave a CTA that fits the
     * 100 KB configuration that one, and only one CTA per SM became resident where two were planned
     * (measured: a call took 169 ms instead of 117 when its CTAs shrank from 101 KB to 98.8 KB) */
    e = cudaFuncSetAttribute(rk4_kernel<RR>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    const unsigned long long items = ((unsigned long long)prob.num_banks << prob.toggle_bits) * prob.num_systems;
    /* warps draw items from the queue until it is empty, so the grid only has to fill the device */
    int device = 0, sms = 0;
    if ((e = cudaGetDevice(&device)) != cudaSuccess || (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return e;
    const unsigned long long resident = (unsigned long long)sms * (unsigned)std::max(1, best / groups);
    const unsigned long long blocks = std::min<unsigned long long>((items + groups - 1) / groups, resident);
    rk4_kernel<RR><<<(unsigned)blocks, warps * 32, smem, stream>>>(batch, prob, lay);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_rk4_validation(const Rk4Problem& prob, cudaStream_t stream) {
    const size_t values = (size_t)prob.total_points * (prob.num_states + 1);
    rk4_validate_kernel<<<(unsigned)std::min<size_t>(1024, (values + 255) / 256), 256, 0, stream>>>(prob);
    return cudaGetLastError();
}

/* Trajectories per lane: the fewest whose pass holds them all, and four beyond 64.  Milliseconds a call with
 * 1 / 2 / 4 of them, 2,048 systems of three states, 200 steps: 32 trajectories 4.6 / 4.7 / 6.1, 33: 7.7 / 4.9 /
 * 6.3, 64: 7.6 / 4.6 / 6.4, 65: 10.5 / 7.7 / 6.7, 128: 14.1 / 8.0 / 6.2, 512: 51 / 26 / 19.  The widest form has
 * 120 registers, so 16 warps per SM instead of 30, and still wins beyond 64 because it walks half the passes;
 * with eight states the two meet between 129 and 192 trajectories (6.3 against 6.6, 6.7 against 7.1 ms for
 * 1,024 systems, 100 steps), before that and after it the wider one is ahead there too. */
cudaError_t launch_rk4(const DeviceBatch& batch, const Rk4Problem& prob, size_t smem_limit, cudaStream_t stream) {
    if (prob.num_trajectories <= 32) return launch_width<1>(batch, prob, smem_limit, stream);
    if (prob.num_trajectories <= 64) return launch_width<2>(batch, prob, smem_limit, stream);
    return launch_width<4>(batch, prob, smem_limit, stream);
}

}  // namespace sb
