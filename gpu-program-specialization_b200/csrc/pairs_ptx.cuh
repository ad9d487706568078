/*
 * pairs_ptx.cuh - the accurate functions and the division on pairs of floats, as PTX text for the
 * interpreters' cores (eval_kernel.cuh, rollout.cu).
 *
 * The same steps, in the same order, as the scalar versions of sbmath.cuh, so a value has the same bits
 * whichever computed it.  They work on named registers the cores declare (SB_PTX_REGISTERS), take the
 * pair to be replaced as their argument, and hold for the common range of arguments only: a core
 * compares the magnitudes first (SB_TOP, SB_LOW: three at a time, NaN wins) and leaves its block with
 * the whole warp when an argument is outside (SB_ALL_OR_LEAVE, a label LEAVE).
 */
#ifndef SECANT_B200_PAIRS_PTX_CUH
#define SECANT_B200_PAIRS_PTX_CUH

#define SB_PTX_REGISTERS ".reg .u32 ad, c0, c1, c2, c3, c4, c5;\n .reg .f32 f0, f1, top, low;\n .reg .b64 m, t, n, r, z, q, hf, nh, mone, k<12>;\n .reg .pred p;\n"
#define SB_PTX_REGISTERS_ANY ".reg .b64 v, at, g<10>;\n .reg .f64 d<4>;\n .reg .b32 w0, w1, u0, u1, s0, s1;\n" /* what SB_SIN_ANY takes besides */
#define SB_PAIR_CONST(R, BITS) "mov.b64 " R ", " BITS ";\n"
#define SB_TOP(A) "mov.b64 {f0, f1}, " A ";\n max.NaN.abs.f32 top, top, f0, f1;\n"
/* the same without regard to NaN, which the steps of sine, cosine and division pass on */
#define SB_TOP_NUMBER(A) "mov.b64 {f0, f1}, " A ";\n max.abs.f32 top, top, f0, f1;\n"
#define SB_LOW_NUMBER(A) "mov.b64 {f0, f1}, " A ";\n min.abs.f32 low, low, f0, f1;\n"
#define SB_LOW(A) "mov.b64 {f0, f1}, " A ";\n min.NaN.f32 low, low, f0, f1;\n"
#define SB_VOTE "vote.sync.all.pred p, p, 0xffffffff;\n"
#define SB_ALL_OR_LEAVE SB_VOTE "@!p bra.uni LEAVE;\n"
/* Constants of the steps below, each the bits of a float32 and written once: the evaluator's core moves them into
 * registers (SB_*_CONSTANTS), the rollout core reads them from a table of pairs (SB_PAIR_WORD, rollout.cu) and
 * the scalar functions name them (sbmath.cuh). */
#define SB_PAIR_TEXT(I, BITS) "mov.b64 k" #I ", 0x" #BITS #BITS ";\n"
#define SB_PAIR_WORD(I, BITS) 0x##BITS##BITS##ull,
#define SB_SIN_LIST(X) \
    X(0, 3EA2F983) X(1, 4B400000) X(2, CB400000) X(3, C0490FDB) X(4, 33BBBD2E) X(5, 27772CED) \
    X(6, B2CD31C1) X(7, 3638B824) X(8, B9500BEC) X(9, 3C088886) X(10, BE2AAAAB)
#define SB_TRIG_LIST(X) \
    X(0, 3FC90FDB) X(1, B94CA22D) X(2, 3C08839E) X(3, BE2AAAA3) X(4, B4920F5C) \
    X(5, 37D00870) X(6, BAB60B5C) X(7, 3D2AAAAB) X(8, BF000000) X(9, 3F800000)
#define SB_EXP_LIST(X) \
    X(0, 3FB8AA3B) X(1, 4B400000) X(2, 32A57060)
#define SB_LOG_LIST(X) \
    X(0, CB400000) X(1, BD9C5854) X(2, 3E02AC14) X(3, BE06C251) X(4, 3E116D42) X(5, BE2A392F) \
    X(6, 3E4CD002) X(7, BE800113) X(8, 3EAAAAAA) X(9, BF000000) X(10, 35BFBE8E) X(11, 3F317200)
#define SB_DIV_LIST(X) \
    X(0, 3F800000)
#define SB_SIN_CONSTANTS SB_SIN_LIST(SB_PAIR_TEXT)
#define SB_EXP_CONSTANTS SB_EXP_LIST(SB_PAIR_TEXT)
#define SB_LOG_CONSTANTS SB_LOG_LIST(SB_PAIR_TEXT)
#define SB_DIV_CONSTANTS SB_DIV_LIST(SB_PAIR_TEXT)
#define SB_TANH_CONSTANTS SB_TANH_LIST(SB_PAIR_TEXT)
#define SB_MINUS_ONE "mov.b64 mone, 0xBF800000BF800000;\n"
/* (the sign is added: shift and addition are one instruction, shift and xor two)
 * sin and cos differ in the shift by half a turn, taken off again after the rounding */
#define SB_SIN_SHIFT "mov.b64 hf, 0;\n mov.b64 nh, 0x8000000080000000;\n"
#define SB_COS_SHIFT "mov.b64 hf, 0x3F0000003F000000;\n mov.b64 nh, 0xBF000000BF000000;\n"
#define SB_SIN_PAIR(A)                                                                                  \
    "fma.rn.f32x2 t, " A ", k0, hf;\n add.rn.f32x2 t, t, k1;\n add.rn.f32x2 n, t, k2;\n add.rn.f32x2 n, n, nh;\n" \
    "fma.rn.f32x2 r, n, k3, " A ";\n fma.rn.f32x2 r, n, k4, r;\n fma.rn.f32x2 r, n, k5, r;\n mul.rn.f32x2 z, r, r;\n" \
    "fma.rn.f32x2 q, k6, z, k7;\n fma.rn.f32x2 q, q, z, k8;\n fma.rn.f32x2 q, q, z, k9;\n fma.rn.f32x2 q, q, z, k10;\n" \
    "mul.rn.f32x2 z, r, z;\n fma.rn.f32x2 r, z, q, r;\n mov.b64 {c0, c1}, t;\n shl.b32 c0, c0, 31;\n shl.b32 c1, c1, 31;\n" \
    "mov.b64 {c2, c3}, r;\n add.u32 c0, c0, c2;\n add.u32 c1, c1, c3;\n mov.b64 " A ", {c0, c1};\n"
/* sin or cos of any pair (the shift says which, TURNS is the address of the table of sbmath.cuh): the steps above, and for a pair
 * with a large argument somewhere in the warp those of sincos_large() as well.  Labels DONE and DONE"D" are the macro's own. */
#define SB_TRIG_TEXT(I, BITS) "mov.b64 g" #I ", 0x" #BITS #BITS ";\n"
#define SB_SIN_TURNS(W, F, Q, TURNS)                                                                    \
    "shr.u32 c0, " W ", 23;\n and.b32 c0, c0, 255;\n max.u32 c0, c0, 177;\n min.u32 c0, c0, 254;\n shl.b32 c0, c0, 4;\n cvt.u64.u32 at, c0;\n" \
    "add.u64 at, at, " TURNS ";\n ld.global.nc.v2.f64 {d0, d1}, [at+-2832];\n and.b32 c0, " W ", 0x007FFFFF;\n shr.u32 c0, c0, 3;\n" \
    "and.b32 c1, " W ", 0x80000000;\n or.b32 c0, c0, c1;\n or.b32 c1, c0, 0x3FF00000;\n shl.b32 c0, " W ", 29;\n mov.b64 d2, {c0, c1};\n" \
    "mul.rn.f64 d0, d2, d0;\n fma.rn.f64 d3, d2, d1, d0;\n add.rn.f64 d3, d3, 0d4338000000000000;\n mov.b64 {" Q ", c1}, d3;\n add.rn.f64 d3, d3, 0dC338000000000000;\n" \
    "sub.rn.f64 d0, d0, d3;\n fma.rn.f64 d0, d2, d1, d0;\n cvt.rn.f32.f64 " F ", d0;\n"
#define SB_SIN_DOUBLE(W, F, Q) /* the same below 2^50, with 2/pi in two parts */                           \
    "mov.b32 " F ", " W ";\n cvt.f64.f32 d2, " F ";\n mul.rn.f64 d0, d2, 0d3FE45F306DC9C883;\n neg.f64 d1, d0;\n" \
    "fma.rn.f64 d1, d2, 0d3FE45F306DC9C883, d1;\n fma.rn.f64 d1, d2, 0dBC86B01EC5417056, d1;\n add.rn.f64 d3, d0, 0d4338000000000000;\n" \
    "mov.b64 {" Q ", c1}, d3;\n add.rn.f64 d3, d3, 0dC338000000000000;\n sub.rn.f64 d0, d0, d3;\n add.rn.f64 d0, d0, d1;\n cvt.rn.f32.f64 " F ", d0;\n"
#define SB_SIN_BEYOND(W, F, Q, TURNS) /* takes it from the table at 2^50 and beyond */                     \
    SB_SIN_TURNS(W, "low", "s1", TURNS) "and.b32 c0, " W ", 0x7FFFFFFF;\n setp.ge.u32 p, c0, 0x58800000;\n" \
    "selp.f32 " F ", low, " F ", p;\n selp.b32 " Q ", s1, " Q ", p;\n"
#define SB_SIN_CHOOSE(W, Q, S, C, V) /* the quadrant's function and sign, where the argument is large and finite */ \
    "add.u32 " Q ", " Q ", c3;\n and.b32 c0, " Q ", 1;\n setp.ne.u32 p, c0, 0;\n selp.b32 c0, " C ", " S ", p;\n and.b32 c1, " Q ", 2;\n" \
    "shl.b32 c1, c1, 30;\n xor.b32 c0, c0, c1;\n and.b32 c1, " W ", 0x7FFFFFFF;\n sub.u32 c1, c1, 0x45800000;\n setp.lt.u32 p, c1, 0x3A000000;\n" \
    "selp.b32 " V ", c0, " V ", p;\n"
#define SB_SIN_ANY(A, TURNS, DONE)                                                                      \
    "mov.b64 v, " A ";\n mov.f32 top, 0f00000000;\n" SB_TOP_NUMBER("v") "setp.lt.f32 p, top, 0f45800000;\n vote.sync.all.pred p, p, 0xffffffff;\n" \
    SB_SIN_PAIR(A) "@p bra.uni " DONE ";\n mov.b64 {w0, w1}, v;\n" SB_SIN_DOUBLE("w0", "f0", "u0") SB_SIN_DOUBLE("w1", "f1", "u1") \
    "setp.lt.f32 p, top, 0f58800000;\n" SB_VOTE "@p bra.uni " DONE "D;\n" SB_SIN_BEYOND("w0", "f0", "u0", TURNS) SB_SIN_BEYOND("w1", "f1", "u1", TURNS) DONE "D:\n" \
    SB_TRIG_LIST(SB_TRIG_TEXT) "mov.b64 r, {f0, f1};\n mul.rn.f32x2 r, r, g0;\n mul.rn.f32x2 z, r, r;\n fma.rn.f32x2 q, g1, z, g2;\n" \
    "fma.rn.f32x2 q, q, z, g3;\n mul.rn.f32x2 t, r, z;\n fma.rn.f32x2 r, t, q, r;\n fma.rn.f32x2 q, g4, z, g5;\n fma.rn.f32x2 q, q, z, g6;\n" \
    "fma.rn.f32x2 q, q, z, g7;\n mul.rn.f32x2 t, z, z;\n mul.rn.f32x2 z, z, g8;\n fma.rn.f32x2 q, t, q, z;\n add.rn.f32x2 q, q, g9;\n" \
    "mov.b64 {c3, c4}, hf;\n shr.u32 c3, c3, 24;\n and.b32 c3, c3, 1;\n"                             \
    "mov.b64 {f0, f1}, r;\n mov.b64 {top, low}, q;\n mov.b64 {s0, s1}, " A ";\n" SB_SIN_CHOOSE("w0", "u0", "f0", "top", "s0") \
    SB_SIN_CHOOSE("w1", "u1", "f1", "low", "s1") "mov.b64 " A ", {s0, s1};\n " DONE ":\n"
#define SB_EXP_PAIR(A)                                                                                  \
    "fma.rn.f32x2 t, " A ", k0, k1;\n fma.rn.f32x2 n, t, mone, k1;\n fma.rn.f32x2 r, " A ", k0, n;\n fma.rn.f32x2 r, " A ", k2, r;\n" \
    "mov.b64 {f0, f1}, r;\n ex2.approx.ftz.f32 f0, f0;\n ex2.approx.ftz.f32 f1, f1;\n mov.b64 {c0, c1}, t;\n" \
    "shl.b32 c0, c0, 23;\n shl.b32 c1, c1, 23;\n mov.b32 c2, f0;\n mov.b32 c3, f1;\n add.u32 c0, c0, c2;\n add.u32 c1, c1, c3;\n" \
    "mov.b64 " A ", {c0, c1};\n"
/* e^x of any pair: the steps of exp_pair() (sbmath.cuh) */
#define SB_EXP_ANY(A)                                                                                   \
    "mov.b64 {f0, f1}, " A ";\n max.NaN.f32 f0, f0, 0fC2D00000;\n max.NaN.f32 f1, f1, 0fC2D00000;\n min.NaN.f32 f0, f0, 0f42B20000;\n" \
    "min.NaN.f32 f1, f1, 0f42B20000;\n mov.b64 m, {f0, f1};\n fma.rn.f32x2 t, m, k0, k1;\n fma.rn.f32x2 n, t, mone, k1;\n" \
    "fma.rn.f32x2 r, m, k0, n;\n fma.rn.f32x2 r, m, k2, r;\n mov.b64 {f0, f1}, r;\n ex2.approx.ftz.f32 f0, f0;\n ex2.approx.ftz.f32 f1, f1;\n" \
    "mov.b64 r, {f0, f1};\n mov.b64 {c0, c1}, t;\n shr.s32 c2, c0, 1;\n shr.s32 c3, c1, 1;\n sub.u32 c0, c0, c2;\n sub.u32 c1, c1, c3;\n" \
    "shl.b32 c0, c0, 23;\n shl.b32 c1, c1, 23;\n shl.b32 c2, c2, 23;\n shl.b32 c3, c3, 23;\n add.u32 c0, c0, 0x3F800000;\n add.u32 c1, c1, 0x3F800000;\n" \
    "add.u32 c2, c2, 0x3F800000;\n add.u32 c3, c3, 0x3F800000;\n mov.b64 m, {c2, c3};\n mul.rn.f32x2 r, r, m;\n mov.b64 m, {c0, c1};\n" \
    "mul.rn.f32x2 " A ", r, m;\n"
/* the exponent becomes a float through the low bits of 1.5 * 2^23: exact, and off the conversion unit; the
 * mantissa is what is left when it is taken off the argument's bits (2^23 times the constant is 0 mod 2^32) */
#define SB_LOG_PAIR(A)                                                                                  \
    "mov.b64 {c0, c1}, " A ";\n add.u32 c2, c0, 0xC0CAFB0D;\n add.u32 c3, c1, 0xC0CAFB0D;\n"             \
    "shr.s32 c2, c2, 23;\n shr.s32 c3, c3, 23;\n add.u32 c2, c2, 0x4B400000;\n add.u32 c3, c3, 0x4B400000;\n mov.b64 n, {c2, c3};\n" \
    "mad.lo.u32 c0, c2, 0xFF800000, c0;\n mad.lo.u32 c1, c3, 0xFF800000, c1;\n mov.b64 r, {c0, c1};\n" \
    "add.rn.f32x2 n, n, k0;\n add.rn.f32x2 r, r, mone;\n fma.rn.f32x2 q, k1, r, k2;\n fma.rn.f32x2 q, q, r, k3;\n fma.rn.f32x2 q, q, r, k4;\n" \
    "fma.rn.f32x2 q, q, r, k5;\n fma.rn.f32x2 q, q, r, k6;\n fma.rn.f32x2 q, q, r, k7;\n fma.rn.f32x2 q, q, r, k8;\n mul.rn.f32x2 z, r, r;\n" \
    "mul.rn.f32x2 t, k9, z;\n mul.rn.f32x2 z, r, z;\n fma.rn.f32x2 t, z, q, t;\n fma.rn.f32x2 t, n, k10, t;\n add.rn.f32x2 r, r, t;\n" \
    "fma.rn.f32x2 " A ", n, k11, r;\n"
/* a / b, correctly rounded: Newton-Raphson from the hardware's reciprocal estimate and two residual
 * corrections (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
 * processor", IBM J. Res. Dev. 34, 1990: with a reciprocal good to half an ulp and the residual
 * a - b q exact, the corrected quotient is the rounded one).  Works on -1/b and -q so that every step is
 * one fused multiply-add; the sign comes from the first product, since the corrections lose that of a
 * zero quotient. */
#define SB_DIV_PAIR(A, B)                                                                               \
    "mov.b64 {f0, f1}, " B ";\n neg.f32 f0, f0;\n neg.f32 f1, f1;\n rcp.approx.ftz.f32 f0, f0;\n rcp.approx.ftz.f32 f1, f1;\n mov.b64 r, {f0, f1};\n" \
    "fma.rn.f32x2 t, " B ", r, k0;\n fma.rn.f32x2 r, r, t, r;\n mul.rn.f32x2 n, " A ", r;\n fma.rn.f32x2 t, " B ", n, " A ";\n"    \
    "fma.rn.f32x2 q, t, r, n;\n fma.rn.f32x2 t, " B ", q, " A ";\n fma.rn.f32x2 q, t, r, q;\n"           \
    "mov.b64 {c0, c1}, q;\n mov.b64 {c2, c3}, n;\n lop3.b32 c0, c0, c2, 0x80000000, 0x72;\n lop3.b32 c1, c1, c3, 0x80000000, 0x72;\n" \
    "mov.b64 " A ", {c0, c1};\n"
/* tanh of anything.  Below 0.9 an odd polynomial (relative error 2^-29.8 before rounding, fitted by weighted
 * least squares), from there on 1 - 2 / (e^2|x| + 1) with the exponential's steps and one Newton step on
 * the reciprocal, |x| cut at 10 where the result is 1; both are computed and one is chosen.  NaN takes the
 * polynomial's side.  At most 1.3 ulp off (all float32 arguments; CUDA's function: 1.8). */
#define SB_TANH_LIST(X) \
    X(0, B9EECA99) X(1, 3B2941E7) X(2, BC0767FD) X(3, 3CB177BC) X(4, BD5CE4F8) X(5, 3E08879A) \
    X(6, BEAAAAA7) X(7, 4038AA3B) X(8, 33257060) X(9, 4B400000) X(10, 3F800000) X(11, 40000000)
#define SB_TANH_PAIR(A)                                                                                 \
    "mov.b64 {c2, c3}, " A ";\n and.b32 c2, c2, 0x7fffffff;\n and.b32 c3, c3, 0x7fffffff;\n mov.b64 m, {c2, c3};\n" \
    "mul.rn.f32x2 z, m, m;\n mov.b32 f0, c2;\n mov.b32 f1, c3;\n min.f32 f0, f0, 0f41200000;\n min.f32 f1, f1, 0f41200000;\n mov.b64 n, {f0, f1};\n" \
    "fma.rn.f32x2 t, n, k7, k9;\n fma.rn.f32x2 q, k0, z, k1;\n fma.rn.f32x2 r, t, mone, k9;\n fma.rn.f32x2 q, q, z, k2;\n" \
    "fma.rn.f32x2 r, n, k7, r;\n fma.rn.f32x2 q, q, z, k3;\n fma.rn.f32x2 r, n, k8, r;\n fma.rn.f32x2 q, q, z, k4;\n" \
    "mov.b64 {f0, f1}, r;\n ex2.approx.ftz.f32 f0, f0;\n ex2.approx.ftz.f32 f1, f1;\n fma.rn.f32x2 q, q, z, k5;\n fma.rn.f32x2 q, q, z, k6;\n" \
    "mov.b64 {c0, c1}, t;\n shl.b32 c0, c0, 23;\n shl.b32 c1, c1, 23;\n mov.b32 c4, f0;\n mov.b32 c5, f1;\n add.u32 c0, c0, c4;\n add.u32 c1, c1, c5;\n" \
    "mov.b64 n, {c0, c1};\n add.rn.f32x2 n, n, k10;\n mov.b64 {f0, f1}, n;\n neg.f32 f0, f0;\n neg.f32 f1, f1;\n" \
    "rcp.approx.ftz.f32 f0, f0;\n rcp.approx.ftz.f32 f1, f1;\n mul.rn.f32x2 z, m, z;\n fma.rn.f32x2 q, z, q, m;\n mov.b64 r, {f0, f1};\n" \
    "fma.rn.f32x2 t, n, r, k10;\n fma.rn.f32x2 r, r, t, r;\n fma.rn.f32x2 r, r, k11, k10;\n"          \
    "mov.b64 {c0, c1}, q;\n mov.b64 {c4, c5}, r;\n mov.b32 f0, c2;\n mov.b32 f1, c3;\n"               \
    "setp.ge.f32 p, f0, 0f3F666666;\n selp.b32 c0, c4, c0, p;\n setp.ge.f32 p, f1, 0f3F666666;\n selp.b32 c1, c5, c1, p;\n" \
    "mov.b64 {c2, c3}, " A ";\n lop3.b32 c0, c0, c2, 0x7fffffff, 0xE4;\n lop3.b32 c1, c1, c3, 0x7fffffff, 0xE4;\n mov.b64 " A ", {c0, c1};\n"
/* |b| within [2^-60, 2^60], |a| too or zero (2|a| - 1 in bits: zero wraps to the top): no step leaves the normal range */
#define SB_LEAST(A) "mov.b64 {c0, c1}, " A ";\n shl.b32 c0, c0, 1;\n shl.b32 c1, c1, 1;\n sub.u32 c0, c0, 1;\n sub.u32 c1, c1, 1;\n min.u32 c2, c2, c0;\n min.u32 c2, c2, c1;\n"
/* no zero among the dividends, the usual case: SB_TOP_NUMBER and SB_LOW_NUMBER over both (top = 0, low = inf before) are enough */
#define SB_DIV_USUAL "setp.le.f32 p, top, 0f5D800000;\n setp.ge.and.f32 p, low, 0f21800000, p;\n vote.sync.all.pred p, p, 0xffffffff;\n"
/* after SB_LEAST over the dividends, SB_TOP_NUMBER over both, SB_LOW_NUMBER over the divisors (c2 = ~0, top = 0, low = inf before) */
#define SB_DIV_RANGE "setp.le.f32 p, top, 0f5D800000;\n setp.ge.and.f32 p, low, 0f21800000, p;\n setp.ge.and.u32 p, c2, 0x42FFFFFF, p;\n"

#endif
