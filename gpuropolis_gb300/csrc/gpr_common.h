/*
 * gpr_common.h -- op codes, op classes and the compiled-program instruction
 * encoding shared by the host library and the kernels.
 *
 * Op codes keep the reference's numbering (enum OPS, main.cu:53) so chain
 * state moves between the reference layout and this library unchanged.
 * Each op's arity, description-length cost (dispatch_length, main.cu:477-526)
 * and node count (dispatch_countnodes, main.cu:553-601) is a property of its
 * class below.
 */
#ifndef GPR_COMMON_H
#define GPR_COMMON_H

#include <stdint.h>

enum gpr_op {
    OP_ONE = 0, OP_CONST, OP_INV, OP_A, OP_B, OP_PLUS, OP_MINUS, OP_RMINUS, OP_CPLUS,
    OP_TIMES, OP_CTIMES, OP_DIV, OP_RDIV, OP_LOG, OP_EXP, OP_POW, OP_CPOW, OP_RPOW,
    OP_CRPOW, OP_SQRT, OP_SIN, OP_ASIN, OP_COS, OP_ACOS, OP_TAN, OP_ATAN, OP_ABS,
    OP_NREF, /* 27 = NOPS of the reference's default op set */
    /* leaves of multivariate data (no reference counterpart): the input
     * variables x1, x2, x3.  A child beyond the heap is x1, as the
     * reference's x (main.cu:374-385). */
    OP_X1 = OP_NREF, OP_X2, OP_X3,
    OP_NALL
};

/* PROGRAM_CODE, main.cu:55: one character per op, used in samples.txt; the
 * variable leaves x1, x2, x3 print as X, Y, Z. */
#define GPR_PROGRAM_CODE "1CIab+-_#*@/|LE^pVPRSsCcTtAXYZ"

enum gpr_opclass {
    CLS_LEAF0 = 0,   /* ONE, CONST: no children                                  */
    CLS_PASS_A,      /* A: value of the left child                               */
    CLS_PASS_B,      /* B: value of the right child                              */
    CLS_UNARY,       /* f(a): length 1+a, count 1+a                              */
    CLS_CUNARY,      /* f(a, C): length CONST_LENGTH_PRIOR+a+1, count a+1        */
    CLS_BINARY,      /* g(a, b): length 1+a+b, count 1+a+b                       */
    CLS_INVALID
};

#if defined(__CUDACC__)
#define GPR_HDI __host__ __device__ __forceinline__
#else
#define GPR_HDI static inline
#endif

/* The class of op o: a 4-bit field per op, eight ops to a 32-bit word, so
 * the lookup is a few integer operations with no branch or jump table. */
#define GPR_CLS_AT(op, cls) ((uint32_t)(cls) << (4 * ((op) & 7)))
#define GPR_CLS_WORD(w)                                                                               \
    ((uint32_t)(GPR_CLS_FIELD((w) * 8 + 0) | GPR_CLS_FIELD((w) * 8 + 1) | GPR_CLS_FIELD((w) * 8 + 2) | \
                GPR_CLS_FIELD((w) * 8 + 3) | GPR_CLS_FIELD((w) * 8 + 4) | GPR_CLS_FIELD((w) * 8 + 5) | \
                GPR_CLS_FIELD((w) * 8 + 6) | GPR_CLS_FIELD((w) * 8 + 7)))
#define GPR_CLS_FIELD(op) GPR_CLS_AT(op, gpr_op_class_slow(op))

#if defined(__CUDACC__)
#define GPR_HDC __host__ __device__ constexpr
#else
#define GPR_HDC static constexpr
#endif

/* The class of op o, written out; only evaluated at compile time, to build
 * the table below. */
GPR_HDC int gpr_op_class_slow(int o) {
    return (o == OP_ONE || o == OP_CONST || o == OP_X1 || o == OP_X2 || o == OP_X3) ? CLS_LEAF0
         : o == OP_A ? CLS_PASS_A
         : o == OP_B ? CLS_PASS_B
         : (o == OP_INV || o == OP_LOG || o == OP_EXP || o == OP_SQRT || o == OP_SIN || o == OP_ASIN ||
            o == OP_COS || o == OP_ACOS || o == OP_TAN || o == OP_ATAN || o == OP_ABS) ? CLS_UNARY
         : (o == OP_CPLUS || o == OP_CTIMES || o == OP_CPOW || o == OP_CRPOW) ? CLS_CUNARY
         : (o == OP_PLUS || o == OP_MINUS || o == OP_RMINUS || o == OP_TIMES || o == OP_DIV || o == OP_RDIV ||
            o == OP_POW || o == OP_RPOW) ? CLS_BINARY
         : CLS_INVALID;
}

GPR_HDI int gpr_op_class(int o) {
    if ((unsigned)o >= 32u) return CLS_INVALID;
    const int w = o >> 3;
    const uint32_t word = w == 0 ? GPR_CLS_WORD(0) : w == 1 ? GPR_CLS_WORD(1) : w == 2 ? GPR_CLS_WORD(2)
                                                                                    : GPR_CLS_WORD(3);
    return (int)((word >> (4 * (o & 7))) & 15u);
}

/* ---- compiled program: a reachable-only postfix form of the heap tree ----
 * One 16-bit word per instruction (gpr_word): bits 0-7 code, bits 8-15 heap
 * node (the constant C[node] an instruction reads).  The evaluator keeps the running
 * value in an accumulator; leaf operands (x1..x3, 1, a constant) are folded into
 * the instruction that consumes them, so the value stack is touched only
 * where both children of a binary node are subtrees. */
typedef uint16_t gpr_word;
/* Codes.  An odd code is a cheap binary op (sum, difference, product): the
 * interpreter runs them all as acc = s acc + b v or acc = acc v, with s and b
 * +1 or -1, so that telling them apart takes no branch but the one between a
 * sum and a product.  Bit 7 of an even code: a quotient or a power; otherwise
 * a load, a push or a unary op. */
#define GPR_CODE_CHEAP 1u      /* sum, difference or product                    */
#define GPR_CODE_ACCNEG 2u     /* cheap: v - acc                                */
#define GPR_CODE_POW 2u        /* long: a power, else a quotient                */
#define GPR_CODE_OPNEG 4u      /* cheap: acc - v                                */
#define GPR_CODE_ACCLEFT 4u    /* long: acc is the left operand                 */
#define GPR_CODE_MUL 8u        /* cheap: a product                              */
#define GPR_CODE_LONG 0x80u    /* even code: quotient or power                  */
#define GPR_CODE_SRC(code) (((code) >> 4) & 7u)
#define GPR_CODE_IS_CONST(code) (((code) & 0x60u) == 0u)   /* binary: operand a constant or 1 */
enum gpr_src { SRC_C = 0, SRC_ONE = 1, SRC_X = 2, SRC_POP = 3, SRC_X2 = 4, SRC_X3 = 5 };
enum gpr_icode {
    I_END = 0,
    I_LDX = 2, I_LDC = 4, I_LD1 = 6, I_PUSH = 8, I_LDNAN = 10, I_LDX2 = 12, I_LDX3 = 14,
    U_INV = 16, U_LOG = 18, U_EXP = 20, U_SQRT = 22, U_SIN = 24, U_ASIN = 26, U_COS = 28, U_ACOS = 30, U_TAN = 32,
    U_ATAN = 34, U_ABS = 36
};
enum gpr_bop { BOP_ADD = 0, BOP_SUB = 1, BOP_MUL = 2, BOP_DIV = 3, BOP_POW = 4 };

#define GPR_BIN(bop, accleft, src)                                                                     \
    (((uint32_t)(src) << 4) |                                                                          \
     ((bop) == BOP_ADD   ? GPR_CODE_CHEAP                                                              \
      : (bop) == BOP_SUB ? (GPR_CODE_CHEAP | ((accleft) ? GPR_CODE_OPNEG : GPR_CODE_ACCNEG))           \
      : (bop) == BOP_MUL ? (GPR_CODE_CHEAP | GPR_CODE_MUL)                                             \
                         : (GPR_CODE_LONG | ((bop) == BOP_POW ? GPR_CODE_POW : 0u) |                   \
                            ((accleft) ? GPR_CODE_ACCLEFT : 0u))))
/* fields of a binary instruction code */
#define GPR_IS_BIN(code) ((code) & (GPR_CODE_CHEAP | GPR_CODE_LONG))
#define GPR_BIN_BOP(code)                                                                              \
    (!((code) & GPR_CODE_CHEAP) ? ((code) & GPR_CODE_POW ? BOP_POW : BOP_DIV)                          \
     : (code) & GPR_CODE_MUL    ? BOP_MUL                                                              \
     : (code) & (GPR_CODE_ACCNEG | GPR_CODE_OPNEG) ? BOP_SUB : BOP_ADD)
#define GPR_BIN_ACCLEFT(code) (((code) >> 2) & 1u)   /* of a difference, quotient or power */

/* Counters the MH kernel accumulates (gpr_get_stats). */
enum gpr_stat {
    GPR_STAT_EVALS = 0,        /* likelihoods scored (one per proposal + one per chain)     */
    GPR_STAT_EVAL_NODES,       /* sum over them of the program's node count                 */
    GPR_STAT_EVAL_POINTS,      /* data points actually evaluated (none for a proposal that
                                * keeps the current values; early exit on invalid)          */
    GPR_STAT_EVAL_NODE_POINTS, /* sum over evaluated points of node count + 4               */
    GPR_STAT_STRUCT_PROPOSED,
    GPR_STAT_STRUCT_ACCEPTED,
    GPR_STAT_CONST_PROPOSED,
    GPR_STAT_CONST_ACCEPTED,
    GPR_NSTATS
};

/* Phases of one chain's block that the instrumented MH kernel times
 * (gpr_debug_phase_profile): clock64 cycles of each warp between phase
 * boundaries, summed over warps.  After the phases, two counts: evaluation
 * passes run, and program instructions interpreted (summed over passes). */
enum gpr_phase {
    GPR_PH_CLAIM = 0,  /* claiming the next chain (group barrier + counter)       */
    GPR_PH_LOAD,       /* chain state in from device memory                        */
    GPR_PH_STEPBAR,    /* step barrier of the free-running / periodic layouts      */
    GPR_PH_STRUCT,     /* structure proposal (main.cu:699-742)                     */
    GPR_PH_CONST,      /* constant proposal (main.cu:743-806)                      */
    GPR_PH_COMPILE,    /* heap tree -> postfix program                             */
    GPR_PH_CAUCHY,     /* Cauchy prior over all constants                          */
    GPR_PH_EPROG,      /* evaluation program (instructions paired with constants)  */
    GPR_PH_BAR1,       /* publishing the program + the first step barrier          */
    GPR_PH_RANK,       /* ranking the CTA's programs by length                     */
    GPR_PH_EVAL,       /* evaluation passes and their reductions                   */
    GPR_PH_BAR2,       /* the second step barrier                                  */
    GPR_PH_COMBINE,    /* combining a chain's pass sums into its likelihood        */
    GPR_PH_ACCEPT,     /* prior, posterior, accept rule, bookkeeping               */
    GPR_PH_STORE,      /* chain state and scores out                               */
    GPR_NPHASES,
    GPR_PH_NPASSES = GPR_NPHASES,   /* count: evaluation passes                    */
    GPR_PH_NINSTR,                  /* count: instructions interpreted             */
    GPR_PH_SLOTS
};

/* Passes (32*K points each) that the lockstep kernel splits a chain's
 * evaluation into, one task each; with K = 8 streamed a task is a range of
 * passes, GPR_TASKS of them per chain at most, and the sums of more than
 * GPR_MAX_PASSES chunks are kept in device memory (KParams::part). */
#define GPR_MAX_PASSES 64
#define GPR_TASKS 16

/* ---- dataset arrays ----
 * Points are kept in chunks of 128, the unit of the likelihood's reduction
 * tree, in which lane l holds points l, l + 32, l + 64 and l + 96.  An array
 * is padded with zeros to whole chunks, and within a chunk lane by lane, so
 * that a lane's four points are one 16-byte load. */
#define GPR_CHUNK_POINTS 128
#define GPR_PAD_POINTS(n) (((n) + GPR_CHUNK_POINTS - 1) / GPR_CHUNK_POINTS * GPR_CHUNK_POINTS)
/* The same for one of many datasets behind each other: of its last chunk only
 * the lanes that have a point, four floats each, so that datasets of a few points
 * take at most four times their size.  A reader of that chunk's other lanes meets
 * the next dataset; after the last one there is a chunk more. */
#define GPR_PACKED_POINTS(n) ((n) / GPR_CHUNK_POINTS * GPR_CHUNK_POINTS + \
                              4 * ((n) % GPR_CHUNK_POINTS < 32 ? (n) % GPR_CHUNK_POINTS : 32))
/* Where point i of a dataset is in its arrays. */
#define GPR_POINT_SLOT(i) (((i) & ~127) | (((i) & 31) << 2) | (((i) >> 5) & 3))

/* Maximum compiled length for a program of PL heap nodes. */
#define GPR_MAX_INSTR(PL) (2 * (PL) + 4)

#endif /* GPR_COMMON_H */
