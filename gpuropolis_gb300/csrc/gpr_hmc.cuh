/*
 * gpr_hmc.cuh -- reverse-mode adjoint of the program evaluator, and the MH
 * kernel whose constant moves are Hamiltonian (HMC; MALA with one leapfrog
 * step) instead of the reference's independence / random-walk proposals.
 *
 * Adjoint.  The compiled postfix program (gpr_common.h) is run forward once
 * per batch of K data points per lane, and the results that the way back needs
 * are kept on a tape: rows of K values per lane in the warp's shared memory
 * (thread-local memory for the rare program that needs more rows than a warp
 * has).  The backward sweep walks the instructions in reverse, carrying
 * d loglik / d acc, splitting it at each binary instruction into the
 * accumulator's and the operand's share, and handing the operand's share to
 * the constant it read (an instruction with a constant operand, or a constant
 * load, reads exactly one heap node's constant).  A popped operand's share
 * takes the place of the pushed value on the tape, until its PUSH.  The value
 * a POP reads is the tape row of its matching PUSH, so the forward sweep needs
 * no value stack.  d loglik / d f at a point is 2 w (y - f) with
 * w = 1/(2 sd^2) (lnormalpdf, main.cu:299-301); sums run per lane in FP32 at
 * the bookkeeping scale 2^-64 and are reduced across lanes per constant, 128
 * points at a time.
 *
 * HMC move (no reference counterpart).  Momentum m ~ N(0, I) over all PL
 * constants; leapfrog with step eps, L steps, on the log-posterior
 * prior + likelihood (main.cu:529-544, 454-468), whose constant part is the
 * Cauchy(0, 1) prior (gradient -2c / (1 + c^2)); accepted with the
 * reference's rule (main.cu:728-740) with forward = -|m0|^2/2 and
 * backward = -|m1|^2/2.  Structure moves are the reference's, every
 * struct_every steps.
 */
#ifndef GPR_HMC_CUH
#define GPR_HMC_CUH

#include "gpr_mh.cuh"

namespace gpr {

/* The kernels come in two widths G: the passes of 128 points (four per lane)
 * that one sweep takes together, its instructions decoded once for all of them.
 * G = 2 has registers for 16 warps per SM, G = 1 for 32.  Which is used: hmc_passes and
 * launch_loglik_grad (gpr_hmc.cu).  Results do not depend on it. */
__host__ __device__ constexpr int hmc_min_ctas(int G) { return G == 1 ? 4 : 2; }   /* of 8 warps, per SM */
#define GPR_GRAD_ROWS 4      /* tape rows in shared memory, of G * 512 bytes per warp */
#define GPR_GRAD_CONSTS 8    /* constants whose shares are reduced together */
#define GPR_GRAD_STRIDE 36   /* floats between their rows of lane shares: conflict-free reads of the reduction */

/* The adjoint's instruction word: code and heap node as in gpr_word; the tape
 * row that keeps the instruction's result (or, for the input variables, that
 * it needs none); and for a binary instruction the row of the value it pops,
 * for one that reads a constant that constant's place among those the program
 * reads.  1 and the invalid-op marker are constants of the nodes below, which
 * no program has (PROGRAM_LENGTH <= 127). */
#define GW_BIN 64u           /* code >= GW_BIN: GW_BIN + bop * 16 + accleft * 8 + source, else as in gpr_icode */
#define GW_CODE(bop, left, src) (GW_BIN + (uint32_t)(bop) * 16u + (uint32_t)(left) * 8u + (uint32_t)(src))
#define GW_BOP(code) (((code) - GW_BIN) >> 4)
#define GW_LEFT(code) (((code) >> 3) & 1u)
#define GW_SRC(code) ((code) & 7u)
#define GW_ROW(w) (((w) >> 16) & 255u)
#define GW_AUX(w) ((w) >> 24)
#define GW_NONE 255u
#define GW_X1 254u           /* the result is x1, x2, x3 */
#define GW_X2 253u
#define GW_X3 252u
#define GW_NODE_ONE 254u
#define GW_NODE_NAN 255u
#define GW_CONSTS 0xffff     /* of grad_prepare's result: the constants the program reads */
#define GW_LONG 0x10000      /* ... whether it has a power, exp, log, root or trigonometric op */

/* Per-warp shared memory of the gradient evaluator and the HMC kernel. */
struct GradSmem {
    uint8_t* ops[2];
    float* Cs[2];       /* [0], [1]: current and proposed constants            */
    gpr_word* prog[2];
    uint32_t* gprog;    /* adjoint instruction words of the program at hand     */
    uint2* eprog;       /* ... paired with the constants they read              */
    uint8_t* cnode;     /* [GPR_GRAD_CONSTS]: nodes of the first constants it reads */
    float* gacc;        /* [PL]: gradient sums of the constants beyond those (lane 0
                         * adds each warp-summed share)                         */
    float* gcur;        /* gradient of the log-posterior at the current state   */
    float* gnew;        /* ... at the trajectory's position                     */
    float* mom;         /* momentum                                             */
    float* rows;        /* the tape: [GPR_GRAD_ROWS][G][32 lanes] of four values */
    /* rows and share together also hold the compiler's scratch (2.5 KB for PL = 127) */
    float* share;       /* [G * GPR_GRAD_CONSTS][GPR_GRAD_STRIDE]: lane shares   */
};

__host__ __device__ __forceinline__ size_t grad_rows_bytes(int PL) { return align16((size_t)PL * 4); }

/* G passes at a time; block: with the buffers that only the MH block has (the
 * proposal's ops, constants and program, the current gradient, the momentum). */
__host__ __device__ __forceinline__ size_t grad_warp_bytes(int PL, int max_instr, int G, bool block) {
    const size_t plp = align16((size_t)PL), n = block ? 2 : 1;
    size_t b = 0;
    b += n * plp;                                              /* ops */
    b += align16(n * plp * 4);                                 /* Cs */
    b += align16(n * (size_t)max_instr * sizeof(gpr_word));    /* prog */
    b += align16((size_t)max_instr * 4);                       /* gprog */
    b += align16((size_t)max_instr * 8);                       /* eprog */
    b += 16;                                                   /* cnode */
    b += grad_rows_bytes(PL);                                  /* gradient sums */
    b += (block ? 3 : 1) * align16(plp * 4);                   /* gnew, gcur, mom */
    b += (size_t)GPR_GRAD_ROWS * G * 512;                      /* rows */
    b += (size_t)G * GPR_GRAD_CONSTS * GPR_GRAD_STRIDE * 4;    /* share */
    return align16(b);
}

__device__ __forceinline__ GradSmem carve_grad(uint8_t* base, int PL, int max_instr, int G, bool block) {
    GradSmem w;
    const size_t plp = align16((size_t)PL), n = block ? 2 : 1;
    uint8_t* p = base;
    w.ops[0] = p; w.ops[1] = block ? p + plp : nullptr; p += n * plp;
    w.Cs[0] = (float*)p; w.Cs[1] = block ? (float*)p + plp : nullptr; p += align16(n * plp * 4);
    w.prog[0] = (gpr_word*)p; w.prog[1] = block ? (gpr_word*)p + max_instr : nullptr;
    p += align16(n * (size_t)max_instr * sizeof(gpr_word));
    w.gprog = (uint32_t*)p; p += align16((size_t)max_instr * 4);
    w.eprog = (uint2*)p; p += align16((size_t)max_instr * 8);
    w.cnode = p; p += 16;
    w.gacc = (float*)p; p += grad_rows_bytes(PL);
    w.gnew = (float*)p; p += align16(plp * 4);
    w.gcur = w.mom = nullptr;
    if (block) {
        w.gcur = (float*)p; p += align16(plp * 4);
        w.mom = (float*)p; p += align16(plp * 4);
    }
    w.rows = (float*)p; p += (size_t)GPR_GRAD_ROWS * G * 512;
    w.share = (float*)p;
    return w;
}

/* An instruction of the adjoint before it has its rows.  A result is kept only
 * if the way back reads it: the factor of a product whose other factor is a
 * constant or popped, an argument or a result where a derivative is written in
 * it, and every pushed value. */
struct GradWord {
    uint32_t code, node;
    bool arg, res;      /* the accumulator before, after is read on the way back */
    bool share;         /* it reads a constant that the program owns              */
};
__device__ __forceinline__ GradWord grad_word(uint32_t ins) {
    GradWord g;
    g.code = ins & 0xffu;
    g.node = (ins >> 8) & 0xffu;
    g.arg = g.res = false;
    if (g.code == I_LD1 || g.code == I_LDNAN) {
        g.node = g.code == I_LD1 ? GW_NODE_ONE : GW_NODE_NAN;
        g.code = I_LDC;
    }
    g.share = g.code == I_LDC && g.node < GW_NODE_ONE;
    if (GPR_IS_BIN(g.code)) {
        const uint32_t bop = GPR_BIN_BOP(g.code), left = GPR_BIN_ACCLEFT(g.code);
        uint32_t src = GPR_CODE_SRC(g.code);
        if (src == SRC_ONE) { src = SRC_C; g.node = GW_NODE_ONE; }
        g.code = GW_CODE(bop, left, src);
        g.share = src == SRC_C && g.node < GW_NODE_ONE;
        const bool takes = src == SRC_POP || g.share;      /* the operand has a share */
        if (bop == BOP_MUL) g.arg = takes;
        else if (bop == BOP_DIV) { g.arg = !left; g.res = !left || takes; }
        else if (bop == BOP_POW) { g.arg = left || takes; g.res = !left || takes; }
    } else if (g.code == I_PUSH) {
        g.res = true;
    } else if (g.code >= U_INV) {
        g.res = g.code == U_INV || g.code == U_EXP || g.code == U_SQRT || g.code == U_TAN;
        g.arg = !g.res;
    }
    return g;
}

/* The adjoint words of a compiled program, into ws.gprog; returns how many
 * constants it reads (GW_CONSTS) and whether it has a long op (GW_LONG).  A lane
 * per instruction: rows and constants are numbered by ballots, and only the
 * pushes and pops are paired one after the other.  As one lane's walk, after
 * every change of structure, it held a warp up for a tenth of a move: 65,536
 * chains of random programs on 30 points, 8 leapfrog steps: 55.1 -> 51.0 ms. */
static __device__ __noinline__ int grad_prepare(const gpr_word* prog, int ninstr, const GradSmem& ws, int lane) {
    const uint32_t below = (1u << lane) - 1u;
    int nconst = 0, rows = 0, sp = 0;
    bool heavy = false;
    uint32_t pending = 0u;       /* lane d: the row of the push pending at depth d (fewer than 32) */
#pragma unroll 1
    for (int base = 0; base < ninstr; base += 32) {
        const int i = base + lane;
        const bool in = i < ninstr;
        /* the last instruction is I_END, which keeps and reads nothing */
        const GradWord g = grad_word(in ? prog[i] : (uint32_t)I_END);
        bool next_arg = __shfl_down_sync(FULLMASK, (int)g.arg, 1) != 0;
        if (lane == 31) next_arg = i + 1 < ninstr && grad_word(prog[i + 1]).arg;
        uint32_t row = g.code == I_LDX ? GW_X1 : g.code == I_LDX2 ? GW_X2 : g.code == I_LDX3 ? GW_X3 : GW_NONE;
        const bool keep = g.res || (next_arg && row == GW_NONE);
        const uint32_t kept = __ballot_sync(FULLMASK, keep), shares = __ballot_sync(FULLMASK, g.share);
        if (keep) row = (uint32_t)(rows + __popc(kept & below));
        rows += __popc(kept);
        uint32_t aux = GW_NONE;
        if (g.share) {
            aux = (uint32_t)(nconst + __popc(shares & below));
            if (aux < GPR_GRAD_CONSTS) ws.cnode[aux] = (uint8_t)g.node;
        }
        nconst += __popc(shares);
        heavy = heavy || (g.code >= GW_BIN ? GW_BOP(g.code) == BOP_POW : g.code > U_INV && g.code < U_ABS);
        const uint32_t push = __ballot_sync(FULLMASK, g.code == I_PUSH);
        uint32_t todo = push | __ballot_sync(FULLMASK, g.code >= GW_BIN && GW_SRC(g.code) == SRC_POP);
#pragma unroll 1
        for (; todo; todo &= todo - 1u) {
            const int b = __ffs(todo) - 1;
            if ((push >> b) & 1u) {
                const uint32_t r = __shfl_sync(FULLMASK, row, b);
                if (lane == sp) pending = r;
                ++sp;
            } else {
                --sp;
                const uint32_t r = __shfl_sync(FULLMASK, pending, sp);
                if (lane == b) aux = r;
            }
        }
        if (in) ws.gprog[i] = g.code | (g.node << 8) | (row << 16) | (aux << 24);
    }
    __syncwarp();
    return nconst | (__any_sync(FULLMASK, heavy) ? GW_LONG : 0);
}

/* The words paired with the constants at hand. */
__device__ __forceinline__ void build_grad_program(const uint32_t* gprog, const float* Cs, int ninstr, uint2* eprog,
                                                   int lane) {
#pragma unroll 1
    for (int i = lane; i < ninstr; i += 32) {
        const uint32_t w = gprog[i], node = (w >> 8) & 0xffu;
        const float c = node == GW_NODE_NAN ? __int_as_float(0x7fc00000) : node == GW_NODE_ONE ? 1.0f : Cs[node];
        eprog[i] = make_uint2(w, __float_as_uint(c));
    }
}

/* One copy each of the long routines, four points at a time. */
static __device__ __noinline__ float4 pow_four(float4 u, float4 w) {
    return make_float4(gx_pow(u.x, w.x), gx_pow(u.y, w.y), gx_pow(u.z, w.z), gx_pow(u.w, w.w));
}
static __device__ __noinline__ float4 log_four(float4 a) {
    return make_float4(gx_log(a.x), gx_log(a.y), gx_log(a.z), gx_log(a.w));
}
/* The derivatives of the trigonometric ops in the argument a (tan: in its
 * result). */
static __device__ __noinline__ float4 trig_slope_four(uint32_t code, float4 a) {
#pragma unroll 1
    for (int n = 0; n < 2; ++n) {
        float2 r;
        switch (code) {
            case U_SIN: r = make_float2(cosf(a.x), cosf(a.y)); break;
            case U_COS: r = make_float2(-sinf(a.x), -sinf(a.y)); break;
            default: {
                const float2 q = make_float2(__fmul_rn(a.x, a.x), __fmul_rn(a.y, a.y));
                if (code == U_ASIN || code == U_ACOS) {
                    r = make_float2(__fdiv_rn(1.0f, __fsqrt_rn(__fsub_rn(1.0f, q.x))),
                                    __fdiv_rn(1.0f, __fsqrt_rn(__fsub_rn(1.0f, q.y))));
                    if (code == U_ACOS) r = make_float2(-r.x, -r.y);
                } else {
                    r = make_float2(__fadd_rn(1.0f, q.x), __fadd_rn(1.0f, q.y));
                    if (code == U_ATAN) r = make_float2(__fdiv_rn(1.0f, r.x), __fdiv_rn(1.0f, r.y));
                }
                break;
            }
        }
        a = make_float4(a.z, a.w, r.x, r.y);
    }
    return a;
}

/* The tape of one lane: GPR_GRAD_ROWS rows in shared memory, the others in
 * thread-local memory. */
template <int K>
struct Tape {
    float4* sm;          /* this lane's first four values of row 0 */
    float4* local;
    __device__ __forceinline__ void put(uint32_t r, const float (&v)[K]) const {
#pragma unroll
        for (int g = 0; g < K / 4; ++g) {
            const float4 q = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            if (r < GPR_GRAD_ROWS) sm[(r * (K / 4) + g) * 32] = q;
            else local[(r - GPR_GRAD_ROWS) * (K / 4) + g] = q;
        }
    }
    __device__ __forceinline__ void get(uint32_t r, float (&v)[K]) const {
#pragma unroll
        for (int g = 0; g < K / 4; ++g) {
            const float4 q = r < GPR_GRAD_ROWS ? sm[(r * (K / 4) + g) * 32] : local[(r - GPR_GRAD_ROWS) * (K / 4) + g];
            v[4 * g] = q.x; v[4 * g + 1] = q.y; v[4 * g + 2] = q.z; v[4 * g + 3] = q.w;
        }
    }
};

/* A result kept in row r, or one of the input variables. */
template <int K, int NV>
__device__ __forceinline__ void result_of(uint32_t r, const float (&x)[NV][K], const Tape<K>& tape, float (&v)[K]) {
    if (r < GW_X3) {
        tape.get(r, v);
    } else {
        const int vi = NV > 1 ? (int)(GW_X1 - r) : 0;
        GPR_EACH v[k] = x[vi][k];
    }
}

/* Value of a binary instruction's operand: an input variable, the constant or
 * the popped value. */
template <int K, int NV>
__device__ __forceinline__ void operand(uint32_t w, float c, const float (&x)[NV][K], const Tape<K>& tape,
                                        float (&v)[K]) {
    const uint32_t src = GW_SRC(w & 0xffu);
    if (src == SRC_C) {
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = c;
    } else if (src == SRC_POP) {
        tape.get(GW_AUX(w), v);
    } else {
        const int vi = NV > 1 && src != SRC_X ? (int)(src - SRC_X2) + 1 : 0;
        GPR_EACH v[k] = x[vi][k];
    }
}

template <int K>
__device__ __forceinline__ void pow_all(const float (&u)[K], const float (&w)[K], float (&r)[K]) {
#pragma unroll
    for (int g = 0; g < K / 4; ++g) {
        const float4 q = pow_four(make_float4(u[4 * g], u[4 * g + 1], u[4 * g + 2], u[4 * g + 3]),
                                  make_float4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]));
        r[4 * g] = q.x; r[4 * g + 1] = q.y; r[4 * g + 2] = q.z; r[4 * g + 3] = q.w;
    }
}
template <int K>
__device__ __forceinline__ void log_all(const float (&a)[K], float (&r)[K]) {
#pragma unroll
    for (int g = 0; g < K / 4; ++g) {
        const float4 q = log_four(make_float4(a[4 * g], a[4 * g + 1], a[4 * g + 2], a[4 * g + 3]));
        r[4 * g] = q.x; r[4 * g + 1] = q.y; r[4 * g + 2] = q.z; r[4 * g + 3] = q.w;
    }
}

template <int K, bool SLOPE>
__device__ __forceinline__ void trig_all(uint32_t code, const float (&a)[K], float (&r)[K]) {
#pragma unroll
    for (int g = 0; g < K / 4; ++g) {
        const float4 u = make_float4(a[4 * g], a[4 * g + 1], a[4 * g + 2], a[4 * g + 3]);
        const float4 q = SLOPE ? trig_slope_four(code, u) : trig_four(code, u);
        r[4 * g] = q.x; r[4 * g + 1] = q.y; r[4 * g + 2] = q.z; r[4 * g + 3] = q.w;
    }
}

/* acc = acc / v, and acc = 1 / acc, with one range check for this lane's K
 * values, where __fdiv_rn checks and branches for each.  65,536 chains of the
 * rational function on 1,024 points, 10 moves of 8 leapfrog steps: 75.9 -> 69.6
 * ms, their gradients 1.14 -> 1.07 ms; 2,048 programs of three variables on
 * 16,384 points the same within the runs.  The interpreter keeps __fdiv_rn,
 * whose code is smaller: with these 131,072 chains of 63 nodes took 208 ms
 * instead of 199, 16,384 chains on 65,536 points 74.7 instead of 65.5. */
template <int K>
__device__ __forceinline__ void divide(float (&acc)[K], float (&v)[K]) {
    if (gx_in_range(acc) && gx_in_range(v)) {
        GPR_EACH acc[k] = gx_quotient(acc[k], v[k], gx_recip(v[k]));
    } else {
        in_turn<K, 1>(acc, v, [](float a, float b) { return __fdiv_rn(a, b); });
    }
}
template <int K>
__device__ __forceinline__ void invert(float (&acc)[K]) {
    if (gx_in_range(acc)) {
        GPR_EACH acc[k] = gx_recip(acc[k]);
    } else {
        float v[K];
        GPR_EACH v[k] = 0.0f;
        in_turn<K, 1>(acc, v, [](float a, float) { return __fdiv_rn(1.0f, a); });
    }
}

/* acc = f(x) for this lane's K points, the results that the way back needs
 * kept on the tape.  The arithmetic is the evaluator's (run_program),
 * operation for operation. */
template <int K, int NV>
__device__ __forceinline__ void forward_tape(const uint2* __restrict__ prog, int ninstr, const float (&x)[NV][K],
                                             const Tape<K>& tape, float (&acc)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = 0.0f;
    uint2 nxt = prog[0];
#pragma unroll 1
    for (int i = 0; i < ninstr - 1; ++i) {
        const uint32_t w = nxt.x, code = w & 0xffu;
        const float c = __uint_as_float(nxt.y);
        nxt = prog[i + 1];
        if (code >= GW_BIN) {
            const uint32_t bop = GW_BOP(code), src = GW_SRC(code);
            const bool left = GW_LEFT(code);
            if (bop <= BOP_MUL && src == SRC_C) {
                if (bop == BOP_ADD) { GPR_EACH acc[k] = __fadd_rn(acc[k], c); }
                else if (bop == BOP_MUL) { GPR_EACH acc[k] = __fmul_rn(acc[k], c); }
                else if (left) { GPR_EACH acc[k] = __fsub_rn(acc[k], c); }
                else { GPR_EACH acc[k] = __fsub_rn(c, acc[k]); }
            } else if (bop <= BOP_MUL && src == SRC_X) {
                if (bop == BOP_ADD) { GPR_EACH acc[k] = __fadd_rn(acc[k], x[0][k]); }
                else if (bop == BOP_MUL) { GPR_EACH acc[k] = __fmul_rn(acc[k], x[0][k]); }
                else if (left) { GPR_EACH acc[k] = __fsub_rn(acc[k], x[0][k]); }
                else { GPR_EACH acc[k] = __fsub_rn(x[0][k], acc[k]); }
            } else {
                float v[K];
                operand<K, NV>(w, c, x, tape, v);
                if (bop == BOP_ADD) { GPR_EACH acc[k] = __fadd_rn(acc[k], v[k]); }
                else if (bop == BOP_MUL) { GPR_EACH acc[k] = __fmul_rn(acc[k], v[k]); }
                else {
                    if (!left) { GPR_EACH { const float t = acc[k]; acc[k] = v[k]; v[k] = t; } }
                    if (bop == BOP_SUB) { GPR_EACH acc[k] = __fsub_rn(acc[k], v[k]); }
                    else if (bop == BOP_DIV) divide<K>(acc, v);
                    else pow_all<K>(acc, v, acc);
                }
            }
        } else if (code >= U_INV) {
            if (code == U_EXP) {
#pragma unroll
                for (int k = 0; k < K; ++k) acc[k] = gx_exp(acc[k]);
            } else if (code == U_LOG) {
                log_all<K>(acc, acc);
            } else if (code == U_INV) {
                invert<K>(acc);
            } else if (code == U_SQRT) {
#pragma unroll
                for (int k = 0; k < K; ++k) acc[k] = __fsqrt_rn(acc[k]);
            } else if (code == U_ABS) {
#pragma unroll
                for (int k = 0; k < K; ++k) acc[k] = fabsf(acc[k]);
            } else {
                trig_all<K, false>(code, acc, acc);
            }
        } else if (code == I_LDC) {
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] = c;
        } else if (code != I_PUSH) {
            const int vi = NV > 1 && code != I_LDX ? (code == I_LDX2 ? 1 : 2) : 0;
            GPR_EACH acc[k] = x[vi][k];
        }
        const uint32_t row = GW_ROW(w);
        if (row < GW_X3) tape.put(row, acc);
    }
}

/* adj * d, where a zero adjoint contributes zero even through a partial that
 * left the FP32 range (0 * inf would poison the sums). */
__device__ __forceinline__ float adj_mul(float adj, float d) {
    float r = adj;
    if (adj != 0.0f) r = __fmul_rn(adj, d);
    return r;
}

/* This lane's share of constant number j: the sum over each pass's four
 * points.  The first GPR_GRAD_CONSTS constants leave it for reduce_shares; the
 * others are summed over the warp at once. */
template <int K>
__device__ __forceinline__ void give_share(const float (&av)[K], uint32_t w, const GradSmem& ws, int lane) {
    const uint32_t j = GW_AUX(w);
    if (j == GW_NONE) return;
    float s[K / 4];
#pragma unroll
    for (int g = 0; g < K / 4; ++g)
        s[g] = __fadd_rn(__fadd_rn(__fadd_rn(av[4 * g], av[4 * g + 1]), av[4 * g + 2]), av[4 * g + 3]);
    if (j < GPR_GRAD_CONSTS) {
        float* q = ws.share + (int)j * GPR_GRAD_STRIDE + lane;
#pragma unroll
        for (int g = 0; g < K / 4; ++g) q[g * GPR_GRAD_CONSTS * GPR_GRAD_STRIDE] = s[g];
    } else {
#pragma unroll
        for (int g = 0; g < K / 4; ++g) {
            const float tot = warp_sum(s[g]);
            if (lane == 0) ws.gacc[(w >> 8) & 0xffu] += tot;
        }
    }
}

/* du = 1 / v, dw = -res / v for arguments out of the fast quotient's range. */
template <int K>
__device__ __forceinline__ void general_slopes(const float (&res)[K], const float (&v)[K], float (&du)[K],
                                               float (&dw)[K], bool w_too) {
    float b[K], t[K];
    GPR_EACH { b[k] = v[k]; du[k] = 1.0f; }
    in_turn<K, 1>(du, b, [](float a, float c) { return __fdiv_rn(a, c); });
    if (!w_too) return;
    GPR_EACH { b[k] = v[k]; t[k] = res[k]; }
    in_turn<K, 1>(t, b, [](float a, float c) { return __fdiv_rn(a, c); });
    GPR_EACH dw[k] = -t[k];
}

/* The backward sweep: adj holds d loglik / d f per point on entry. */
template <int K, int NV>
__device__ __forceinline__ void backward_tape(const uint2* __restrict__ prog, int ninstr, const float (&x)[NV][K],
                                              const Tape<K>& tape, float (&adj)[K], const GradSmem& ws, int lane) {
    uint2 nxt = prog[ninstr - 2];
#pragma unroll 1
    for (int i = ninstr - 2; i >= 0; --i) {
        const uint32_t w = nxt.x, code = w & 0xffu;
        const float c = __uint_as_float(nxt.y);
        nxt = prog[i > 0 ? i - 1 : 0];
        const uint32_t arg = GW_ROW(nxt.x);       /* where the accumulator before this instruction is */
        if (code >= GW_BIN) {
            const uint32_t bop = GW_BOP(code), src = GW_SRC(code);
            const bool left = GW_LEFT(code);
            if (bop == BOP_ADD) {
                if (src == SRC_C) give_share<K>(adj, w, ws, lane);
                else if (src == SRC_POP) tape.put(GW_AUX(w), adj);   /* the pushed value is done with */
                continue;
            }
            if (bop == BOP_MUL && src == SRC_X) {
                GPR_EACH adj[k] = adj_mul(adj[k], x[0][k]);
                continue;
            }
            if (bop == BOP_MUL && src == SRC_C) {
                if (arg != GW_NONE && GW_AUX(w) != GW_NONE) {
                    float a[K];
                    result_of<K, NV>(arg, x, tape, a);
                    GPR_EACH a[k] = adj_mul(adj[k], a[k]);
                    give_share<K>(a, w, ws, lane);
                }
                GPR_EACH adj[k] = adj_mul(adj[k], c);
                continue;
            }
            const bool takes = GW_AUX(w) != GW_NONE;   /* the operand has a share: popped, or a constant of the program */
            float av[K];          /* the operand's share per point */
            if (bop == BOP_SUB) {
                GPR_EACH av[k] = -adj[k];
                if (!left) { GPR_EACH { const float t = av[k]; av[k] = adj[k]; adj[k] = t; } }
            } else {
                float v[K];
                operand<K, NV>(w, c, x, tape, v);
                if (bop == BOP_MUL) {
                    if (takes && arg != GW_NONE) {
                        result_of<K, NV>(arg, x, tape, av);
                        GPR_EACH av[k] = adj_mul(adj[k], av[k]);
                    }
                    GPR_EACH adj[k] = adj_mul(adj[k], v[k]);
                } else {
                    float a[K], res[K];
                    if (arg != GW_NONE) result_of<K, NV>(arg, x, tape, a);
                    if (GW_ROW(w) < GW_X3) tape.get(GW_ROW(w), res);
                    if (bop == BOP_DIV) {
                        /* u / w: du = 1 / w, dw = -res / w, from one reciprocal */
                        if (!left) { GPR_EACH v[k] = a[k]; }
                        float du[K], dw[K];
                        const bool w_too = !left || takes;
                        if (gx_in_range(v) && (!w_too || gx_in_range(res))) {
                            GPR_EACH du[k] = gx_recip(v[k]);
                            if (w_too) { GPR_EACH dw[k] = -gx_quotient(res[k], v[k], du[k]); }
                        } else {
                            general_slopes<K>(res, v, du, dw, w_too);
                        }
                        if (left) {
                            GPR_EACH { av[k] = adj_mul(adj[k], dw[k]); adj[k] = adj_mul(adj[k], du[k]); }
                        } else {
                            GPR_EACH { av[k] = adj_mul(adj[k], du[k]); adj[k] = adj_mul(adj[k], dw[k]); }
                        }
                    } else {
                        /* u^w: du = w u^(w - 1), dw = u^w log u */
                        if (!left) { GPR_EACH { const float t = a[k]; a[k] = v[k]; v[k] = t; } }
                        float du[K], dw[K];
                        if (left || takes) {
                            float e[K];
                            GPR_EACH e[k] = __fsub_rn(v[k], 1.0f);
                            pow_all<K>(a, e, du);
                            GPR_EACH du[k] = __fmul_rn(v[k], du[k]);
                        }
                        if (!left || takes) {
                            log_all<K>(a, dw);
                            GPR_EACH dw[k] = res[k] == 0.0f ? 0.0f : __fmul_rn(res[k], dw[k]);
                        }
                        if (left) {
                            GPR_EACH { av[k] = adj_mul(adj[k], dw[k]); adj[k] = adj_mul(adj[k], du[k]); }
                        } else {
                            GPR_EACH { av[k] = adj_mul(adj[k], du[k]); adj[k] = adj_mul(adj[k], dw[k]); }
                        }
                    }
                }
            }
            if (src == SRC_POP) tape.put(GW_AUX(w), av);
            else if (src == SRC_C) give_share<K>(av, w, ws, lane);
        } else if (code == I_PUSH) {
            tape.get(GW_ROW(w), adj);
        } else if (code >= U_INV) {
            float a[K], res[K];
            if (arg != GW_NONE) result_of<K, NV>(arg, x, tape, a);
            if (GW_ROW(w) < GW_X3) tape.get(GW_ROW(w), res);
            if (code == U_EXP) { GPR_EACH adj[k] = adj_mul(adj[k], res[k]); }
            else if (code == U_INV) { GPR_EACH adj[k] = adj_mul(adj[k], -__fmul_rn(res[k], res[k])); }
            else if (code == U_LOG) { GPR_EACH adj[k] = adj_mul(adj[k], __fdiv_rn(1.0f, a[k])); }
            else if (code == U_SQRT) { GPR_EACH adj[k] = adj_mul(adj[k], __fdiv_rn(0.5f, res[k])); }
            else if (code == U_ABS) {
                GPR_EACH adj[k] = adj_mul(adj[k], a[k] > 0.0f ? 1.0f : (a[k] < 0.0f ? -1.0f : 0.0f));
            } else {
                if (code == U_TAN) { GPR_EACH a[k] = res[k]; }
                trig_all<K, true>(code, a, a);
                GPR_EACH adj[k] = adj_mul(adj[k], a[k]);
            }
        } else if (code == I_LDC) {
            give_share<K>(adj, w, ws, lane);
        }
    }
}

/* The lane shares of pass group g summed over the warp, constant j in the
 * four lanes 4j .. 4j + 3: the tree of an xor butterfly (distances 16, 8, 4,
 * 2, 1) for all constants at once, where one butterfly after the other takes
 * ten instructions each. */
__device__ __forceinline__ float reduce_shares(const float* share, int g, int lane) {
    const float* p = share + (g * GPR_GRAD_CONSTS + (lane >> 2)) * GPR_GRAD_STRIDE + (lane & 3);
    const float t0 = __fadd_rn(p[0], p[16]), t1 = __fadd_rn(p[4], p[20]);
    const float t2 = __fadd_rn(p[8], p[24]), t3 = __fadd_rn(p[12], p[28]);
    float v = __fadd_rn(__fadd_rn(t0, t2), __fadd_rn(t1, t3));
    v = __fadd_rn(v, __shfl_xor_sync(FULLMASK, v, 2));
    return __fadd_rn(v, __shfl_xor_sync(FULLMASK, v, 1));
}

/* What the sweeps of a program leave. */
struct GradSums {
    float s, mine;       /* this lane's share of S; lanes 4j..4j+3: the sum of constant j */
    int pts;
    bool bad;
};

/* Passes [pass, end) of a program, G at a time (the last of them may be without
 * a point). */
template <int G, int NV, bool STREAM>
__device__ __forceinline__ void grad_passes_of(const uint2* prog, int ninstr, int nconst, float4* local_rows,
                                               const GradSmem& ws, const DataView& dv, float w_to_df, int lane,
                                               int pass, int end, GradSums& sum) {
    constexpr int K = 4 * G;
    Tape<K> tape;
    tape.sm = (float4*)ws.rows + lane;
    tape.local = local_rows;
#pragma unroll 1
    for (; pass < end && !sum.bad; pass += G) {
        float x[NV][K], adj[K];
        load_points<K, NV, STREAM>(dv, pass, lane, x);
        forward_tape<K, NV>(prog, ninstr, x, tape, adj);
        int good = 0;              /* passes before the first with an invalid point */
#pragma unroll
        for (int gi = 0; gi < G; ++gi) {
            const int left = dv.nd - (pass + gi) * GPR_CHUNK_POINTS;
            if (sum.bad || (gi > 0 && left <= 0)) {
#pragma unroll
                for (int k = 4 * gi; k < 4 * gi + 4; ++k) adj[k] = 0.0f;
                continue;
            }
            const float4 y4 = data_at<STREAM>(dv, DA_Y, pass + gi, lane), w4 = data_at<STREAM>(dv, DA_W, pass + gi, lane);
            const float y[4] = {y4.x, y4.y, y4.z, y4.w}, w[4] = {w4.x, w4.y, w4.z, w4.w};
            bool b = false;
            auto term = [&](int kk) {
                /* the 2^-64-scaled weight: dw carries 2^-e; the factor 2^(e-64) is exact */
                const float wi = __fmul_rn(w[kk], w_to_df);
                const float r = __fsub_rn(adj[4 * gi + kk], y[kk]);
                const float q = __fmul_rn(r, r);
                b |= !(q <= FLT_MAX);
                sum.s = fmaf(q, wi, sum.s);
                adj[4 * gi + kk] = __fmul_rn(__fmul_rn(-2.0f, wi), r);
            };
            if (left >= GPR_CHUNK_POINTS) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) term(kk);
            } else {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    if (lane + 32 * kk < left) term(kk);
                    else adj[4 * gi + kk] = 0.0f;
                }
            }
            sum.pts += min(GPR_CHUNK_POINTS, left);
            sum.bad = __any_sync(FULLMASK, b);
            if (sum.bad) {
#pragma unroll
                for (int k = 4 * gi; k < 4 * gi + 4; ++k) adj[k] = 0.0f;
            } else {
                good = gi + 1;
            }
        }
        if (good > 0) {
            backward_tape<K, NV>(prog, ninstr, x, tape, adj, ws, lane);
            if (nconst > 0) {
                __syncwarp();
#pragma unroll
                for (int gi = 0; gi < G; ++gi) sum.mine = __fadd_rn(sum.mine, reduce_shares(ws.share, gi, lane));
                __syncwarp();
            }
        }
    }
}

/* Log-likelihood of one program (double-float at scale 2^-64, -inf when any
 * point is invalid, as eval_loglik) and its gradient over all PL constants:
 * g[i] = 2^-64 d loglik / d C[i] in FP32, at the bookkeeping scale like the
 * likelihood (0 for constants the program does not read).  The gradient is
 * meaningful only when the likelihood is finite.  info: of grad_prepare.
 *
 * Bound by issued instructions, most of them the interpreter's, and by their
 * latency: hence only the rows that are read again are kept, and in shared
 * memory (a row for every instruction in thread-local memory made 8 GB of
 * DRAM writes per 44 ms), an instruction is decoded once for G passes, sums
 * and products with a constant or x take their operand where it is, and the
 * constants' shares are reduced together.  65,536 chains of the rational model,
 * 1,024 points, 10 moves of 8 leapfrog steps: 146 -> 66 ms; their gradients
 * 2.16 -> 0.98 ms, with the copy to the host.  In mixed populations the warps wait
 * for instructions (22 of 30 cycles between issues: 8,192 chains with structure
 * moves on 128 points). */
template <int MAXR, int G, int NV, bool STREAM>
__device__ __forceinline__ df eval_loglik_grad(const uint2* prog, int ninstr, int info, const GradSmem& ws,
                                               const DataView& dv, const KParams& p, int lane, int& pts_out, float* g) {
    const int PL = p.PL, nconst = info & GW_CONSTS;
    float4 local_rows[MAXR * G];   /* rows beyond the warp's: a program of PL nodes keeps at most 3 PL / 2 */
#pragma unroll 1
    for (int j = lane; j < PL; j += 32) ws.gacc[j] = 0.0f;
    __syncwarp();
    GradSums sum = {0.0f, 0.0f, 0, false};
    const int npass = (dv.nd + 127) / 128;
    int pass = 0;
    if constexpr (G > 1) {
        /* A single pass is swept alone.  An odd last one is not: it would save
         * half a sweep, but bring the code of another into the instruction cache
         * (6,000 chains of random programs, 1,100 points of one variable, 8
         * leapfrog steps: 19.5 ms alone, 17.1 in a pair; fixed programs 4.4 and
         * 4.3 ms). */
        pass = npass > 1 ? npass : 0;
        grad_passes_of<G, NV, STREAM>(prog, ninstr, nconst, local_rows, ws, dv, p.w_to_df, lane, 0, pass, sum);
    }
    grad_passes_of<1, NV, STREAM>(prog, ninstr, nconst, local_rows, ws, dv, p.w_to_df, lane, pass, npass, sum);
    __syncwarp();
#pragma unroll 1
    for (int c = lane; c < PL; c += 32) g[c] = ws.gacc[c];
    __syncwarp();
    if ((lane & 3) == 0 && (lane >> 2) < nconst) g[ws.cnode[lane >> 2]] = sum.mine;
    __syncwarp();
    pts_out = sum.pts;
    if (sum.bad) return df_make(-INFINITY, 0.0f);
    df S = warp_sum_df(df_make(sum.s, 0.0f));
    if (!isfinite(S.hi)) return df_make(-INFINITY, 0.0f);
    return df_sub(df_neg(S), df_make(dv.ns_hi, dv.ns_lo));
}

/* d/dc of lcauchypdf(c, 1) (main.cu:303-305). */
__device__ __forceinline__ float dcauchy(float c) {
    return __fdiv_rn(__fmul_rn(-2.0f, c), __fadd_rn(1.0f, __fmul_rn(c, c)));
}

/* Standard normal momentum for constant i at MH step t of a chain: Philox
 * keyed by (seed ^ 0x484d43, chain), counter (t, i), Box-Muller on two
 * 24-bit uniforms with the project's exactly reproducible log and sin
 * (gpr_rngmath.h), so a host restatement draws the same values. */
__device__ __forceinline__ float hmc_momentum(uint32_t seed, uint32_t chain, uint32_t t, uint32_t i) {
    uint32_t c[4] = {t, i, 0x4d4f4du, 0u};
    gpr_philox4x32_10(c, seed ^ 0x484d43u, chain);
    const float u1 = __fmul_rn((float)((c[0] >> 8) + 1u), 5.9604644775390625e-08f);   /* (0, 1] */
    const float u2 = __fmul_rn((float)(c[1] >> 8), 5.9604644775390625e-08f);          /* [0, 1) */
    const float a = __fsqrt_rn(__fmul_rn(-2.0f, gpr_rng_logf(u1)));
    return __fmul_rn(a, gpr_rng_sinf(gpr_rng_twopi_times(u2)));
}

/* Two uniforms in [0, 1) for move t of a chain's trajectory jitter, from the
 * momentum's Philox stream at a counter the momenta never use. */
__device__ __forceinline__ void hmc_jitter_uniforms(uint32_t seed, uint32_t chain, uint32_t t, float& u1, float& u2) {
    uint32_t c[4] = {t, 0xffffffffu, 0x4a4954u, 0u};
    gpr_philox4x32_10(c, seed ^ 0x484d43u, chain);
    u1 = __fmul_rn((float)(c[0] >> 8), 5.9604644775390625e-08f);
    u2 = __fmul_rn((float)(c[1] >> 8), 5.9604644775390625e-08f);
}

/* The dataset: staged into this CTA's shared memory, or (STREAM) read from
 * device memory.  Returns where the per-warp regions start, or nullptr (the
 * same in every thread) when the staging copy timed out. */
template <bool STREAM>
__device__ __forceinline__ uint8_t* grad_dataset(uint8_t* smem, const KParams& p, DataView& dv) {
    float* fx = (float*)(smem + GPR_STAGED_OFFSET);
    dv = data_view(p, fx, STREAM);
    if (STREAM) return smem + GPR_STAGED_OFFSET;
    if (!stage_dataset(fx, (uint64_t*)smem, p, dv)) return nullptr;
    return smem + GPR_STAGED_OFFSET + align16((size_t)data_arrays(p) * p.nd_pad * 4);
}

/* ------------------------------------------------------------------------ */
/* d loglik / d C for every chain's current state (gpr_loglik_grad): one warp
 * per chain, grad[i*N + chain] (double, unscaled) and lik[chain].  A chain reads
 * every point once, so the data are read from device memory.  later (may be
 * null): a list of chains, its length first; the kernel with G = 2 leaves the
 * programs with a long op there, the one with G = 1 takes the listed ones. */
template <int MAXR, int G, int NV>
__global__ void __launch_bounds__(128, 2 * hmc_min_ctas(G)) loglik_grad_kernel(const __grid_constant__ KParams p,
                                                                              double* grad, double* lik_out,
                                                                              int* later) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    int chain = blockIdx.x * (blockDim.x >> 5) + warp;
    if (G == 1 && later) {
        if (chain >= later[0]) return;
        chain = later[1 + chain];
    }
    if (chain >= p.N) return;
    const GradSmem ws = carve_grad(smem + (size_t)warp * grad_warp_bytes(p.PL, p.max_instr, G, false), p.PL,
                                   p.max_instr, G, false);
    const DataView dv = data_view(p, nullptr, true, p.nds > 0 ? chain_dataset(p, chain) : -1);
    const int PL = p.PL;
    for (int i = lane; i < PL; i += 32) {
        const int o = p.P[(size_t)i * p.N + chain];
        ws.ops[0][i] = (uint8_t)((o >= 0 && o < OP_NALL) ? o : 255);
        ws.Cs[0][i] = p.C[(size_t)i * p.N + chain];
    }
    __syncwarp();
    const CompileOut co = compile_parallel<NV>(ws.ops[0], PL, ws.prog[0], compile_scratch(ws.rows, PL), lane);
    __syncwarp();
    const int info = grad_prepare(ws.prog[0], co.ninstr, ws, lane);
    if (G > 1 && later && (info & GW_LONG)) {
        if (lane == 0) later[1 + atomicAdd(later, 1)] = chain;
        return;
    }
    build_grad_program(ws.gprog, ws.Cs[0], co.ninstr, ws.eprog, lane);
    __syncwarp();
    int pts = 0;
    const df lik = eval_loglik_grad<MAXR, G, NV, true>(ws.eprog, co.ninstr, info, ws, dv, p, lane, pts, ws.gnew);
    for (int i = lane; i < PL; i += 32) grad[(size_t)i * p.N + chain] = (double)ws.gnew[i] * GPR_DF_UNSCALE;
    if (lane == 0) lik_out[chain] = df_to_double_unscaled(lik);
}

/* The compiler out of line: it runs at a structure move, and inlined it takes
 * registers from the leapfrog loop (rational model 82 -> 75 ms, 16,384 points
 * of three variables 79 -> 76 ms). */
template <int NV>
static __device__ __noinline__ CompileOut compile_apart(const uint8_t* ops, int PL, gpr_word* prog,
                                                        const CompileScratch& cs, int lane) {
    return compile_parallel<NV>(ops, PL, prog, cs, lane);
}

/* The gradient out of line, called from two places.  (The gradient kernel,
 * with one, has it inline: the call's arguments go through local memory.) */
template <int MAXR, int G, int NV, bool STREAM>
static __device__ __noinline__ df eval_apart(const uint2* prog, int ninstr, int info, const GradSmem ws,
                                             const DataView dv, const KParams& p, int lane, int& pts, float* g) {
    return eval_loglik_grad<MAXR, G, NV, STREAM>(prog, ninstr, info, ws, dv, p, lane, pts, g);
}

/* ------------------------------------------------------------------------ */
/* The MH block with Hamiltonian constant moves.  One warp per chain, chains
 * claimed from the global counter; evaluation with the adjoint on 4 G points
 * per lane. */
template <int MAXR, int G, int RNG, bool STREAM, int NV>
__global__ void __launch_bounds__(256, hmc_min_ctas(G)) mh_hmc_kernel(const __grid_constant__ KParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    DataView dv;
    uint8_t* wbase = grad_dataset<STREAM>(smem, p, dv);
    if (!wbase) return;   /* the staging copy timed out: the error flag is set */
    const GradSmem ws = carve_grad(wbase + (size_t)warp * grad_warp_bytes(p.PL, p.max_instr, G, true), p.PL,
                                   p.max_instr, G, true);
    const int PL = p.PL;
    const bool adapt = p.chain_scale && p.adapt_target > 0.0f;
    const uint32_t seed = p.seed;
    const float unscale = (float)GPR_DF_UNSCALE;
    const LaneJump ljump = make_lane_jump(p, lane);

#pragma unroll 1
    for (;;) {
        int chain = 0;
        if (lane == 0) chain = atomicAdd(p.next_chain, 1);
        chain = __shfl_sync(FULLMASK, chain, 0);
        if (chain >= p.N) break;
        if (STREAM && p.nds > 0) dv = data_view(p, nullptr, true, chain_dataset(p, chain));   /* batched: streamed */

        for (int i = lane; i < PL; i += 32) {
            const int o = p.P[(size_t)i * p.N + chain];
            ws.ops[0][i] = (uint8_t)((o >= 0 && o < OP_NALL) ? o : 255);
            ws.Cs[0][i] = p.C[(size_t)i * p.N + chain];
        }
        __syncwarp();

        Rng r;
        r.key0 = seed; r.key1 = (uint32_t)chain; r.blk = 0xffffffffu; r.drawn = 0;
        r.w0 = r.w1 = r.w2 = r.w3 = 0u;
        r.s = (RNG == 0) ? ((seed + (uint32_t)chain) & 0x7fffffffu) : 0u;

        /* leapfrog step: the configured one or this chain's own; with
         * adaptation, dual averaging of log(step) toward the target acceptance
         * (Hoffman and Gelman, JMLR 2014, section 3.2: gamma 0.05, t0 10,
         * kappa 0.75, mu = log(10 step0)) */
        const float eps0 = p.chain_scale ? p.chain_scale[chain] : p.hmc_eps;
        float log_eps = logf(eps0), log_eps_bar = log_eps, hbar = 0.0f;
        const float mu = logf(__fmul_rn(10.0f, eps0));
        int n_adapt = 0;

        int cur = 0, gcur = 0, ccur = 0, cur_count = 0, cur_ninstr = 0;   /* ops, program, constants buffers */
        int nconst = 0, prepared = -1;   /* of the program whose adjoint words ws.gprog holds, and its buffer */
        float cur_len = 0.0f;
        df cur_prior = df_make(0.f, 0.f), cur_lik = df_make(0.f, 0.f), cur_post = df_make(0.f, 0.f);
        df cur_cs = df_make(0.f, 0.f);
        unsigned long long st_nodes = 0, st_np = 0, st_pts = 0;
        int st_evals = 0, st_sp = 0, st_sa = 0, st_cp = 0, st_ca = 0;

#pragma unroll 1
        for (int step = -1; step < p.steps; ++step) {
            const bool init = step < 0;
            const bool structural = init || (p.struct_every > 0 && step % p.struct_every == 0);
            if (structural) {
                /* the reference's structure move (or the initial evaluation) */
                int pbuf = cur, gbuf = gcur;
                df forward = df_make(0.f, 0.f);
                bool changed = true;   /* the proposal's program is not the current one (mh_block_kernel) */
                if (!init) {
                    forward = df_make(__fmul_rn(-p.logcount[cur_count], GPR_DF_SCALE), 0.0f);
                    changed = structure_move<RNG>(r, ws.ops[cur], ws.ops[cur ^ 1], df_invalid(cur_post), p, ljump, lane);
                    pbuf = cur ^ 1;
                    if (changed) gbuf = gcur ^ 1;
                }
                __syncwarp();
                CompileOut co;
                co.ninstr = cur_ninstr; co.length = cur_len; co.count = cur_count;
                const df cs = init ? cauchy_sum(ws.Cs[ccur], p, lane) : cur_cs;
                df lik = cur_lik;
                int pe = 0;
                if (changed) {
                    co = compile_apart<NV>(ws.ops[pbuf], PL, ws.prog[gbuf], compile_scratch(ws.rows, PL), lane);
                    __syncwarp();
                    nconst = grad_prepare(ws.prog[gbuf], co.ninstr, ws, lane);
                    prepared = gbuf;
                    build_grad_program(ws.gprog, ws.Cs[ccur], co.ninstr, ws.eprog, lane);
                    __syncwarp();
                    lik = eval_apart<MAXR, G, NV, STREAM>(ws.eprog, co.ninstr, nconst, ws, dv, p, lane, pe, ws.gnew);
                }
                const df backward = df_make(__fmul_rn(-p.logcount[co.count], GPR_DF_SCALE), 0.0f);
                st_pts += (unsigned)pe;
                const df prior = df_add(length_prior(co.length, p), cs);
                const df post = df_add(prior, lik);
                st_evals++; st_nodes += (unsigned)co.count; st_np += (unsigned long long)(co.count + 4) * pe;
                bool accept = true;
                if (!init) {
                    accept = mh_accept<RNG>(post, cur_post, backward, forward, r, p);
                    st_sp++; st_sa += accept;
                }
                if (accept) {
                    cur = pbuf; gcur = gbuf; cur_len = co.length; cur_count = co.count; cur_ninstr = co.ninstr; cur_cs = cs;
                    cur_prior = prior; cur_lik = lik; cur_post = post;
                    if (changed)
                        for (int i = lane; i < PL; i += 32)
                            ws.gcur[i] = __fadd_rn(__fmul_rn(ws.gnew[i], unscale), dcauchy(ws.Cs[ccur][i]));
                }
                __syncwarp();
            } else {
                /* ---- Hamiltonian constant move ---- */
                st_cp++;
                if (!df_invalid(cur_post)) {
                    float eps = expf(log_eps);
                    int nleap = p.hmc_L;
                    if (p.hmc_jit_eps > 0.0f || p.hmc_jit_len > 0.0f) {
                        /* this move's trajectory: jittered step and leapfrog count */
                        float ue, ul;
                        hmc_jitter_uniforms(seed, (uint32_t)chain, (uint32_t)step, ue, ul);
                        eps = __fmul_rn(eps, __fadd_rn(1.0f, __fmul_rn(p.hmc_jit_eps, __fsub_rn(__fmul_rn(2.0f, ue), 1.0f))));
                        if (p.hmc_jit_len > 0.0f) {
                            const float L = (float)p.hmc_L;
                            const int lo = max(1, __float2int_rn(__fmul_rn(L, __fsub_rn(1.0f, p.hmc_jit_len))));
                            const int hi = max(lo, __float2int_rn(__fmul_rn(L, __fadd_rn(1.0f, p.hmc_jit_len))));
                            nleap = lo + min((int)__fmul_rn(ul, (float)(hi - lo + 1)), hi - lo);
                        }
                    }
                    const float heps = __fmul_rn(0.5f, eps);
                    /* the last structure step may have left the adjoint words of a
                     * rejected proposal */
                    if (prepared != gcur) {
                        nconst = grad_prepare(ws.prog[gcur], cur_ninstr, ws, lane);
                        prepared = gcur;
                    }
                    const float* q0 = ws.Cs[ccur];
                    float* q = ws.Cs[ccur ^ 1];
                    float k0 = 0.0f;
                    for (int i = lane; i < PL; i += 32) {
                        const float m = hmc_momentum(seed, (uint32_t)chain, (uint32_t)step, (uint32_t)i);
                        k0 = fmaf(m, m, k0);
                        ws.mom[i] = __fadd_rn(m, __fmul_rn(heps, ws.gcur[i]));
                        q[i] = q0[i];
                    }
                    k0 = __fmul_rn(0.5f, warp_sum(k0));
                    df lik = df_make(-INFINITY, 0.0f);
                    bool ok = true;
#pragma unroll 1
                    for (int l = 1; l <= nleap && ok; ++l) {
                        bool fin = true;
                        for (int i = lane; i < PL; i += 32) {
                            q[i] = __fadd_rn(q[i], __fmul_rn(eps, ws.mom[i]));
                            fin &= isfinite(q[i]);
                        }
                        ok = __all_sync(FULLMASK, fin);
                        __syncwarp();
                        if (!ok) break;
                        build_grad_program(ws.gprog, q, cur_ninstr, ws.eprog, lane);
                        __syncwarp();
                        int pe = 0;
                        lik = eval_apart<MAXR, G, NV, STREAM>(ws.eprog, cur_ninstr, nconst, ws, dv, p, lane, pe, ws.gnew);
                        st_pts += (unsigned)pe;
                        st_evals++; st_nodes += (unsigned)cur_count;
                        st_np += (unsigned long long)(cur_count + 4) * (unsigned)pe;
                        if (df_invalid(lik)) { ok = false; break; }
                        const float f = l < nleap ? eps : heps;
                        for (int i = lane; i < PL; i += 32) {
                            const float gt = __fadd_rn(__fmul_rn(ws.gnew[i], unscale), dcauchy(q[i]));
                            ws.gnew[i] = gt;
                            ws.mom[i] = __fadd_rn(ws.mom[i], __fmul_rn(f, gt));
                        }
                        __syncwarp();
                    }
                    bool accept = false;
                    float alpha = 0.0f;
                    if (ok) {
                        float k1 = 0.0f;
                        for (int i = lane; i < PL; i += 32) k1 = fmaf(ws.mom[i], ws.mom[i], k1);
                        k1 = __fmul_rn(0.5f, warp_sum(k1));
                        const df cs = cauchy_sum(q, p, lane);
                        const df prior = df_add(length_prior(cur_len, p), cs);
                        const df post = df_add(prior, lik);
                        const df forward = df_make(__fmul_rn(-k0, GPR_DF_SCALE), 0.0f);
                        const df backward = df_make(__fmul_rn(-k1, GPR_DF_SCALE), 0.0f);
                        if (isfinite(k1)) alpha = accept_prob(post, cur_post, backward, forward);
                        accept = isfinite(k1) && mh_accept<RNG>(post, cur_post, backward, forward, r, p);
                        if (accept) {
                            ccur ^= 1;
                            cur_cs = cs; cur_prior = prior; cur_lik = lik; cur_post = post;
                            for (int i = lane; i < PL; i += 32) ws.gcur[i] = ws.gnew[i];
                        }
                    }
                    st_ca += accept;
                    if (adapt) {
                        ++n_adapt;
                        const float t = (float)(n_adapt + 10);
                        hbar = __fadd_rn(__fmul_rn(__fsub_rn(1.0f, __fdiv_rn(1.0f, t)), hbar),
                                         __fdiv_rn(__fsub_rn(p.adapt_target, alpha), t));
                        log_eps = fminf(fmaxf(__fsub_rn(mu, __fmul_rn(sqrtf((float)n_adapt) * 20.0f, hbar)),
                                              -30.0f), 5.0f);
                        const float w = __powf((float)n_adapt, -0.75f);
                        log_eps_bar = __fadd_rn(__fmul_rn(w, log_eps), __fmul_rn(__fsub_rn(1.0f, w), log_eps_bar));
                    }
                    __syncwarp();
                }
            }
            if (p.trace && !init && lane < p.trace_n && chain < p.trace_chains)
                p.trace[((size_t)chain * p.steps + step) * p.trace_n + lane] = ws.Cs[ccur][lane];
        }

        for (int i = lane; i < PL; i += 32) {
            const uint8_t o = ws.ops[cur][i];
            if (o != 255) p.P[(size_t)i * p.N + chain] = (int32_t)o;
            p.C[(size_t)i * p.N + chain] = ws.Cs[ccur][i];
        }
        if (lane == 0) {
            p.prior[chain] = df_to_double_unscaled(cur_prior);
            p.lik[chain] = df_to_double_unscaled(cur_lik);
            if (adapt && n_adapt > 0) p.chain_scale[chain] = expf(log_eps_bar);
            if (p.stats) {
                atomicAdd(&p.stats[GPR_STAT_EVALS], (unsigned long long)st_evals);
                atomicAdd(&p.stats[GPR_STAT_EVAL_NODES], st_nodes);
                atomicAdd(&p.stats[GPR_STAT_EVAL_POINTS], st_pts);
                atomicAdd(&p.stats[GPR_STAT_EVAL_NODE_POINTS], st_np);
                atomicAdd(&p.stats[GPR_STAT_STRUCT_PROPOSED], (unsigned long long)st_sp);
                atomicAdd(&p.stats[GPR_STAT_STRUCT_ACCEPTED], (unsigned long long)st_sa);
                atomicAdd(&p.stats[GPR_STAT_CONST_PROPOSED], (unsigned long long)st_cp);
                atomicAdd(&p.stats[GPR_STAT_CONST_ACCEPTED], (unsigned long long)st_ca);
            }
        }
        __syncwarp();
    }
}

/* The kernels for three input variables (gpr_hmc_v.cu). */
const void* grad_kernel_v3(int maxr, int G);
const void* hmc_kernel_v3(const KParams& p, int G, int stream);

}  // namespace gpr

#endif /* GPR_HMC_CUH */
