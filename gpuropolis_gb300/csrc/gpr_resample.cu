/*
 * gpr_resample.cu -- selection over chain posteriors on the device.
 *
 *  - the resampling cutoff of main.cu:1215-1219 (the posterior at rank
 *    (int)(N * quantile) in the order of the reference's comparator,
 *    main.cu:987-995) or max - delta, by radix selection instead of qsort;
 *  - the re-draw of every chain strictly below the cutoff from the initial
 *    distribution (main.cu:1221-1229), driven by a counter-based stream per
 *    chain instead of the host's rand();
 *  - the candidate list of the k best chains, which replaces the external
 *    `sort -g -k3 samples.txt | tail -n k` behind tops.txt (run-all.sh:45).
 *
 * This is integer and byte work over N doubles (1 MB at 131,072 chains): one
 * cluster of CTAs per segment holds the order-preserving 64-bit keys in
 * registers and radix-selects over them (8 bits per round), and a CTA re-draws
 * a group of the chains below the cutoff in phases.
 */
#include <cooperative_groups.h>
#include <algorithm>

#include "gpr_mh.cuh"
#include "gpr_select.h"

namespace gpr {

#define GPR_SEL_THREADS 1024
#define GPR_SEL_REGS 8       /* keys a thread holds in registers; the rest are re-read from `keys` (L2) */
#define GPR_SEL_CLUSTER 16   /* CTAs per segment above GPR_SEL_ONE keys: 131,072 keys stay in registers */
#define GPR_SEL_ONE 4096

/* The key of rank `rank` (0-based, ascending) among the N keys of a segment,
 * into out[segment]; every key is left in keys[] (launch_collect reads them),
 * and *zero set to 0 for the counting kernel that follows.  host (may be null;
 * one segment): the key also goes to host->key.
 * The last rank is a maximum: one reduction, which also gives the smallest
 * index that holds it (host->first).  Otherwise a radix selection:
 * per 8-bit digit a histogram of the keys that match the digits fixed so far,
 * summed over the cluster through distributed shared memory, and the bin that
 * holds the rank; it ends as soon as one key is left in that bin.
 *
 * Bound by latency: a round is a histogram in shared memory, a cluster
 * barrier and a read of the other CTAs' bins, 3 us or so.  131,072 keys, rank
 * N/2: 22 us, the maximum 13 us; 252 us for either with one CTA that re-read
 * the keys from L2 in each of the 8 rounds, added the shared leading digits to
 * one bin key by key and never ended early; 31 us with 8 CTAs of 16 keys a
 * thread. */
__global__ void __launch_bounds__(GPR_SEL_THREADS) select_rank_kernel(const double* prior, const double* lik,
                                                                      unsigned long long* keys, int N, int rank,
                                                                      unsigned long long* out, int* zero,
                                                                      SelectResult* host) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned ncta = cluster.num_blocks(), cta = cluster.block_rank();
    const int seg = blockIdx.x / ncta;
    const size_t off = (size_t)seg * (size_t)N;
    prior += off; lik += off; keys += off; out += seg;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) *zero = 0;
    /* key number i of this thread: chain t0 + i * stride */
    const int t0 = (int)(cta * blockDim.x + threadIdx.x), stride = (int)(ncta * blockDim.x);

    unsigned long long mine[GPR_SEL_REGS];
#pragma unroll
    for (int j = 0; j < GPR_SEL_REGS; ++j) {
        const int i = t0 + j * stride;
        mine[j] = 0ull;
        if (i < N) { mine[j] = gpr_post_key(prior[i] + lik[i]); keys[i] = mine[j]; }
    }
    for (long long i = t0 + (long long)GPR_SEL_REGS * stride; i < N; i += stride)
        keys[i] = gpr_post_key(prior[i] + lik[i]);

    if (rank == N - 1) {
        __shared__ unsigned long long s_max[32];
        __shared__ int s_idx[32];
        unsigned long long best = 0ull;
        int idx = 0x7fffffff;
        auto take = [&](unsigned long long k, int i) {
            if (k > best || (k == best && i < idx)) { best = k; idx = i; }
        };
#pragma unroll
        for (int j = 0; j < GPR_SEL_REGS; ++j)
            if (t0 + j * stride < N) take(mine[j], t0 + j * stride);
        for (long long i = t0 + (long long)GPR_SEL_REGS * stride; i < N; i += stride) take(keys[i], (int)i);
        auto warp_best = [&]() {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long k = __shfl_xor_sync(FULLMASK, best, o);
                const int i = __shfl_xor_sync(FULLMASK, idx, o);
                take(k, i);
            }
        };
        warp_best();
        if (lane == 0) { s_max[warp] = best; s_idx[warp] = idx; }
        __syncthreads();
        if (warp == 0) {
            best = lane < nwarps ? s_max[lane] : 0ull;
            idx = lane < nwarps ? s_idx[lane] : 0x7fffffff;
            warp_best();
            __syncwarp();
            if (lane == 0) { s_max[0] = best; s_idx[0] = idx; }
        }
        cluster.sync();
        if (cta == 0 && threadIdx.x == 0) {
            for (unsigned c = 1; c < ncta; ++c)
                take(*cluster.map_shared_rank(&s_max[0], c), *cluster.map_shared_rank(&s_idx[0], c));
            *out = best;
            if (host) { host->key = best; host->first = idx; }
        }
        cluster.sync();   /* no CTA leaves while its shared memory is read */
        return;
    }

    __shared__ unsigned hist[2][256];      /* this CTA's counts, alternating between rounds */
    __shared__ unsigned s_tot[256];
    __shared__ unsigned long long s_prefix;
    __shared__ int s_rank;
    __shared__ unsigned s_left;
    unsigned long long prefix = 0ull, mask = 0ull;
    int r = rank, round = 0;
#pragma unroll 1
    for (int shift = 56; shift >= 0; shift -= 8, ++round) {
        /* last read by other CTAs two rounds ago, before the last round's cluster barrier */
        unsigned* h = hist[round & 1];
        for (int i = threadIdx.x; i < 256; i += blockDim.x) { h[i] = 0u; s_tot[i] = 0u; }
        __syncthreads();
        auto add = [&](unsigned long long k, bool in) {
            const bool hit = in && (k & mask) == prefix;
            const unsigned d = (unsigned)(k >> shift) & 255u;
            /* the leading digits are mostly shared: one add per warp where they are */
            const unsigned act = __ballot_sync(FULLMASK, hit);
            if (!act) return;
            const unsigned d0 = __shfl_sync(FULLMASK, d, __ffs(act) - 1);
            if (__all_sync(FULLMASK, !hit || d == d0)) {
                if (lane == 0) atomicAdd(&h[d0], (unsigned)__popc(act));
            } else if (hit) {
                atomicAdd(&h[d], 1u);
            }
        };
#pragma unroll
        for (int j = 0; j < GPR_SEL_REGS; ++j)
            if (j * stride < N) add(mine[j], t0 + j * stride < N);
        for (long long i0 = (long long)GPR_SEL_REGS * stride; i0 < N; i0 += stride) {
            const long long i = i0 + t0;
            add(i < N ? keys[i] : 0ull, i < N);
        }
        cluster.sync();
        if (ncta == 1) {
            for (int i = threadIdx.x; i < 256; i += blockDim.x) s_tot[i] = h[i];
        } else {
            /* a cluster has 1024 threads per CTA: four threads per bin, four CTAs' counts each */
            const int bin = threadIdx.x & 255, part = threadIdx.x >> 8;
            unsigned v = 0;
#pragma unroll
            for (int c = 0; c < GPR_SEL_CLUSTER / 4; ++c)
                v += *cluster.map_shared_rank(&h[bin], part * (GPR_SEL_CLUSTER / 4) + c);
            if (v) atomicAdd(&s_tot[bin], v);
        }
        __syncthreads();
        if (warp == 0) {
            unsigned c[8];
            unsigned sum = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) { c[j] = s_tot[lane * 8 + j]; sum += c[j]; }
            unsigned incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(FULLMASK, incl, o);
                if (lane >= o) incl += t;
            }
            unsigned cum = incl - sum;
            if (cum <= (unsigned)r && (unsigned)r < incl) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if ((unsigned)r >= cum && (unsigned)r < cum + c[j]) {
                        s_prefix = prefix | ((unsigned long long)(lane * 8 + j) << shift);
                        s_rank = r - (int)cum;
                        s_left = c[j];
                    }
                    cum += c[j];
                }
            }
        }
        __syncthreads();
        prefix = s_prefix;
        r = s_rank;
        mask |= 0xffull << shift;
        if (s_left == 1u) break;   /* the same in every CTA of the cluster */
    }
    /* the key with this prefix: the prefix itself after all digits, else the one key that has it */
    auto found = [&](unsigned long long k) {
        *out = k;
        if (host) host->key = k;
    };
    if (mask == ~0ull) {
        if (cta == 0 && threadIdx.x == 0) found(prefix);
    } else {
#pragma unroll
        for (int j = 0; j < GPR_SEL_REGS; ++j)
            if (t0 + j * stride < N && (mine[j] & mask) == prefix) found(mine[j]);
        for (long long i = t0 + (long long)GPR_SEL_REGS * stride; i < N; i += stride)
            if ((keys[i] & mask) == prefix) found(keys[i]);
    }
    cluster.sync();   /* no CTA leaves while its bins are read */
}

/* The chains whose posterior is strictly below the cutoff, appended to list
 * (each CTA's in order), and their number added to *n.  seg_len > 0: chain c
 * compares with the cutoff of its segment, sel_key[c / seg_len]. */
__global__ void __launch_bounds__(256) below_kernel(const double* prior, const double* lik, int N,
                                                    const unsigned long long* sel_key, int seg_len, int map_delta,
                                                    double delta, int* list, int* n) {
    __shared__ int s_cnt[8], s_base;
    const int chain = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool below = false;
    if (chain < N) {
        double cutoff = gpr_key_value(sel_key[seg_len > 0 ? chain / seg_len : 0]);
        if (map_delta) cutoff -= delta;
        below = prior[chain] + lik[chain] < cutoff;
    }
    const unsigned b = __ballot_sync(FULLMASK, below);
    if (lane == 0) s_cnt[warp] = __popc(b);
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        before += w < warp ? s_cnt[w] : 0;
        total += s_cnt[w];
    }
    if (threadIdx.x == 0) s_base = total ? atomicAdd(n, total) : 0;
    __syncthreads();
    if (below) list[s_base + before + __popc(b & ((1u << lane) - 1u))] = chain;
}

#define GPR_RD_THREADS 256

/* Where draw q of a chain is kept, in rows of CH.  With fewer than 32 chains a
 * row is left out after every 32 draws, so that the threads of a warp that work
 * on different words of them meet different banks. */
__host__ __device__ __forceinline__ constexpr int redraw_row(int CH, int q) { return CH < 32 ? q + (q >> 5) : q; }
/* Shared memory of a CTA that re-draws CH chains and keeps `draws` draws of
 * each (a multiple of 32). */
__host__ __device__ __forceinline__ size_t redraw_smem_bytes(int CH, int PL, int draws) {
    return (size_t)CH * ((size_t)redraw_row(CH, draws) * 4 + (size_t)(draws / 32) * 12 + (size_t)PL * 4);
}

/* A draw as the CTA keeps it: what it would be as a uniform's integer, as an
 * order and as an op index, and the distance to the next constant's order if
 * it is an order itself (GPR_RD_FAR: to be looked for). */
#define GPR_RD_UNIFORM(w) ((w) & 0xfffffu)
#define GPR_RD_ORDER(w) (((w) >> 20) & 7u)
#define GPR_RD_OP(w) (((w) >> 23) & 31u)
#define GPR_RD_STEP(w) ((w) >> 28)
#define GPR_RD_FAR 15u

/* Re-draw the listed chains in the reference's order (all PL ops, then all PL
 * constants; main.cu:1224-1228): op = ops[random_int(n_ops - 1)], constant =
 * 10^(random_int(8) - 4) * random_normal().  Draws come from the Philox stream
 * keyed by (seed, (chain + chain_offset) | 2^31): with the offset of a
 * handle's first chain in a population spread over several handles or GPUs,
 * every chain of the population has its own stream.
 *
 * random_int rejects (one op draw in n_ops, one order draw in nine, one
 * uniform's in 4,400), so which draw belongs to what is only known one after
 * the other; the draws themselves (counter-based, 90 instructions per four)
 * and the normals (about 95 each) are not serial.  A CTA takes CH chains, its
 * threads in groups of one per chain, in phases:
 *   1. all groups make the first `draws` draws of every chain and, 32 at a time,
 *      the bits that say which random_int would take as an op, as an order, and
 *      not as a uniform;
 *   2. all groups, a word of those bits each: the ops' positions by their rank,
 *      and for every draw the distance to the order that follows if it is one;
 *   3. one thread per chain follows those distances and notes each constant's
 *      position, while the other warps write the ops;
 *   4. all groups make the constants.
 * A chain that needs more draws than were made is drawn one after the other by
 * its own thread.
 * 65,536 of 131,072 chains of 63 nodes: 89 us.  One thread per chain for
 * all of it: 195 us (long dependent sequences in few warps, and a Philox block
 * issued by the warp whenever one of its threads ran out of draws).  Phases 2
 * and 3 as one thread's walk over the bits: 122 us (the other warps wait).
 * CH: see launch_redraw. */
template <int CH>
__global__ void __launch_bounds__(GPR_RD_THREADS) redraw_kernel(const __grid_constant__ KParams p, const int* list,
                                                                const int* n_list, uint32_t seed,
                                                                uint32_t chain_offset, Magic mag_ops1,
                                                                Magic mag_order, uint32_t op_below,
                                                                uint32_t order_below, uint32_t uniform_below,
                                                                int draws) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float s_pow10[8];
    __shared__ int32_t s_map[32];
    __shared__ int s_start[CH];                                /* first draw after the ops (-1: too few draws) */
    __shared__ int s_slow[CH];
    const int PL = p.PL, nw = draws / 32;
    const int tid = (int)threadIdx.x, c = tid % CH, group = tid / CH, groups = GPR_RD_THREADS / CH;
    const int rows = redraw_row(CH, draws);
    uint32_t* s_draw = (uint32_t*)smem + c;                    /* [rows][CH], this chain's column */
    uint32_t* s_opbit = s_draw + rows * CH;                    /* [draws / 32][CH]: taken as an op ... */
    uint32_t* s_orbit = s_opbit + nw * CH;                     /* ... as an order ... */
    uint32_t* s_unbit = s_orbit + nw * CH;                     /* ... rejected as a uniform */
    uint16_t* s_oppos = (uint16_t*)((uint32_t*)smem + (rows + 3 * nw) * CH) + c;   /* [PL][CH] */
    uint16_t* s_cpos = s_oppos + PL * CH;                      /* [PL][CH] */
    auto draw = [&](int q) -> uint32_t& { return s_draw[redraw_row(CH, q) * CH]; };
    const int n = *n_list;
    const int first = blockIdx.x * CH;
    if (first >= n) return;
    if (tid < 8) s_pow10[tid] = gpr_pow10_order(tid - 4);
    if (tid >= 32 && tid < 64) s_map[tid - 32] = p.opmap[tid - 32];
    if (tid >= 64 && tid < 64 + CH) s_start[tid - 64] = -1;
    /* threads past the list's end follow its last chain and write nothing */
    const bool live = first + c < n;
    const int chain = list[min(first + c, n - 1)];
    const uint32_t key1 = ((uint32_t)chain + chain_offset) | 0x80000000u;
#pragma unroll 1
    for (int w = group; w < nw; w += groups) {
        uint32_t ob = 0u, rb = 0u, ub = 0u;
#pragma unroll 2
        for (int b = 0; b < 8; ++b) {
            uint32_t r[4] = {(uint32_t)(8 * w + b), 0u, 0u, 0u};
            gpr_philox4x32_10(r, seed, key1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t x = r[j] >> 1;
                draw(32 * w + 4 * b + j) =
                    (magic_div(x, p.mag_1e6) & 0xfffffu) | ((magic_div(x, mag_order) & 7u) << 20) |
                    ((magic_div(x, mag_ops1) & 31u) << 23);
                ob |= (x < op_below ? 1u : 0u) << (4 * b + j);
                rb |= (x < order_below ? 1u : 0u) << (4 * b + j);
                ub |= (x < uniform_below ? 0u : 1u) << (4 * b + j);
            }
        }
        s_opbit[w * CH] = ob;
        s_orbit[w * CH] = rb;
        s_unbit[w * CH] = ub;
    }
    __syncthreads();
#pragma unroll 1
    for (int w = group; w < nw; w += groups) {
        int rank = 0;
        for (int v = 0; v < w; ++v) rank += __popc(s_opbit[v * CH]);
        uint32_t m = s_opbit[w * CH];
        for (; m && rank < PL; ++rank, m &= m - 1u) {
            const int pos = 32 * w + __ffs(m) - 1;
            s_oppos[rank * CH] = (uint16_t)pos;
            if (rank == PL - 1) s_start[c] = pos + 1;
        }
        /* an order, two uniforms, and on to the next order */
        const uint32_t r0 = s_orbit[w * CH], r1 = w + 1 < nw ? s_orbit[(w + 1) * CH] : 0u;
        const uint32_t u0 = s_unbit[w * CH], u1 = w + 1 < nw ? s_unbit[(w + 1) * CH] : ~0u;
#pragma unroll
        for (int b = 0; b < 32; ++b) {
            const uint32_t next = b + 3 < 32 ? __funnelshift_r(r0, r1, (b + 3) & 31) : r1 >> ((b + 3) & 31);
            const uint32_t uni = b + 1 < 32 ? __funnelshift_r(u0, u1, (b + 1) & 31) : u1;
            const uint32_t step = (uint32_t)__ffs(next) + 2u;
            const bool far = next == 0u || step >= GPR_RD_FAR || (uni & 3u);
            draw(32 * w + b) |= (far ? GPR_RD_FAR : step) << 28;
        }
    }
    __syncthreads();
    auto find = [&](const uint32_t* bits, int q, uint32_t flip) {   /* the first draw from q on whose bit is set */
        while (q < draws && !(((bits[(q >> 5) * CH] ^ flip) >> (q & 31)) & 1u)) ++q;
        return q;
    };
    const size_t N = (size_t)p.N;
    if (tid < CH) {
        int pos = s_start[c];
        bool slow = pos < 0;
        if (!slow) pos = find(s_orbit, pos, 0u);
#pragma unroll 1
        for (int node = 0; node < PL && !slow; ++node) {
            if (pos + 2 >= draws) { slow = true; break; }
            s_cpos[node * CH] = (uint16_t)pos;
            const uint32_t step = GPR_RD_STEP(draw(pos));
            if (step != GPR_RD_FAR) {
                pos += (int)step;
            } else {
                pos = find(s_unbit, find(s_unbit, pos + 1, ~0u) + 1, ~0u) + 1;
                slow = pos > draws;
                pos = find(s_orbit, pos, 0u);
            }
        }
        s_slow[c] = slow;
    } else if (tid >= 32 && live && s_start[c] >= 0) {
#pragma unroll 4
        for (int i = group - 32 / CH; i < PL; i += groups - 32 / CH)
            p.P[(size_t)i * N + chain] = s_map[GPR_RD_OP(draw(s_oppos[i * CH]))];
    }
    __syncthreads();
    const bool fast = live && !s_slow[c];
#pragma unroll 1
    for (int i = group; i < PL; i += groups) {
        if (!fast) continue;
        const int q = s_cpos[i * CH];
        const uint32_t w = draw(q);
        int qu = q + 1, qv = q + 2;
        if (GPR_RD_STEP(w) == GPR_RD_FAR) { qu = find(s_unbit, qu, ~0u); qv = find(s_unbit, qu + 1, ~0u); }
        const float u = gpr_rng_k_over_1e6((int)GPR_RD_UNIFORM(draw(qu)));
        const float v = gpr_rng_k_over_1e6((int)GPR_RD_UNIFORM(draw(qv)));
        const float a = __fsqrt_rn(__fmul_rn(-2.0f, gpr_rng_logf(u)));
        const float z = __fmul_rn(a, gpr_rng_sinf(gpr_rng_twopi_times(v)));
        p.C[(size_t)i * N + chain] = __fmul_rn(s_pow10[GPR_RD_ORDER(w)], z);
    }
    if (tid < CH && live && !fast) {
        Rng r;
        r.s = 0u; r.key0 = seed; r.key1 = key1; r.blk = 0xffffffffu; r.drawn = 0u;
        r.w0 = r.w1 = r.w2 = r.w3 = 0u;
#pragma unroll 1
        for (int i = 0; i < PL; ++i) p.P[(size_t)i * N + chain] = s_map[random_int<1>(r, p.nops - 1, mag_ops1)];
#pragma unroll 1
        for (int i = 0; i < PL; ++i) {
            const int order = random_int<1>(r, 8, mag_order);
            p.C[(size_t)i * N + chain] = __fmul_rn(s_pow10[order], random_normal<1>(r, p));
        }
    }
}

/* Chains whose posterior is at least that of key *sel less margin (NaN
 * never; every other chain when *sel is NaN's key), appended in any order. */
__global__ void collect_kernel(const unsigned long long* keys, int N, const unsigned long long* sel, double margin,
                               int* out, int cap, int* count) {
    const unsigned long long k0 = *sel;
    const unsigned long long kmin = k0 == 0ull ? 1ull : gpr_post_key(gpr_key_value(k0) - margin);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const unsigned long long k = keys[i];
        if (k != 0ull && k >= kmin) {
            const int j = atomicAdd(count, 1);
            if (j < cap) out[j] = i;
        }
    }
}

static int grid_for(int n, int threads) {
    int b = (n + threads - 1) / threads;
    return b < 1 ? 1 : (b > 4096 ? 4096 : b);
}

cudaError_t launch_select(const KParams& p, int rank, unsigned long long* keys, unsigned long long* out,
                          int* zero, SelectResult* host, cudaStream_t st, int segments) {
    if (segments < 1 || p.N % segments) return cudaErrorInvalidValue;
    const int n = p.N / segments;
    /* One CTA up to GPR_SEL_ONE keys (four per thread): a round over them takes
     * less than a cluster barrier, and a batched handle's segments (hundreds of
     * them, 15 us for 256 of 512 keys) fill the device by themselves. */
    int ncta = n > GPR_SEL_ONE ? GPR_SEL_CLUSTER : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3((unsigned)std::min(GPR_SEL_THREADS, (n + 31) / 32 * 32));
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaFuncSetAttribute((const void*)select_rank_kernel,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        ncta = 1;
    }
    /* Where a cluster of that size cannot be resident (it is beyond the portable
     * eight) the launch says so, and one CTA selects. */
    for (;; ncta = 1) {
        cfg.gridDim = dim3((unsigned)segments * ncta);
        attr[0].val.clusterDim.x = ncta;
        e = cudaLaunchKernelEx(&cfg, select_rank_kernel, p.prior, p.lik, keys, n, rank, out, zero, host);
        if (e == cudaSuccess || ncta == 1) return e;
        (void)cudaGetLastError();
    }
}

/* Chains per CTA (CH): the most of 32, 16 and 8 whose draws leave room for three
 * CTAs per SM, whose phases then overlap.  131,072 chains, 95% of them re-drawn,
 * 8 ops: 127 nodes 446 us with 32 chains (98 KB), 410 with 16; 255 nodes 1,359
 * with 32 (186 KB), 1,118 with 16 and 1,028 with 8, 1,086 with a thread per chain
 * (selection over one CTA included).  Two ops, 255 nodes: 14.2 ms where 200 KB for
 * 32 chains cut their draws short, 1.30 now, 1.43 with a thread per chain. */
#define GPR_RD_SMEM (72 * 1024)

cudaError_t launch_redraw(const KParams& p, const unsigned long long* sel_key, int seg_len, int map_delta,
                          double delta, uint32_t seed, Magic mag_ops1, Magic mag_order, int* list, int* n_redrawn,
                          cudaStream_t st, uint32_t chain_offset) {
    below_kernel<<<(p.N + 255) / 256, 256, 0, st>>>(p.prior, p.lik, p.N, sel_key, seg_len, map_delta, delta, list,
                                                    n_redrawn);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    /* Draws per chain kept in shared memory: the mean and eight standard
     * deviations (an op takes a draw in n_ops - 1 of n_ops cases, an order one in
     * 8 of 9): at most 1,536, of 255 nodes and two ops. */
    const double q = 1.0 / p.nops, mean = p.PL * (1.0 / (1.0 - q) + 2.0 + 9.0 / 8.0),
                 sd = sqrt(p.PL * (q / ((1.0 - q) * (1.0 - q)) + 9.0 / 64.0));
    const int draws = ((int)(mean + 8.0 * sd + 4.0) + 31) / 32 * 32;
    /* x / d < n  <=>  x < n d, d the divisor of random_int(n) */
    const uint32_t op_below = (uint32_t)(p.nops - 1) * (2147483647u / (uint32_t)p.nops),
                   order_below = 8u * (2147483647u / 9u), uniform_below = 1000000u * (2147483647u / 1000001u);
    int CH = 32;
    while (CH > 8 && redraw_smem_bytes(CH, p.PL, draws) > GPR_RD_SMEM) CH /= 2;
    const size_t smem = redraw_smem_bytes(CH, p.PL, draws);
    const auto f = CH == 32 ? redraw_kernel<32> : CH == 16 ? redraw_kernel<16> : redraw_kernel<8>;
    e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    f<<<(p.N + CH - 1) / CH, GPR_RD_THREADS, smem, st>>>(p, list, n_redrawn, seed, chain_offset, mag_ops1, mag_order,
                                                         op_below, order_below, uniform_below, draws);
    return cudaGetLastError();
}

cudaError_t launch_collect(const unsigned long long* keys, int N, const unsigned long long* sel, double margin,
                           int* out, int cap, int* count, cudaStream_t st) {
    collect_kernel<<<grid_for(N, 256), 256, 0, st>>>(keys, N, sel, margin, out, cap, count);
    return cudaGetLastError();
}

}  // namespace gpr
