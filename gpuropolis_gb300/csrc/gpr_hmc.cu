/*
 * gpr_hmc.cu -- instantiations and launchers of the adjoint kernel
 * (gpr_loglik_grad) and of the MH kernel with Hamiltonian constant moves
 * (gpr_hmc.cuh).  The tape's thread-local part holds up to 96 rows
 * (PROGRAM_LENGTH <= 63) or 192 (PROGRAM_LENGTH <= 127); the Hamiltonian kernel
 * has a short dataset staged per CTA and reads a longer one from device memory.
 */
#include "gpr_hmc.cuh"

namespace gpr {


size_t grad_smem_bytes(const KParams& p, int G, int warps_per_cta, int stream) {
    return 16 + (stream ? 0 : align16((size_t)data_arrays(p) * p.nd_pad * 4)) +
           (size_t)warps_per_cta * grad_warp_bytes(p.PL, p.max_instr, G, true);
}

bool grad_supported(const KParams& p) { return p.max_instr <= 258 && p.PL <= 127; }

/* Passes a sweep of the Hamiltonian kernel takes together (hmc_min_ctas).
 *
 * With fixed programs a sweep of two saves decoding: 65,536 chains of the
 * rational model on 1,024 points, 10 moves of 8 leapfrog steps: 72 ms with G = 1, 66 with
 * 2; on 128 points, one pass, 5.2 and 6.7 ms (4 steps, 6 moves).  With structure moves beside
 * them, the warps of an SM are in programs of all kinds, whose long ops wait:
 * what counts is the warps per SM.  65,536 chains of basic ops, PL 31: 128 points
 * 14.5 and 19.3 ms, 1,024 points 43.9 and 68.6 ms.
 * With at most 16 warps per SM for all chains, those of G = 2 have more registers
 * at no cost (2,048 chains of three variables, 4,096 points: 24.5 and 17.9 ms);
 * up to 32 it is as fast or faster (4,096 chains: 1,024 points 9.1 and 6.9 ms), but
 * for three passes, which take two sweeps (384 points 3.9 and 4.7 ms); up to 48
 * from four passes on (6,000 chains, 1,024 points: 10.5 and 9.4 ms). */
int hmc_passes(const KParams& p, int sms) {
    const int passes = (p.nd + GPR_CHUNK_POINTS - 1) / GPR_CHUNK_POINTS;
    if (p.N <= 16 * sms) return 2;
    if (passes <= 1) return 1;
    if (p.struct_every == 0) return 2;
    return p.N <= 32 * sms && passes != 3 || p.N <= 48 * sms && passes > 3 ? 2 : 1;
}

template <int MAXR>
static const void* grad_kernel_t(int G, int nv) {
    if (nv == 3) return grad_kernel_v3(MAXR, G);
    return G == 1 ? (const void*)loglik_grad_kernel<MAXR, 1, 1> : (const void*)loglik_grad_kernel<MAXR, 2, 1>;
}

static cudaError_t launch_grad(const KParams& p, int G, int wpc, double* grad, double* lik, int* later,
                               cudaStream_t st) {
    const size_t smem = (size_t)wpc * grad_warp_bytes(p.PL, p.max_instr, G, false);
    const void* f = p.max_instr <= 130 ? grad_kernel_t<96>(G, p.nv) : grad_kernel_t<192>(G, p.nv);
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    KParams pp = p;
    void* args[] = {(void*)&pp, (void*)&grad, (void*)&lik, (void*)&later};
    return cudaLaunchKernel(f, dim3((p.N + wpc - 1) / wpc), dim3(wpc * 32), args, smem, st);
}

/* Which programs the chains hold is not known here.  Programs of sums, products
 * and quotients are fastest with G = 2, those with a long op (mixed populations)
 * with the warps of G = 1: 65,536 chains of PL 31 on 1,024 points, the rational
 * model 1.06 ms with G = 1 and 0.97 with 2, random programs 2.88 and 4.4 ms.  So
 * from four passes on both run: G = 2 lists the programs with a long op for G = 1
 * (1.00 and 3.01 ms).  With fewer, the second compile costs more than G = 2 gives:
 * G = 1 for all (300 points: 0.59 and 1.70 ms, listed 0.67 and 1.87).  Up to
 * 32 chains per SM G = 2 takes them all (2,048 chains on 1,024 points: 92 and 267
 * us with G = 1, 80 and 230 with 2), if not for one pass of many chains.
 * One warp per CTA with G = 1, where programs differ in length (random
 * programs on 300 points: 1.70 ms, 1.84 with two warps). */
cudaError_t launch_loglik_grad(const KParams& p, int sms, double* grad, double* lik, int* later, cudaStream_t st) {
    if (!grad_supported(p)) return cudaErrorInvalidValue;
    const int passes = (p.nd + GPR_CHUNK_POINTS - 1) / GPR_CHUNK_POINTS;
    if (p.N <= (passes > 1 ? 32 : 16) * sms) return launch_grad(p, 2, 4, grad, lik, nullptr, st);
    if (passes < 4) return launch_grad(p, 1, 1, grad, lik, nullptr, st);
    cudaError_t e = cudaMemsetAsync(later, 0, sizeof(int), st);
    if (e == cudaSuccess) e = launch_grad(p, 2, 4, grad, lik, later, st);
    if (e == cudaSuccess) e = launch_grad(p, 1, 1, grad, lik, later, st);
    return e;
}

template <int MAXR, int G>
static const void* hmc_kernel_t(int rng, int stream) {
    if (rng) return stream ? (const void*)mh_hmc_kernel<MAXR, G, 1, true, 1>
                           : (const void*)mh_hmc_kernel<MAXR, G, 1, false, 1>;
    return stream ? (const void*)mh_hmc_kernel<MAXR, G, 0, true, 1>
                  : (const void*)mh_hmc_kernel<MAXR, G, 0, false, 1>;
}

static const void* hmc_kernel(const KParams& p, int G, int stream) {
    if (p.nv == 3) return hmc_kernel_v3(p, G, stream);
    if (p.max_instr <= 130)
        return G == 1 ? hmc_kernel_t<96, 1>(p.rng_mode, stream) : hmc_kernel_t<96, 2>(p.rng_mode, stream);
    return G == 1 ? hmc_kernel_t<192, 1>(p.rng_mode, stream) : hmc_kernel_t<192, 2>(p.rng_mode, stream);
}

/* The shared-memory share of the L1/shared array: the rest is L1, which holds
 * spilled registers, streamed data and the tape rows beyond those in shared
 * memory.  carveout 0 leaves the driver's default. */
static cudaError_t set_carveout(const void* f, int carveout) {
    return cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                                carveout > 0 ? carveout : -1);
}

cudaError_t hmc_occupancy(const KParams& p, int G, int warps_per_cta, size_t smem, int carveout, int stream,
                          int* ctas_per_sm) {
    if (!grad_supported(p)) return cudaErrorInvalidValue;
    const void* f = hmc_kernel(p, G, stream);
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = set_carveout(f, carveout);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, f, warps_per_cta * 32, smem);
}

cudaError_t launch_hmc_block(const KParams& p, const LaunchCfg& lc, cudaStream_t st) {
    if (!grad_supported(p) || (p.nds > 0 && !lc.stream)) return cudaErrorInvalidValue;
    const void* f = hmc_kernel(p, lc.K / 4, lc.stream);
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lc.smem_bytes);
    if (e == cudaSuccess) e = set_carveout(f, lc.carveout);
    if (e != cudaSuccess) return e;
    KParams pp = p;
    void* args[] = {(void*)&pp};
    return cudaLaunchKernel(f, dim3(lc.ctas), dim3(lc.warps_per_cta * 32), args, lc.smem_bytes, st);
}

}  // namespace gpr
