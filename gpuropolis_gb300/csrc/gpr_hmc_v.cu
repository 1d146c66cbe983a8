/*
 * gpr_hmc_v.cu -- the adjoint and Hamiltonian-move kernels for data with three
 * input variables (x1, x2, x3); a translation unit of its own so that they
 * compile in parallel with the univariate ones (gpr_hmc.cu).
 */
#include "gpr_hmc.cuh"

namespace gpr {

const void* grad_kernel_v3(int maxr, int G) {
    if (maxr <= 96)
        return G == 1 ? (const void*)loglik_grad_kernel<96, 1, 3> : (const void*)loglik_grad_kernel<96, 2, 3>;
    return G == 1 ? (const void*)loglik_grad_kernel<192, 1, 3> : (const void*)loglik_grad_kernel<192, 2, 3>;
}

template <int MAXR, int G>
static const void* pick(int rng, int stream) {
    if (rng) return stream ? (const void*)mh_hmc_kernel<MAXR, G, 1, true, 3>
                           : (const void*)mh_hmc_kernel<MAXR, G, 1, false, 3>;
    return stream ? (const void*)mh_hmc_kernel<MAXR, G, 0, true, 3>
                  : (const void*)mh_hmc_kernel<MAXR, G, 0, false, 3>;
}

const void* hmc_kernel_v3(const KParams& p, int G, int stream) {
    if (p.max_instr <= 130) return G == 1 ? pick<96, 1>(p.rng_mode, stream) : pick<96, 2>(p.rng_mode, stream);
    return G == 1 ? pick<192, 1>(p.rng_mode, stream) : pick<192, 2>(p.rng_mode, stream);
}

}  // namespace gpr
