/*
 * gpr_hmc_v.cu -- the adjoint and Hamiltonian-move kernels for data with three
 * input variables (x1, x2, x3); a translation unit of its own so that they
 * compile in parallel with the univariate ones (gpr_hmc.cu).
 */
#include "gpr_hmc.cuh"

namespace gpr {

const void* grad_kernel_v3(int maxr, int stream) {
    if (maxr <= 96)
        return stream ? (const void*)loglik_grad_kernel<96, true, 3>
                      : (const void*)loglik_grad_kernel<96, false, 3>;
    return stream ? (const void*)loglik_grad_kernel<192, true, 3>
                  : (const void*)loglik_grad_kernel<192, false, 3>;
}

template <int MAXR, int RNG>
static const void* pick(int stream) {
    return stream ? (const void*)mh_hmc_kernel<MAXR, RNG, true, 3>
                  : (const void*)mh_hmc_kernel<MAXR, RNG, false, 3>;
}

const void* hmc_kernel_v3(const KParams& p, int stream) {
    if (p.max_instr <= 130) return p.rng_mode ? pick<96, 1>(stream) : pick<96, 0>(stream);
    return p.rng_mode ? pick<192, 1>(stream) : pick<192, 0>(stream);
}

}  // namespace gpr
