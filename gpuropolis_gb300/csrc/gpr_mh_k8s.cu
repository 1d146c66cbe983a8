/* Instantiations of the MH block kernel for streamed data of many passes, one
 * or three input variables: K = 8 points per lane (a translation unit of its
 * own so the kernels compile in parallel). */
#include "gpr_mh.cuh"

namespace gpr {
template __global__ void mh_block_kernel<8, false, 0, false, true, 1, false>(const __grid_constant__ KParams p);
template __global__ void mh_block_kernel<8, false, 1, false, true, 1, false>(const __grid_constant__ KParams p);
template __global__ void mh_block_kernel<8, false, 0, false, true, 3, false>(const __grid_constant__ KParams p);
template __global__ void mh_block_kernel<8, false, 1, false, true, 3, false>(const __grid_constant__ KParams p);
const void* mh_kernel_k8s(int rng, int nv) {
    if (nv == 3) return rng ? (const void*)mh_block_kernel<8, false, 1, false, true, 3, false>
                            : (const void*)mh_block_kernel<8, false, 0, false, true, 3, false>;
    return rng ? (const void*)mh_block_kernel<8, false, 1, false, true, 1, false>
               : (const void*)mh_block_kernel<8, false, 0, false, true, 1, false>;
}
}  // namespace gpr
