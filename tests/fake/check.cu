/* What a launch of the block kernels needs of its parameters: the rows for the
 * chunk sums that its shared-memory board does not hold, inside a live block of
 * device memory. */
#include <stdio.h>

#include "gpr_kernels.cuh"

extern "C" size_t fake_room(const void* p);

extern "C" int fake_check(const void* f, void** args, unsigned grid, char* why, size_t n) {
    using namespace gpr;
    int need = -1, rows = 0;
    const KParams& p = *(const KParams*)args[0];
    for (int rng = 0; rng < 2; ++rng) {
        for (int nv = 1; nv <= 3; nv += 2) {
            if (f == mh_kernel_k8s(rng, nv)) { need = mh_part_stride(p.nd); rows = 8; }
            if (f == pipe_kernel_k8s(rng, nv)) { need = pipe_part_stride(p.nd); rows = 16; }
        }
        for (int stream = 0; stream < 2; ++stream) {
            if (f == pipe_kernel_k4(rng, 0, 0, stream) || f == pipe_kernel_k4v(rng, 0, stream) ||
                f == pipe_kernel_k4b(rng, 0, stream, 1) || f == pipe_kernel_k4b(rng, 0, stream, 3)) {
                need = pipe_part_stride(p.nd);
                rows = 16;
            }
        }
    }
    if (need <= 0) return 1;
    if (p.part_stride < need) {
        snprintf(why, n, "%d points with rows of %d sums", p.nd, p.part_stride);
        return 0;
    }
    if (fake_room(p.part) < (size_t)grid * rows * p.part_stride * sizeof(float)) {
        snprintf(why, n, "%u CTAs of %d rows of %d sums in %zu bytes", grid, rows, p.part_stride, fake_room(p.part));
        return 0;
    }
    return 1;
}

extern "C" unsigned fake_cluster(const void* config) {
    const cudaLaunchConfig_t* c = (const cudaLaunchConfig_t*)config;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) return c->attrs[i].val.clusterDim.x;
    return 1;
}
