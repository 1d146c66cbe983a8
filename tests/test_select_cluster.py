"""Selection where a cluster of 16 CTAs cannot be resident: the launch is made
again with one CTA per segment (CPU: a runtime that refuses such clusters), and
one CTA selects from any number of keys (GPU), by rank and for the largest."""
import os
import shutil
import subprocess

import pytest

from tests import fake_cuda

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
def test_selection_without_large_clusters(tmp_path):
    fake_cuda.run(fake_cuda.link(tmp_path), """
import numpy as np
s = g.Sampler(8192, program_length=3)
s.set_scores(np.zeros(8192), np.zeros(8192))
for limit, sizes in ((16, (0, 3)), (8, (3, 0)), (1, (3, 0))):
    before = [fake.fake_clusters(1), fake.fake_clusters(16)]
    fake.fake_max_cluster(limit)
    s.map_chain()
    s.top_chains(10)
    s.resample(0, 0.5, 3)
    assert (fake.fake_clusters(1) - before[0], fake.fake_clusters(16) - before[1]) == sizes
""")


_SOURCE = r"""
#include "gpr_resample.cu"
#include <stdio.h>
#include <algorithm>
#include <vector>
using namespace gpr;
int main() {
    const int sizes[] = {1, 31, 1024, 4097, 8192, 8193, 170001};
    for (int N : sizes) {
        std::vector<double> lik(N), prior(N, -1.0);
        std::vector<unsigned long long> want(N);
        unsigned x = 12345u + N;
        for (int i = 0; i < N; ++i) {
            x = x * 1664525u + 1013904223u;
            lik[i] = i % 97 == 0 ? -INFINITY : i % 89 == 0 ? NAN : -(double)((x >> 8) % (N / 2 + 3)) * 0.37;
            want[i] = gpr_post_key(prior[i] + lik[i]);
        }
        std::vector<unsigned long long> sorted = want;
        std::sort(sorted.begin(), sorted.end());
        double *dl, *dp;
        unsigned long long *keys, *out;
        int* zero;
        SelectResult* host;
        if (cudaMalloc(&dl, N * 8) || cudaMalloc(&dp, N * 8) || cudaMalloc(&keys, N * 8) || cudaMalloc(&out, 8) ||
            cudaMalloc(&zero, 4) || cudaHostAlloc((void**)&host, sizeof *host, 0)) return 2;
        cudaMemcpy(dl, lik.data(), N * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(dp, prior.data(), N * 8, cudaMemcpyHostToDevice);
        const int ranks[] = {0, N / 3, N / 2, N - 1};
        for (int r : ranks) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1);
            cfg.blockDim = dim3((unsigned)std::min(GPR_SEL_THREADS, (N + 31) / 32 * 32));
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaLaunchKernelEx(&cfg, select_rank_kernel, (const double*)dp, (const double*)dl, keys, N, r, out, zero, host)) return 3;
            unsigned long long got;
            std::vector<unsigned long long> all(N);
            cudaMemcpy(&got, out, 8, cudaMemcpyDeviceToHost);
            if (cudaMemcpy(all.data(), keys, N * 8, cudaMemcpyDeviceToHost)) return 4;
            if (got != sorted[r] || host->key != got || all != want) { printf("N %d rank %d\n", N, r); return 1; }
            if (r == N - 1 && host->first != (int)(std::find(want.begin(), want.end(), got) - want.begin())) return 5;
        }
        cudaFree(dl); cudaFree(dp); cudaFree(keys); cudaFree(out); cudaFree(zero); cudaFreeHost(host);
    }
    return 0;
}
"""


@pytest.mark.gpu
def test_one_cta_selects_from_any_number_of_keys(tmp_path):
    (tmp_path / "s.cu").write_text(_SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(_ROOT, "gpuropolis_gb300", "csrc"), "-I",
                    os.path.join(_ROOT, "include"), "-o", str(tmp_path / "s"), str(tmp_path / "s.cu")], check=True)
    r = subprocess.run([str(tmp_path / "s")], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
