"""Re-drawing long programs: few ops take many draws (a redrawn op is rejected
once in n_ops), and a CTA re-draws 32, 16 or 8 chains by the shared memory they
take.  Against the oracle's re-draw, bit for bit, with list lengths that are no
multiple of any of them.  Then the kernel's own way out, a chain that needs more
draws than were kept: with fewer kept than the launcher keeps, some or all chains
take it, beside others that do not, and the result stays the same."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
g = pytest.importorskip("gpuropolis_gb300")
port = pytest.importorskip("oracle.port")

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("PL", [1, 63, 95, 127, 255])
@pytest.mark.parametrize("n_ops", [2, 3, 8, 27])
def test_redraw_of_long_programs(PL, n_ops):
    N, ops = 1003, list(g.OPSET_REFERENCE)[:n_ops]
    P0, C0 = g.host_init_chains(N, PL, PL, ops=ops)
    prior, lik = H.mixed_scores(N, seed=n_ops)
    s = g.Sampler(N, program_length=PL, ops=ops)
    try:
        s.set_state(P0, C0)
        s.set_scores(prior, lik)
        n, cut = s.resample(0, 0.62, seed=PL + 7)
        P1, C1, _, _ = s.get_state()
    finally:
        s.close()
    n_ref, cut_ref = port.resample(port.cfg(PL=PL, ops=ops), P0, C0, prior, lik, 0, 0.62, PL + 7)
    assert n == n_ref and n % 8 and cut == cut_ref
    assert np.array_equal(P1, P0) and np.array_equal(C1.view(np.uint32), C0.view(np.uint32))


_SOURCE = r"""
#include "gpr_resample.cu"
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <vector>
using namespace gpr;
static Magic magic(uint32_t n) {         /* divisor 2147483647 / (n + 1), as the library's */
    const uint32_t d = 2147483647u / (n + 1);
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;
    Magic m;
    m.s = 31 + l;
    m.m = (uint32_t)(((1ull << m.s) + d - 1) / d);
    return m;
}
template <int CH>
static bool run(int N, int PL, int nops, int draws, std::vector<int>& P, std::vector<float>& C) {
    KParams p;
    memset(&p, 0, sizeof p);
    p.N = N; p.PL = PL; p.nops = nops; p.mag_1e6 = magic(1000000);
    for (int i = 0; i < nops; ++i) p.opmap[i] = (int8_t)(i + 1);
    int *list, *n;
    std::vector<int> all(N);
    for (int i = 0; i < N; ++i) all[i] = N - 1 - i;
    const size_t cells = (size_t)N * PL;
    if (cudaMalloc(&p.P, cells * 4) || cudaMalloc(&p.C, cells * 4) || cudaMalloc(&list, N * 4) || cudaMalloc(&n, 4)) return false;
    cudaMemset(p.P, 0, cells * 4);
    cudaMemset(p.C, 0, cells * 4);
    cudaMemcpy(list, all.data(), N * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(n, &N, 4, cudaMemcpyHostToDevice);
    const size_t smem = redraw_smem_bytes(CH, PL, draws);
    if (smem > 220 * 1024) return false;
    cudaFuncSetAttribute(redraw_kernel<CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    redraw_kernel<CH><<<(N + CH - 1) / CH, GPR_RD_THREADS, smem>>>(
        p, list, n, 77u, 5u, magic(nops - 1), magic(8), (uint32_t)(nops - 1) * (2147483647u / (uint32_t)nops),
        8u * (2147483647u / 9u), 1000000u * (2147483647u / 1000001u), draws);
    P.resize(cells); C.resize(cells);
    cudaMemcpy(P.data(), p.P, cells * 4, cudaMemcpyDeviceToHost);
    const bool ok = cudaMemcpy(C.data(), p.C, cells * 4, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(p.P); cudaFree(p.C); cudaFree(list); cudaFree(n);
    return ok;
}
int main(int argc, char** argv) {
    const int N = 203, PL = atoi(argv[1]), nops = atoi(argv[2]);
    std::vector<int> P0, P;
    std::vector<float> C0, C;
    int checked = 0;
    if (!run<8>(N, PL, nops, (9 * PL + 400) / 32 * 32, P0, C0)) return 2;      /* more than any chain needs */
    for (int i = 3; i < argc; ++i) {
        const int draws = atoi(argv[i]);
        for (int k = 0; k < 3; ++k) {
            if (!(k == 0 ? run<8>(N, PL, nops, draws, P, C) : k == 1 ? run<16>(N, PL, nops, draws, P, C)
                                                            : run<32>(N, PL, nops, draws, P, C))) return 3;
            if (P != P0 || memcmp(C.data(), C0.data(), C.size() * 4)) { printf("differs: %d draws, variant %d\n", draws, k); return 1; }
            ++checked;
        }
    }
    for (int v : P0) if (v < 1 || v > nops) return 4;
    printf("%d\n", checked);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("redraw")
    (d / "r.cu").write_text(_SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(_ROOT, "gpuropolis_gb300", "csrc"), "-I",
                    os.path.join(_ROOT, "include"), "-o", str(d / "r"), str(d / "r.cu")], check=True)
    return str(d / "r")


@pytest.mark.parametrize("PL,n_ops,draws", [
    # none, some and all of the 203 chains within the draws (an op takes 1 / (1 - 1 / n_ops), a constant 3.125)
    (63, 8, (32, 64, 256, 288, 352)), (63, 2, (128, 320, 352, 448)), (255, 2, (256, 1280, 1312, 1344)),
    (1, 8, (32,))])
def test_chains_that_need_more_draws(program, PL, n_ops, draws):
    out = subprocess.run([program, str(PL), str(n_ops), *map(str, draws)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert int(out.stdout) == 3 * len(draws)
