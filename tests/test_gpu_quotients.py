"""The adjoint's quotients (gx_recip, gx_quotient, gpr_fastmath.cuh) are the
correctly rounded ones, bit for bit, wherever gx_in_range takes them: against
CUDA's __frcp_rn and __fdiv_rn on the device, for every mantissa of the
divisor, at both ends and in the middle of the exponent range.  Where a NaN
passes the range check the quotient is a NaN as well; zeros, infinities and
magnitudes beyond the range are not taken."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SOURCE = r"""
#include "gpr_fastmath.cuh"
#include <stdio.h>
#include <stdlib.h>
using namespace gpr;
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ unsigned mix(unsigned x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; return x ^ (x >> 16);
}
/* out: reciprocals wrong, quotients wrong, uncorrected products wrong, pairs */
__global__ void check(int eb, int ea, unsigned long long* out) {
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23; m += gridDim.x * blockDim.x)
        for (int j = 0; j < 64; ++j) {
            const unsigned r = mix(m * 64u + j);
            unsigned am = r & 0x7fffffu;
            if (j < 16) am = (m + j - 8u) & 0x7fffffu;
            else if (j < 20) am = j - 16;
            else if (j < 24) am = 0x7fffffu - (j - 20);
            const float b = __uint_as_float((unsigned)(eb + 127) << 23 | m | (r & 0x80000000u));
            const float a = __uint_as_float((unsigned)(ea + 127) << 23 | am | (j & 1 ? 0x80000000u : 0u));
            const float ab[2] = {a, b};
            if (!gx_in_range(ab)) continue;
            const float y = gx_recip(b), q = __fdiv_rn(a, b);
            if (!same(y, __frcp_rn(b))) atomicAdd(out, 1ull);
            if (!same(gx_quotient(a, b, y), q)) atomicAdd(out + 1, 1ull);
            if (!same(__fmul_rn(a, y), q)) atomicAdd(out + 2, 1ull);
            atomicAdd(out + 3, 1ull);
        }
}
__global__ void special(unsigned long long* out) {
    const float big = 1.152921504606847e18f, small = 8.673617379884035e-19f;
    const float bad[] = {0.0f, -0.0f, INFINITY, -INFINITY, 2 * big, small / 2, 1e-45f, 3e38f};
    const float good[] = {1.0f, -big, small};
    const float nan = __int_as_float(0x7fc00000);
    for (float g : good) {
        const float one[1] = {g};
        if (!gx_in_range(one)) out[0]++;
        for (float x : bad) {
            const float two[2] = {g, x};
            if (gx_in_range(two)) out[1]++;
        }
        if (!isnan(gx_quotient(nan, g, gx_recip(g))) || !isnan(gx_quotient(g, nan, gx_recip(nan)))) out[2]++;
    }
    const float n[1] = {nan};
    if (gx_in_range(n)) out[3]++;
}
int main(int argc, char** argv) {
    unsigned long long *d, h[4];
    if (cudaMalloc(&d, sizeof h) != cudaSuccess) return 2;
    cudaMemset(d, 0, sizeof h);
    if (argc > 2) check<<<608, 256>>>(atoi(argv[1]), atoi(argv[2]), d);
    else special<<<1, 1>>>(d);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("%llu %llu %llu %llu\n", h[0], h[1], h[2], h[3]);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(_SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(_ROOT, "gpuropolis_gb300", "csrc"), "-o", str(d / "q"),
                    str(d / "q.cu")], check=True)
    return str(d / "q")


def _run(program, *args):
    out = subprocess.run([program, *map(str, args)], check=True, capture_output=True, text=True).stdout
    return [int(v) for v in out.split()]


@pytest.mark.parametrize("eb", [-60, -1, 0, 1, 59])
@pytest.mark.parametrize("ea", [-60, 0, 59])
def test_quotients_are_correctly_rounded(program, eb, ea):
    recip, quotient, product, pairs = _run(program, eb, ea)
    assert pairs == 64 << 23
    assert recip == 0 and quotient == 0
    assert product > pairs // 10         # the comparison sees the last place


def test_range_and_special_values(program):
    assert _run(program) == [0, 0, 0, 0]
