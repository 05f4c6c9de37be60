"""The ionization rate of the time passes (ion_rate_form, searay_gb300/csrc/time_common.cuh) at the ends of the FP32 range:
fields whose value in atomic units is zero, subnormal, near the largest number or infinite, with and without the zero below
em_min.  The branch-free reciprocal of the closed form gives there what the formula with CUDA's own reciprocal gives: the
same bits, or NaN where that is NaN."""
import pathlib
import subprocess

import pytest

from test_gpu_adjoint import cuda_ready  # noqa: F401 (the fixture builds the extension)

pytestmark = pytest.mark.gpu

PROBE = r"""
#include <cstdio>
#include <cmath>
#include "time_common.cuh"
__device__ float formula(const TimeParams& tp, float e) {
    const float em = fmaf(tp.fconv, fabsf(e), tp.cutoff);
    if (em < tp.em_min) return 0.f;
    return exp2f(fmaf(tp.ypow, __log2f(em), fmaf(tp.yexp, __frcp_rn(em), tp.y0)));
}
__global__ void check(TimeParams tp, const float* e, int n, unsigned* bad) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float x = formula(tp, e[i]), y = ion_rate_form<true>(tp, e[i]);
        if (!(x != x && y != y) && __float_as_uint(x) != __float_as_uint(y)) {
            printf("pow %g cutoff %g em_min %g: e = %g gives %g, formula %g\n", tp.ypow, tp.cutoff, tp.em_min, e[i], y, x);
            atomicAdd(bad, 1u);
        }
    }
}
int main() {
    float e[600];
    int n = 0;
    e[n++] = 0.f;
    e[n++] = INFINITY;
    e[n++] = 3.4028235e38f;
    for (int k = -149; k < 128; ++k) {
        e[n++] = ldexpf(1.f, k);
        e[n++] = -1.37f * ldexpf(1.f, k);
    }
    float* de;
    unsigned *bad, host = 1;
    cudaMalloc(&de, sizeof(e));
    cudaMalloc(&bad, sizeof(host));
    cudaMemcpy(de, e, sizeof(e), cudaMemcpyHostToDevice);
    cudaMemset(bad, 0, sizeof(host));
    for (float pow : {-1.09f, 0.f, 0.5f})
        for (float cutoff : {0.f, 1e-3f})
            for (float em_min : {0.f, 4e-3f}) {
                TimeParams tp{};
                tp.fconv = 2.f;
                tp.cutoff = cutoff;
                tp.em_min = em_min;
                tp.ypow = pow;
                tp.yexp = -1.1f;
                tp.y0 = 9.5f;
                check<<<1, 128>>>(tp, de, n, bad);
            }
    if (cudaMemcpy(&host, bad, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%u", host);
    return 0;
}
"""


def test_closed_form_at_the_ends_of_the_range(tmp_path):
    from searay_gb300 import build
    src, exe = tmp_path / "rate.cu", tmp_path / "rate"
    src.write_text(PROBE)
    inc = pathlib.Path(build.__file__).resolve().parent
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", str(inc / "csrc"), "-o", str(exe), str(src)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out == "0", out
