"""The ionizing path of the time passes (searay_gb300/csrc/time_common.cuh, timepass_reg.cu, timepass.cu) where its branch-free
forms change over: fields from far below the rate threshold to full ionization within one time window, the closed form and the
series, windows whose ramps (68 samples at each end) cover from a thirtieth of the samples to all of them.

One time pass of uppe_finish (J and the spectrum of the density) against the FP64 oracle on the same field.  The
rate is exp2 of a sum of size up to 150 in FP32, so its relative error is up to 150 ln 2 2^-23 < 1.3e-5
plus the hardware log2's; the density, bounded by the gas, follows with at most that relative error, and J with it:
5e-5 of the maximum for both."""
import pathlib
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda_ready():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from searay_gb300 import build
    build.build()


class Series:
    """A rate model without a closed form: its log is fitted."""

    def __init__(self, model):
        self.model = model

    def GetCoeff(self):
        return 0.0, 0.0, 0.0

    def Rate(self, E):
        return self.model.Rate(E)

    def get_mks_length(self):
        return self.model.get_mks_length()


@pytest.mark.parametrize("form", ["closed", "series"])
@pytest.mark.parametrize("n0", [33, 129, 257, 513, 1025, 2049])
def test_rates_and_density(n0, form):
    import torch
    from oracle import uppe_oracle as O
    from searay_gb300 import grid, ionization, uppe, workloads
    vd = workloads.cart_filament_128(steps=400)
    vd["wave grid"] = (n0, 16, 16, 2)
    if form == "series":
        vd["ionizer"] = Series(vd["ionizer"])
    g = grid.VolumeGrid(vd)
    dev = uppe.DeviceGrid(g, vd, ionization.RateCoefficients(vd["ionizer"]), "mixed")
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cartesian", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    orc = O.Oracle(vd)
    mat.UpdateMaterial(0.0)
    orc.mat.update(0.0)
    # a pulse a twelfth of the window long, its peak from 1/50 to 5 times the filament workload's across the slice
    T = 2 * np.pi / (g.w[1] - g.w[0])
    tau = T / 12
    amp = np.geomspace(0.02, 5.0, 256).reshape(16, 16)
    E0 = workloads.field_from_intensity(workloads.Units(0.8e-6 / (2 * np.pi)), 2e13)
    spec = np.exp(-(g.w - 1) ** 2 * tau ** 2 / 4 + 0.5j * g.w * T)
    spec *= E0 * g.Nt * tau * (g.w[1] - g.w[0]) / (4 * np.sqrt(np.pi))
    a = (spec[:, None, None] * amp[None]).astype(np.complex64)
    dev.load_field(torch.from_numpy(a).cuda())
    out = [dev.empty_field() for _ in range(4)]
    dev.finish(0.0, *out)
    A, J, _, ne = [x.cpu().numpy() for x in out]
    J_ref, _, ne_t, _ = orc.update_current(1j * orc.mat.kz * A.astype(np.complex128))
    ne_ref = np.fft.rfft(ne_t, axis=0)
    assert ne_t.max() > 0.05 * vd["density reference"] or n0 == 33  # (the window is 0 or a ramp over all of 64 samples)
    errs = [np.max(np.abs(x - r)) / np.max(np.abs(r)) for x, r in ((J, J_ref), (ne, ne_ref))]
    print(n0, form, ["%.1e" % e for e in errs])
    assert max(errs) < 5e-5
    dev.close()


RCP = r"""
#include <cstdio>
#include "time_common.cuh"
__global__ void check(unsigned long long* bad, unsigned e) {
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 23); m += gridDim.x * blockDim.x) {
        const float x = __uint_as_float((e << 23) | m);
        if (__float_as_uint(rcp_normal(x)) != __float_as_uint(__frcp_rn(x))) atomicAdd(bad, 1ull);
    }
}
int main() {
    unsigned long long *bad, host = 1;
    cudaMalloc(&bad, sizeof(host));
    cudaMemset(bad, 0, sizeof(host));
    for (unsigned e = 1; e <= 252; e += (e == 1 || e >= 250) ? 1 : 8) check<<<608, 256>>>(bad, e);
    if (cudaMemcpy(&host, bad, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%llu", host);
    return 0;
}
"""


def test_reciprocal_is_correctly_rounded(tmp_path):
    """rcp_normal against CUDA's __frcp_rn: every significand, exponents over the whole normal range it is for."""
    from searay_gb300 import build
    src, exe = tmp_path / "rcp.cu", tmp_path / "rcp"
    src.write_text(RCP)
    inc = pathlib.Path(build.__file__).resolve().parent
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", str(inc / "csrc"), "-o", str(exe), str(src)],
                   check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0"
