"""The fused slice passes in their two forms: the one for a real medium in the mixed precision form (one phasor for both
propagator factors where they are at the same z, no Im kz) and the general one (searay_gb300/csrc/slice_reg.cuh, slice_big.cu).

The same volume is stepped with a real medium and with one that absorbs in the last frequency bin only,
which selects the general form.  That bin lies above the nonlinear band and holds no field, so every
output agrees to rounding: both forms evaluate the same FP32 expressions, whose sums of four transforms
and stages differ by at most a few FP32 roundings, 1e-6 of the maximum."""
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


class LastBinAbsorbs:
    def __init__(self, medium):
        self.medium = medium

    def chi(self, w):
        chi = np.array(self.medium.chi(w), dtype=np.cdouble)
        chi[-1] += 1e-9j
        return chi


@pytest.mark.parametrize("adaptive", [False, True], ids=["fixed", "adaptive"])
@pytest.mark.parametrize("shape", [(65, 16, 16), (65, 16, 128), (129, 64, 32), (65, 128, 128), (33, 256, 128),
                                   (33, 128, 256), (33, 256, 256)],
                         ids=lambda s: "x".join(map(str, s)))
def test_real_and_general_medium(shape, adaptive):
    import torch
    from searay_gb300 import grid, ionization, uppe, workloads
    out = {}
    for form in ("real", "general"):
        vd = workloads.cart_filament_128(steps=400)
        vd["wave grid"] = shape + (2,)
        g = grid.VolumeGrid(vd)
        dev = uppe.DeviceGrid(g, vd, ionization.RateCoefficients(vd["ionizer"]), "mixed")
        medium = vd["dispersion inside"] if form == "real" else LastBinAbsorbs(vd["dispersion inside"])
        chi = np.asarray(medium.chi(g.w)).astype(np.cdouble)
        mat = uppe.Material(dev, g, "cartesian", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                            vd["density lambda"])
        wave = 2.0 * vd["incoming wave"](g.w, g.x1, g.x2)
        wave[-1] = 0.0
        L = vd["size"][2] / 400
        a = torch.from_numpy(wave.astype(np.complex64)).cuda()
        A, J, chi_w, ne, _ = uppe.propagator(dev, mat, a, 2, 0.0, 2 * L, 0.0 if adaptive else L)
        out[form] = [x.cpu().numpy() for x in (A, J, chi_w)]
        dev.close()
    for x, y in zip(out["general"], out["real"]):
        assert np.max(np.abs(x - y)) <= 1e-6 * np.max(np.abs(y))
