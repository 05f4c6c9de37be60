"""Radial grids with far fewer modes than nodes (the inverse transform's operand then has fewer 64-element tiles than
the forward transform's), mixed-precision form: two RK4 steps, whose stage estimates write the next inverse
transform's operand tiles, against the FP64 oracle within 1e-4 of the maximum, the bound of the split-BF16
transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (N0, Nr, modes, N2)
SHAPES = [(257, 128, 40, 1), (257, 256, 64, 1), (257, 256, 129, 1), (129, 128, 24, 4), (257, 128, 64, 2)]


@pytest.fixture(scope="module", autouse=True)
def cuda_ready():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from searay_gb300 import build
    build.build()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_few_modes(shape):
    import torch
    from oracle import uppe_oracle as O
    from searay_gb300 import grid, uppe, workloads
    n0, nr, nk, n2 = shape
    vd = workloads.cyl_kerr_64(100)
    vd["wave grid"] = (n0, nr, n2, 2)
    vd["radial modes"] = nk
    vd["frequency band"] = (0.0, 4.0)
    vd["nonlinear band"] = (0.0, 3.5)
    g = grid.VolumeGrid(vd)
    dev = uppe.DeviceGrid(g, vd, None, "mixed")
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cylindrical", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    orc = O.Oracle(vd)
    phi = 2 * np.pi * np.arange(n2) / n2
    wave = vd["incoming wave"](g.w, g.x1, g.x2) * (1 + 0.2 * np.cos(phi))[None, None, :]
    L = vd["size"][2] / 50
    A_ref = orc.propagator(wave, 0.0, L, 2, L / 2)[0]
    A = uppe.propagator(dev, mat, torch.from_numpy(wave.astype(np.complex64)).cuda(), 2, 0.0, L, L / 2)[0].cpu().numpy()
    err = np.max(np.abs(A - A_ref)) / np.max(np.abs(A_ref))
    print(shape, f"{err:.2e}")
    assert err < 1e-4
    dev.close()
