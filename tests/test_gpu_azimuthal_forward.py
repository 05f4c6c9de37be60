"""The forward transform of azimuthal grids in the mixed-precision form (searay_gb300/csrc/hankel.cu,
launch_spec_cyl): azimuthal DFT, tensor-core product stored over the current, then the elementwise spectral update.
The right-hand side and one RK4 step against the FP64 oracle within 1e-4 of the maximum, the bound of the split-BF16
transforms, with radial grids, mode counts and frequency counts off the tiles' edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (N0, Nr, modes, N2)
SHAPES = [(17, 4, 3, 2), (65, 32, 31, 4), (129, 128, 100, 2), (257, 64, 61, 8), (33, 16, 16, 16)]


@pytest.fixture(scope="module", autouse=True)
def cuda_ready():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from searay_gb300 import build
    build.build()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_azimuthal_forward(shape):
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
    mat.UpdateMaterial(0.0)
    orc.mat.update(0.0)
    z = 0.5 * vd["size"][2] / 100
    wave = vd["incoming wave"](g.w, g.x1, g.x2)
    phi = 2 * np.pi * np.arange(n2) / n2
    wave = wave * (1 + 0.2 * np.cos(phi) + 0.1j * np.sin(phi))[None, None, :]
    q_dev = torch.from_numpy(orc.g.kspace(wave).astype(np.complex64)).cuda()
    S_dev = dev.empty_field()
    dev.eval_rhs(q_dev, z, S_dev)
    S, ref = S_dev.cpu().numpy()[4:], orc.load_source(q_dev.cpu().numpy().astype(np.complex128), z)[4:]
    err = np.max(np.abs(S - ref)) / np.max(np.abs(ref))
    L = vd["size"][2] / 100
    A_ref = orc.propagator(wave, 0.0, L, 1, L)[0]
    A = uppe.propagator(dev, mat, torch.from_numpy(wave.astype(np.complex64)).cuda(), 1, 0.0, L, L)[0].cpu().numpy()
    step = np.max(np.abs(A - A_ref)) / np.max(np.abs(A_ref))
    print(shape, f"rhs {err:.2e} step {step:.2e}")
    assert err < 1e-4 and step < 1e-4
    dev.close()
