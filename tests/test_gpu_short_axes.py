"""The time pass and its vector-Jacobian product at the short time axes that have compile-time sizes (64 and 128 packed
samples, 16 transverse points per block): one RK4 step on a 16 x 16 Cartesian grid with the filamentation medium and an
ionizing pulse, against FP64 torch autograd of the same step.  Bound: the VJP tolerance of the FP32 transforms, 2e-4."""
import numpy as np
import pytest

from test_gpu_adjoint import cuda_ready, rel_err  # noqa: F401 (the fixture builds the extension)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n0", [65, 129])
def test_vjp_short_time_axes(n0):
    import torch
    from oracle import uppe_oracle as O
    from searay_gb300 import grid, ionization, uppe, workloads
    from torch_reference import TorchStep
    vd = workloads.cart_filament_128(steps=400, n_perp=16)
    vd["wave grid"] = (n0, 16, 16, 2)
    wave = vd["incoming wave"]
    vd["incoming wave"] = lambda w, x1, x2: 3.0 * wave(w, x1, x2)
    g = grid.VolumeGrid(vd)
    dev = uppe.DeviceGrid(g, vd, ionization.RateCoefficients(vd["ionizer"]), "mixed")
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cartesian", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    zmat = 100.0
    mat.UpdateMaterial(zmat)
    orc = O.Oracle(vd)
    orc.mat.update(zmat)
    redchi3 = vd["chi3"] / vd["density reference"]
    ts = TorchStep(orc)
    q0 = orc.g.kspace(vd["incoming wave"](g.w, g.x1, g.x2))
    rng = np.random.default_rng(11)
    lam = (rng.standard_normal(q0.shape) + 1j * rng.standard_normal(q0.shape)) * (np.abs(q0) + 1e-3 * np.abs(q0).max())
    z, dz = 50.0, vd["size"][2] / 400
    x = torch.tensor(q0.real, requires_grad=True)
    y = torch.tensor(q0.imag, requires_grad=True)
    c3 = torch.tensor(redchi3, dtype=torch.float64, requires_grad=True)
    q1 = ts.step(torch.complex(x, y), z, dz, c3)
    L = (torch.as_tensor(lam).conj() * q1).real.sum()
    L.backward()
    g_ref = x.grad.numpy() + 1j * y.grad.numpy()
    dred_ref = float(c3.grad)
    out = dev.empty_field()
    dred = dev.adjoint_step(torch.from_numpy(q0.astype(np.complex64)).cuda(),
                            torch.from_numpy(lam.astype(np.complex64)).cuda(), out, z, dz)
    e = rel_err(out.cpu().numpy(), g_ref)
    ed = abs(dred - dred_ref) / abs(dred_ref)
    print(n0, f"vjp {e:.2e} dchi3 {ed:.2e}")
    assert e < 2e-4 and ed < 2e-4
    dev.close()
