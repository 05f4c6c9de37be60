"""Cylindrical time passes on both sides of the rule that gives each of their blocks a multiprocessor of its own
(time_spread_smem, searay_gb300/csrc/timepass.cu): grids of at most as many blocks as multiprocessors ask for half of a
multiprocessor's shared memory, larger ones for what they need.  Register time pass (257 and 1025 frequencies), shared-memory
pass (65, 2049 and 4097) and its Raman forms, 1 to 256 blocks.

The right-hand side against the FP64 oracle within 1e-4 of the maximum, the bound of the split-BF16 Hankel transforms."""
import numpy as np
import pytest

from parity import rel_err
from test_gpu_adjoint import cuda_ready  # noqa: F401 (the fixture builds the extension)
from test_gpu_raman import n2_rotator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("medium", ["ionizing", "raman"])
@pytest.mark.parametrize("shape", [(65, 16), (257, 16), (257, 512), (1025, 512), (2049, 256), (2049, 512), (4097, 64)],
                         ids=lambda s: "x".join(map(str, s)))
def test_rhs(shape, medium):
    import torch
    from oracle import uppe_oracle as O
    from searay_gb300 import grid, ionization, uppe, workloads
    n0, nr = shape
    vd = workloads.cart_filament_128(steps=400)
    unit = workloads.Units(0.8e-6 / (2 * np.pi))
    E0 = workloads.field_from_intensity(unit, 3e13)
    vd.update({"wave grid": (n0, nr, 1, 2), "wave coordinates": "cylindrical", "radial modes": nr,
               "incoming wave": workloads.gaussian_pulse(E0, unit.fs(35.0), unit.mm(0.3), cylindrical=True),
               "rotator": n2_rotator() if medium == "raman" else None})
    if medium == "raman":
        vd["ionizer"] = None
    g = grid.VolumeGrid(vd)
    rates = ionization.RateCoefficients(vd["ionizer"]) if vd["ionizer"] is not None else None
    dev = uppe.DeviceGrid(g, vd, rates, "mixed")
    dev.set_rotator(vd["rotator"])
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cylindrical", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    orc = O.Oracle(vd)
    mat.UpdateMaterial(0.0)
    orc.mat.update(0.0)
    q = orc.g.kspace(vd["incoming wave"](g.w, g.x1, g.x2)).astype(np.complex64)
    S = dev.empty_field()
    dev.eval_rhs(torch.from_numpy(q).cuda(), 0.0, S)
    err = rel_err(S.cpu().numpy()[4:], orc.load_source(q.astype(np.complex128), 0.0)[4:])
    print(shape, medium, f"{err:.2e}")
    assert err < 1e-4
    dev.close()
