"""Operand tiles that a step leaves for the next one on grids with azimuthal nodes (mixed precision form): the spectral
update writes the next inverse transform's, the azimuthal DFT the forward transform's (searay_gb300/csrc/uppe_kernels.cu,
k_spec_point; hankel.cu, k_azimuth_tiles).

Against SEARAY_UPPE_TC_NEXT=0, where every transform forms its operand itself: the same arithmetic on the same values, so
every output agrees bit for bit, over plain steps, adaptive steps, and with each entry point that makes the carried
tiles stale called between two steps."""
import numpy as np
import pytest

from test_gpu_adjoint import cuda_ready  # noqa: F401 (the fixture builds the extension)

pytestmark = pytest.mark.gpu

# (N0, Nr, modes, N2): one tile and several of radial nodes and of frequencies, all modes and some
SHAPES = [(33, 16, 12, 2), (65, 64, 64, 4), (129, 128, 100, 2), (257, 64, 50, 8)]
BETWEEN = ["nothing", "set_field", "load_field", "material", "chi3", "finish", "eval_rhs", "rotator"]


def run(shape, between, adaptive):
    import torch
    from searay_gb300 import grid, ionization, uppe, workloads
    n0, nr, nk, n2 = shape
    vd = workloads.cart_filament_128(steps=400)
    vd.update({"wave grid": (n0, nr, n2, 2), "wave coordinates": "cylindrical", "radial modes": nk,
               "density lambda": lambda x, y, z, r2: (1 + 1e-7 * z) * np.ones(x.shape)})
    g = grid.VolumeGrid(vd)
    dev = uppe.DeviceGrid(g, vd, ionization.RateCoefficients(vd["ionizer"]), "mixed")
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cylindrical", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    L = vd["size"][2] / 400
    mat.UpdateMaterial(0.5 * L)
    E0 = workloads.field_from_intensity(workloads.Units(0.8e-6 / (2 * np.pi)), 4e13)
    unit = workloads.Units(0.8e-6 / (2 * np.pi))
    wave = workloads.gaussian_pulse(E0, unit.fs(35.0), unit.mm(0.3), cylindrical=True)(g.w, g.x1, g.x2)
    phi = 2 * np.pi * np.arange(n2) / n2
    wave = wave * (1 + 0.2 * np.cos(phi) + 0.1j * np.sin(phi))[None, None, :]
    a = torch.from_numpy(wave.astype(np.complex64)).cuda()
    dzmin = L / 8 if adaptive else L
    fields = [dev.empty_field() for _ in range(4)]
    dev.load_field(a)
    z = dev.rk4_step(0.0, L, 0.0, dzmin)
    q = dev.empty_field()
    out = []
    for step in range(2):
        if between == "set_field":
            dev.get_field(q)
            dev.set_field((0.5 + 0.25j) * q)
        elif between == "load_field":
            dev.load_field(0.75 * a)
        elif between == "material":
            mat.UpdateMaterial((step + 2) * 1e4)
        elif between == "chi3":
            dev.set_chi3((0.5 + step) * vd["chi3"] / vd["density reference"])
        elif between == "finish":
            dev.finish(z, *fields)
            out += [f.cpu().numpy() for f in fields]
        elif between == "eval_rhs":
            dev.get_field(q)
            S = dev.empty_field()
            dev.eval_rhs(0.5 * q, 0.3 * L, S)
            out.append(S.cpu().numpy())
        elif between == "rotator":
            dev.set_rotator(workloads.n2_rotator(unit) if step == 0 else None)
        z += dev.rk4_step(z, L, 0.0, dzmin)
    dev.finish(z, *fields)
    dev.get_field(q)
    out += [f.cpu().numpy() for f in fields] + [q.cpu().numpy(), np.float64(z)]
    assert not dev.nonfinite()
    dev.close()
    return out


@pytest.mark.parametrize("adaptive", [False, True], ids=["fixed", "adaptive"])
@pytest.mark.parametrize("between", BETWEEN)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_carried_tiles(shape, between, adaptive, monkeypatch):
    monkeypatch.delenv("SEARAY_UPPE_TC_NEXT", raising=False)
    carried = run(shape, between, adaptive)
    monkeypatch.setenv("SEARAY_UPPE_TC_NEXT", "0")
    for x, y in zip(carried, run(shape, between, adaptive)):
        assert np.array_equal(x, y)
