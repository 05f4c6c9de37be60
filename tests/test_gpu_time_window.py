"""The soft time window on the electron density (SoftTimeWindow, fft.cl:331-355) at cutoffs and widths other than the
reference's 4 and 64, through the configuration of the C ABI: ramps that just meet in the middle of the window, that
overlap by one sample to all of them, a width that is no power of two (the division instead of the product with the
reciprocal), and no window.  Register time passes (257, 513 and 1025 frequencies) and the shared-memory one (129).

J and the spectrum of the density of one uppe_finish against the FP64 oracle with the same window, on the field of
test_gpu_rates.py and within its bound, 5e-5 of the maximum: the window is a factor of at most 1 from exact sample numbers,
a few FP32 roundings.  A factor applied twice would show at the size of the window itself."""
import numpy as np
import pytest

from test_gpu_adjoint import cuda_ready  # noqa: F401 (the fixture builds the extension)

pytestmark = pytest.mark.gpu

# (n0, cutoff, width): M = n0 - 1 samples is half of the time axis
WINDOWS = [(257, 4, 252), (257, 4, 253), (257, 4, 256), (257, 2, 510), (257, 0, 512), (257, 100, 600), (257, 7, 49),
           (257, 0, 0), (513, 4, 512), (513, 0, 1024), (513, 5, 100), (1025, 4, 1024), (1025, 1, 1500), (1025, 3, 65),
           (129, 4, 128), (129, 5, 200)]


@pytest.mark.parametrize("n0,cutoff,width", WINDOWS)
def test_window(n0, cutoff, width, monkeypatch):
    import torch
    from oracle import uppe_oracle as O
    from searay_gb300 import _native, grid, ionization, uppe, workloads

    lib, window = _native.lib(), O.soft_time_window

    class Library:
        """The library with the window of every configuration replaced."""

        def uppe_create(self, cfg, out):
            cfg._obj.window_cutoff, cfg._obj.window_width = cutoff, width
            return lib.uppe_create(cfg, out)

        def __getattr__(self, name):
            return getattr(lib, name)

    monkeypatch.setattr(_native, "lib", Library)
    monkeypatch.setattr(O, "soft_time_window", lambda ne, *_: window(ne, cutoff, width))
    vd = workloads.cart_filament_128(steps=400)
    vd["wave grid"] = (n0, 16, 16, 2)
    g = grid.VolumeGrid(vd)
    dev = uppe.DeviceGrid(g, vd, ionization.RateCoefficients(vd["ionizer"]), "mixed")
    assert (dev.cfg.window_cutoff, dev.cfg.window_width) == (cutoff, width)
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cartesian", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    orc = O.Oracle(vd)
    mat.UpdateMaterial(0.0)
    orc.mat.update(0.0)
    T = 2 * np.pi / (g.w[1] - g.w[0])
    tau = T / 12
    amp = np.geomspace(0.02, 5.0, 256).reshape(16, 16)
    E0 = workloads.field_from_intensity(workloads.Units(0.8e-6 / (2 * np.pi)), 2e13)
    spec = np.exp(-(g.w - 1) ** 2 * tau ** 2 / 4 + 0.5j * g.w * T)
    spec *= E0 * g.Nt * tau * (g.w[1] - g.w[0]) / (4 * np.sqrt(np.pi))
    dev.load_field(torch.from_numpy((spec[:, None, None] * amp[None]).astype(np.complex64)).cuda())
    out = [dev.empty_field() for _ in range(4)]
    dev.finish(0.0, *out)
    A, J, _, ne = [x.cpu().numpy() for x in out]
    J_ref, _, ne_t, _ = orc.update_current(1j * orc.mat.kz * A.astype(np.complex128))
    ne_ref = np.fft.rfft(ne_t, axis=0)
    errs = [np.max(np.abs(x - r)) / max(np.max(np.abs(r)), 1e-30) for x, r in ((J, J_ref), (ne, ne_ref))]
    print(n0, cutoff, width, ["%.1e" % e for e in errs])
    assert max(errs) < 5e-5
    dev.close()
