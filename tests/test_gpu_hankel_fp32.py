"""The plain FP32 Hankel GEMM (searay_gb300/csrc/hankel.cu) in each of its tile shapes, with radial grids and mode
counts off the tiles' edges.

* Load (q = Mfwd a) and the finish at z = 0 (A = Minv q) against FP64 products of the same inputs.  A sum of n
  products in FP32, the matrix rounded to FP32 before, is within (n + 2) 2^-24 sum |M_ik| |x_k| of the
  exact one (1 + O(n 2^-24) of it: under 1e-4 for the n here), per element; on azimuthal grids the DFT over
  N2 nodes adds N2 + 2 terms of that kind.
* One right-hand side against the FP64 oracle: 1e-5 of the maximum on bins >= 4, the bound of the other
  FP32 transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (N0, Nr, modes, N2): 16 x 64 tiles, then 64, 128 and 256 columns (152 multiprocessors)
SHAPES = [(17, 4, 3, 1), (33, 16, 13, 1), (65, 32, 31, 4), (257, 128, 101, 1), (4097, 64, 61, 1), (2049, 256, 243, 1),
          (2049, 512, 487, 1), (4097, 256, 256, 1)]


@pytest.fixture(scope="module", autouse=True)
def cuda_ready():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from searay_gb300 import build
    build.build()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_fp32_hankel(shape):
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
    dev = uppe.DeviceGrid(g, vd, None, "fp32")
    chi = vd["dispersion inside"].chi(g.w).astype(np.cdouble)
    mat = uppe.Material(dev, g, "cylindrical", None, chi, vd["chi3"], vd["density reference"], vd["window speed"],
                        vd["density lambda"])
    orc = O.Oracle(vd)
    mat.UpdateMaterial(0.0)
    orc.mat.update(0.0)
    rng = np.random.default_rng(n0 + nr)
    a = (rng.standard_normal((n0, nr, n2)) + 1j * rng.standard_normal((n0, nr, n2))).astype(np.complex64)
    a_dev = torch.from_numpy(a).cuda()
    dev.load_field(a_dev)
    q = dev.empty_field()
    dev.get_field(q)
    A = dev.empty_field()
    dev.finish_field(0.0, A)
    q, A = q.cpu().numpy(), A.cpu().numpy()
    H, lam = g.H, g.Lambda
    eps = 2.0 ** -24
    extra = 0 if n2 == 1 else n2 + 2
    for m in range(n2):
        fwd = H[:, :, m] * lam[None, :] / lam[:nk, None]
        inv = (H[:, :, m] * lam[:nk, None] / lam[None, :]).T
        x = np.fft.fft(a.astype(np.complex128), axis=2)[:, :, m]
        size = np.abs(a).sum(axis=2) if n2 > 1 else np.abs(x)
        bound = (nr + 2 + extra) * eps * 1.0001 * size @ np.abs(fwd).T
        assert np.all(np.abs(q[:, :nk, m] - x @ fwd.T) <= bound)
        assert np.all(q[:, nk:, m] == 0)
        if n2 == 1:
            y = q[:, :nk, 0].astype(np.complex128)
            bound = (nk + 2) * eps * 1.0001 * np.abs(y) @ np.abs(inv).T
            assert np.all(np.abs(A[:, :, 0] - y @ inv.T) <= bound)
    z = 0.5 * vd["size"][2] / 100
    wave = vd["incoming wave"](g.w, g.x1, g.x2)
    q_ref = orc.g.kspace(wave)
    q_dev = torch.from_numpy(q_ref.astype(np.complex64)).cuda()
    S_dev = dev.empty_field()
    dev.eval_rhs(q_dev, z, S_dev)
    S, ref = S_dev.cpu().numpy()[4:], orc.load_source(q_dev.cpu().numpy().astype(np.complex128), z)[4:]
    err = np.max(np.abs(S - ref)) / np.max(np.abs(ref))
    print(shape, f"rhs {err:.2e}")
    assert err < 1e-5
    dev.close()
