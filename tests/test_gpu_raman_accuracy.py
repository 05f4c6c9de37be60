"""The rotational Raman response at one damping rate for all transitions is summed as at any others: by the recurrences of
raman_pass (searay_gb300/csrc/time_common.cuh), whose sum over time is compensated in the mixed form.

A transition whose population difference is below the smallest FP32 number adds exactly zero, whatever its damping.  So a
rotator whose dampings are all equal and one that differs from it in the damping of such a transition give the same current
and chi, bit for bit, in both precision forms and at every thread layout of the UPPE and envelope time passes."""
import numpy as np
import pytest

import cases
from test_gpu_adjoint import cuda_ready  # noqa: F401 (the fixture builds the extension)
from test_gpu_paraxial import _device
from test_gpu_raman import _setup, n2_rotator

pytestmark = pytest.mark.gpu

UPPE = [(17, 4, 4), (33, 16, 16), (65, 16, 16), (129, 16, 16), (257, 16, 16), (513, 16, 8), (1025, 4, 4), (2049, 8, 8),
        (4097, 4, 4)]
ENVELOPE = [(16, 64), (32, 64), (64, 512), (128, 64), (256, 256), (512, 64), (4096, 16), (8192, 16)]


def rotators():
    for damping in (1.0, 0.5):
        rot = n2_rotator()
        rot.dalpha *= 10
        rot.Tj[9] = 1e-60  # (0 would take the transition out of the tables)
        rot.Wj[9] = rot.Wj[9].real + 1j * damping * rot.Wj[9].imag
        yield rot


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("shape", UPPE, ids=lambda s: "x".join(map(str, s)))
def test_uppe(shape, precision):
    import torch
    from searay_gb300 import uppe
    vd, g, dev, mat = _setup(shape, None, ionize=False, precision=precision)
    a = torch.from_numpy(vd["incoming wave"](g.w, g.x1, g.x2).astype(np.complex64)).cuda()
    L = vd["size"][2] / 400
    out = []
    for rot in rotators():
        dev.set_rotator(rot)
        out.append([x.cpu().numpy() for x in uppe.propagator(dev, mat, a, 1, 0.0, L, L)[:3]])
    dev.close()
    for x, y in zip(*out):
        assert np.isfinite(x).all() and np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("shape", ENVELOPE, ids=lambda s: "x".join(map(str, s)))
def test_envelope(shape, precision):
    import torch
    from searay_gb300 import dispersion
    c = cases.PARAXIAL_CASES["par_cyl_raman"]
    vd = dict(c["keys"])
    vd.update({"wave grid": (shape[0], shape[1], 1, 2), "radial modes": shape[1], "ionizer": None, "precision": precision,
               "dispersion inside": dispersion.SimpleAir(cases.MKS_LENGTH),
               "density lambda": cases.density_lambda(c["density"]),
               "incoming wave": cases.make_wave(c["wave"], c["keys"]["size"][0]), "rotator": n2_rotator()})
    g, dev, mat, orc = _device(vd, precision)
    mat.UpdateMaterial(0.0)
    q = orc.g.kspace(np.fft.ifftshift(vd["incoming wave"](g.w, g.x1, g.x2), axes=0)).astype(np.complex64)
    q = torch.from_numpy(q).cuda()
    out = []
    for rot in rotators():
        dev.set_rotator(rot)
        S = dev.empty_field()
        dev.eval_rhs(q, 0.0, S)
        out.append(S.cpu().numpy())
    dev.close()
    assert np.isfinite(out[0]).all() and np.array_equal(*out)
