"""The two forms of the rotational Raman response in the time pass (searay_gb300/csrc/time_common.cuh): a convolution
where all transitions share one damping rate and the window is short against it, else the recurrences.  Rotators on
both sides of that rule, at time axes of every thread layout, against the FP64 oracle: chi and the current within 1e-5
of the maximum, the bound of FP32 transforms; with the polarizability difference raised ten-fold the Raman part is
most of chi."""
import numpy as np
import pytest

import cases
from parity import rel_err
from test_gpu_paraxial import _device
from test_gpu_raman import _setup, n2_rotator

pytestmark = pytest.mark.gpu

SHAPES = [(17, 4, 4), (65, 16, 16), (257, 16, 16), (513, 16, 8), (1025, 4, 4), (2049, 8, 8), (4097, 4, 4)]
KINDS = ["uniform", "undamped", "window_near_limit", "window_past_limit", "one_state_off"]


@pytest.fixture(scope="module", autouse=True)
def cuda_ready():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from searay_gb300 import build
    build.build()


def rotator(kind, window):
    """2 g T: 0.9 and 1.1 on the two sides of the limit of 1; one state off: two damping rates."""
    rot = n2_rotator()
    rot.dalpha *= 10
    j = np.arange(rot.Wj.shape[0]) >= 2
    g = rot.Wj[2].imag
    g = {"undamped": 0.0, "window_near_limit": 0.45 / window, "window_past_limit": 0.55 / window}.get(kind, g)
    rot.Wj = rot.Wj.real + 1j * np.where(j, g, 0.0)
    if kind == "one_state_off":
        rot.Wj[8] += 0.5j * g
    return rot


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_forms_match_oracle(shape, kind):
    import torch
    from oracle import uppe_oracle as O
    from searay_gb300 import uppe
    vd, g, dev, mat = _setup(shape, None, ionize=False)
    rot = rotator(kind, 2 * np.pi / (g.w[1] - g.w[0]))
    vd["rotator"] = rot
    dev.set_rotator(rot)
    L = vd["size"][2] / 400
    a = vd["incoming wave"](g.w, g.x1, g.x2)
    ref = O.Oracle(vd).propagator(a, 0.0, L, 1, L)
    out = uppe.propagator(dev, mat, torch.from_numpy(a.astype(np.complex64)).cuda(), 1, 0.0, L, L)
    errs = [rel_err(out[k].cpu().numpy(), ref[k]) for k in (0, 1, 2)]
    print(shape, kind, " ".join(f"{n} {e:.2e}" for n, e in zip(("A", "J", "chi"), errs)))
    assert max(errs) < 1e-5
    dev.close()


@pytest.mark.parametrize("kind", ["uniform", "one_state_off"])
@pytest.mark.parametrize("shape", [(64, 16), (64, 512), (256, 256), (512, 64), (4096, 16), (8192, 16)],
                         ids=lambda s: "x".join(map(str, s)))
def test_envelope_forms_match_oracle(shape, kind):
    import torch
    from searay_gb300 import dispersion
    c = cases.PARAXIAL_CASES["par_cyl_raman"]
    vd = dict(c["keys"])
    vd.update({"wave grid": (shape[0], shape[1], 1, 2), "radial modes": shape[1], "ionizer": None, "precision": "fp32",
               "dispersion inside": dispersion.SimpleAir(cases.MKS_LENGTH),
               "density lambda": cases.density_lambda(c["density"]),
               "incoming wave": cases.make_wave(c["wave"], c["keys"]["size"][0])})
    dw = (vd["frequency band"][1] - vd["frequency band"][0]) / shape[0]
    vd["rotator"] = rotator(kind, 2 * np.pi / dw)
    g, dev, mat, orc = _device(vd, "fp32")
    mat.UpdateMaterial(0.0)
    orc.mat.update(0.0)
    a = np.fft.ifftshift(vd["incoming wave"](g.w, g.x1, g.x2), axes=0)
    q = orc.g.kspace(a).astype(np.complex64)
    S = dev.empty_field()
    dev.eval_rhs(torch.from_numpy(q).cuda(), 0.0, S)
    err = rel_err(S.cpu().numpy(), orc.load_source(q.astype(np.complex128), 0.0))
    print(shape, kind, f"{err:.2e}")
    assert err < 2e-5
    dev.close()
