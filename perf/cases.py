"""Performance cases of the propagator: what a user has it compute, through its public entry points.

Three kinds of pass:

* ``wave``: one diagnostic interval of a volume, ``uppe.propagator`` or ``paraxial.propagator``: load
  the field, advance it through the subcycles (RK4, fixed or adaptive steps), give the field, the current
  and the spectra of the susceptibility and the electron density at its end;
* ``grad``: ``adjoint.propagate`` over a few fixed steps and its backward pass (the output field, the
  gradients with respect to the incoming field and to chi3);
* ``track``: the whole ``uppe.track`` call, host arrays in and out.

A case names a grid, a medium and a number of steps; the media and pulses are the analytic ones of
this repository's workloads (filaments in air, self-focusing in air, fused silica, rotating N2, the
N2 envelope), at other sizes too.  ``exact`` computes the same outputs in FP64 with plain torch.
"""
import math

import numpy as np
import torch

from searay_gb300 import adjoint, paraxial, uppe
from searay_gb300.grid import VolumeGrid
from searay_gb300.ionization import RateCoefficients
from searay_gb300.rotations import Rotator

# SI constants (CODATA 2022; c, e and hbar exact)
_C, _E, _HBAR = 299792458.0, 1.602176634e-19, 1.054571817646156e-34
_ME, _EPS0, _ALPHA = 9.1093837139e-31, 8.8541878188e-12, 7.2973525643e-3


# ---------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------
def _case(kind, medium, n0, n1, n2, steps, *, coords="cartesian", modes=0, precision="mixed", ion="none",
          adaptive=False, jet=False, planes=2, name=None):
    c = {"kind": kind, "medium": medium, "coords": coords, "n0": n0, "n1": n1, "n2": n2, "modes": modes,
         "steps": steps, "precision": precision, "ion": ion, "adaptive": adaptive, "jet": jet, "planes": planes}
    if name:
        c["name"] = name
    return c


def listed():
    cyl = "cylindrical"
    return [
        # self-focusing on the smallest radial grid that is used: a parameter scan's unit of work
        _case("wave", "air_kerr", 257, 64, 1, 30, coords=cyl, modes=64, name="radial_kerr_64"),
        # fused silica with ionization on a long time axis, default (mixed) form
        _case("wave", "silica", 2049, 512, 1, 10, coords=cyl, modes=512, ion="ppt", name="radial_silica_512"),
        # the same volume in plain FP32, with fewer modes than radial nodes: the form to check the default one against
        _case("wave", "silica", 2049, 512, 1, 4, coords=cyl, modes=487, ion="ppt", precision="fp32",
              name="radial_silica_512_fp32"),
        # rotational Raman in N2, real field
        _case("wave", "n2", 2049, 256, 1, 10, coords=cyl, modes=256, name="radial_raman_256"),
        # rotational Raman with the envelope solver, whose steps are always adaptive
        _case("wave", "n2_envelope", 256, 256, 1, 4, coords=cyl, modes=256, adaptive=True, name="envelope_raman_256"),
        # a gas jet on a radial grid with azimuthal modes: the medium changes at every subcycle
        _case("wave", "air", 257, 64, 8, 8, coords=cyl, modes=61, ion="adk", jet=True, name="azimuthal_jet_64x8"),
        # a small, oblong box with adaptive steps: exploratory runs
        _case("wave", "air", 129, 64, 32, 4, ion="ppt", adaptive=True, jet=True, name="box_adaptive_64x32"),
        # filamentation of a 5 critical power pulse
        _case("wave", "air", 513, 128, 128, 6, ion="ppt", name="filament_128"),
        # filamentation of a 10 critical power pulse, the largest grid in use
        _case("wave", "air", 1025, 256, 256, 2, ion="ppt", name="filament_256"),
        # pulse shaping: gradients through a radial Kerr volume
        _case("grad", "air_kerr", 1025, 256, 1, 4, coords=cyl, modes=256, name="gradient_radial_256"),
        # pulse shaping: gradients through a filament
        _case("grad", "air", 513, 128, 128, 2, ion="ppt", name="gradient_filament_128"),
        # a whole call, host arrays in and out, two planes after the first
        _case("track", "air", 257, 64, 64, 20, ion="ppt", planes=3, name="track_box_64"),
    ]


def draw(rng):
    def pow2(lo, hi):
        return 2 ** rng.randint(lo, hi)

    def steps_for(points, most):
        return max(1, min(most, int(6e7 / points)))

    kind = rng.choice(["box", "box", "radial", "radial", "silica", "raman", "envelope", "azimuthal", "gradient",
                       "track"])
    precision = rng.choice(["mixed", "mixed", "mixed", "fp32"])
    ion = rng.choice(["none", "ppt", "ppt", "adk", "series"])
    if kind == "box":
        n0 = pow2(5, 10) + 1
        n1, n2 = pow2(4, 8), pow2(4, 8)
        if n1 * n2 > 16384:
            n1, n2 = max(n1, 128), max(n2, 128)
        adaptive = rng.random() < 0.3
        return _case("wave", "air", n0, n1, n2, rng.randint(1, steps_for(n0 * n1 * n2, 6)), precision=precision,
                     ion=ion, adaptive=adaptive, jet=rng.random() < 0.3)
    nr = pow2(4, 9)
    modes = nr if rng.random() < 0.5 else rng.randint(nr // 2, nr)
    if kind == "radial":
        return _case("wave", "air", pow2(6, 12) + 1, nr, 1, rng.randint(1, 8), coords="cylindrical", modes=modes,
                     precision=precision, ion=ion, adaptive=rng.random() < 0.3, jet=rng.random() < 0.3)
    if kind == "silica":
        nr = pow2(6, 9)
        modes = nr if rng.random() < 0.5 else rng.randint(nr // 2, nr)
        return _case("wave", "silica", pow2(9, 12) + 1, nr, 1, rng.randint(1, 8), coords="cylindrical", modes=modes,
                     precision=precision, ion="ppt")
    if kind == "raman":
        return _case("wave", "n2", pow2(8, 12) + 1, nr, 1, rng.randint(1, 8), coords="cylindrical", modes=modes,
                     precision=precision)
    if kind == "envelope":
        return _case("wave", "n2_envelope", pow2(6, 9), nr, 1, rng.randint(1, 4), coords="cylindrical", modes=modes,
                     precision=precision, adaptive=True)
    if kind == "azimuthal":
        nr = pow2(4, 7)
        return _case("wave", "air", pow2(6, 9) + 1, nr, pow2(1, 3), rng.randint(1, 8), coords="cylindrical",
                     modes=rng.randint(nr // 2, nr), precision=precision, ion=ion, jet=rng.random() < 0.5)
    if kind == "gradient":
        if rng.random() < 0.5:
            return _case("grad", "air", pow2(6, 9) + 1, pow2(4, 7), pow2(4, 7), rng.randint(1, 2), precision=precision,
                         ion=rng.choice(["none", "ppt"]))
        return _case("grad", "air", pow2(7, 11) + 1, nr, 1, rng.randint(1, 4), coords="cylindrical", modes=modes,
                     precision=precision, ion=rng.choice(["none", "ppt"]))
    return _case("track", "air", pow2(6, 8) + 1, pow2(4, 6), pow2(4, 6), rng.randint(4, 20), precision=precision,
                 ion=ion, planes=rng.randint(2, 4))


# ---------------------------------------------------------------------------------------------
# Media and pulses
# ---------------------------------------------------------------------------------------------
class _Units:
    """Simulation units: lengths in lambda0 / (2 pi), so that the carrier has w = 1."""

    def __init__(self, lam):
        self.x1 = lam / (2 * math.pi)
        self.t1 = self.x1 / _C
        self.n1 = _EPS0 * _ME / self.t1 ** 2 / _E ** 2
        self.u1 = _ME * _C ** 2
        self.N1 = self.n1 * self.x1 ** 3

    def fs(self, v):
        return v * 1e-15 / self.t1

    def m(self, v):
        return v / self.x1

    def cm3(self, v):
        return v * 1e6 / self.n1

    def eV(self, v):
        return v * _E / self.u1

    def field(self, W_cm2):
        return math.sqrt(2 * W_cm2 * 1e4 * self.t1 * self.x1 ** 2 / self.N1 / self.u1)

    def chi3(self, n, n2):
        return 4 / 3 * n ** 2 * n2 * self.N1 * self.u1 / self.x1 ** 2 / self.t1


class _Sellmeier:
    """chi(w) = sum b / (c - (w / lambda0)^2), b and c in um^-2: two-term air, three-term fused silica."""

    def __init__(self, lam, b, c):
        self.b = [v * (lam * 1e6) ** 2 for v in b]
        self.c = [v * (lam * 1e6) ** 2 for v in c]

    def chi(self, w):
        return sum(b / (c - w * w) for b, c in zip(self.b, self.c)) + 0.0 * w

    def group_velocity(self):
        n2 = 1 + self.chi(1.0)
        d = sum(2 * b / (c - 1.0) ** 2 for b, c in zip(self.b, self.c))  # d chi / dw at w = 1
        return math.sqrt(n2) / (n2 + 0.5 * d)


def _air(lam):
    return _Sellmeier(lam, [2 * 0.05792105, 2 * 0.00167917], [238.0185, 57.362])


def _silica(lam):
    lines = [0.0684043, 0.1162414, 9.896161]  # Malitson
    return _Sellmeier(lam, [a / s ** 2 for a, s in zip([0.6961663, 0.4079426, 0.8974794], lines)],
                      [1 / s ** 2 for s in lines])


class _Rate:
    """Tunneling ionization rate pre E^pow exp(exp / E), E = |E| + 1e-3, in atomic units: the PPT limit or ADK
    for an s state, static form; ``series``: the closed form withheld, so that its log is fitted."""

    def __init__(self, form, lam, u_eV, Z):
        self.series = form == "series"
        self.mks = lam / (2 * math.pi)
        ua = _ME * _C ** 2 * _ALPHA ** 2
        U = u_eV * _E / ua
        ns = Z / math.sqrt(2 * U)
        if form == "adk":
            pre = math.sqrt(3 / math.pi ** 3) * (math.e / ns) ** 1.5 * Z ** 2 / ns ** 3
            pre *= (4 * math.e * Z ** 3 / ns ** 4) ** (2 * ns - 1.5)
        else:
            f0 = Z ** 3 / ns ** 3
            pre = U * 2 ** (2 * ns) / (ns * math.gamma(ns + 1) * math.gamma(ns)) * math.sqrt(6 / math.pi)
            pre *= (0.5 / f0) ** 1.5 * (2 * f0) ** (2 * ns)
        self.pre = pre * (2 * U) ** 0.75 / math.sqrt(3 / math.pi)
        self.pow = 1.0 - 2 * ns
        self.exp = -2 * Z ** 3 / (3 * ns ** 3)

    def get_mks_length(self):
        return self.mks

    def GetCoeff(self):
        return (0.0, 0.0, 0.0) if self.series else (self.pre, self.pow, self.exp)

    def Rate(self, E):
        E = np.abs(E) + 1e-3
        return self.pre * E ** self.pow * np.exp(self.exp / E)


def _setup(case):
    """The volume's numbers, plain values only: grid, medium, pulse (peak field, duration, radius)."""
    m, n0 = case["medium"], case["n0"]
    lam = 1e-6 if m == "silica" else 0.8e-6
    u = _Units(lam)
    disp = _silica(lam) if m == "silica" else _air(lam)
    s = {"u": u, "disp": disp, "vg": disp.group_velocity(), "ion": None, "rot": False, "rel": 1.0}
    if m == "silica":
        n = math.sqrt(1 + disp.chi(1.0))
        s.update(band=(0.0, 4.0), nl=(0.3, 3.5), box=u.m(2e-3), dz=u.m(0.2e-6), chi3=u.chi3(n, 2.5e-20),
                 nref=u.cm3(2.2e22), E0=u.field(1e13) / math.sqrt(n), tau=u.fs(100.0), r0=u.m(60e-6),
                 ion=(9.0, 1.0))
    elif m in ("n2", "n2_envelope"):
        s.update(band=(0.0, 8.0), nl=(0.0, 4.0), box=u.m(2e-3), dz=u.m(0.441e-4), chi3=u.chi3(1.0, 14.8e-24),
                 nref=u.cm3(2.7e19), rel=90.0 / 760.0, rot=True, E0=u.field(4.5e13),
                 tau=u.fs(40.0) / math.sqrt(2 * math.log(2)), r0=u.m(150e-6))
        if m == "n2_envelope":
            s.update(band=(0.5, 1.5), nl=None)
    elif m == "air_kerr":
        W = 2 * math.pi * n0 / u.fs(400.0) if n0 <= 257 else 2 * math.pi * n0 / u.fs(400.0) * (n0 - 1) / n0 * 257 / 256
        s.update(band=(0.0, W), nl=(0.0, W), box=u.m(2e-3), dz=u.m(1e-3) if n0 <= 257 else u.m(0.5e-3),
                 chi3=u.chi3(1.0, 3e-23), nref=1.0, E0=u.field(1e13), tau=u.fs(50.0), r0=u.m(200e-6))
    else:
        big = max(case["n1"], case["n2"]) > 128
        n2 = 3e-23
        pcr = 3.77 * lam ** 2 / (8 * math.pi * n2)
        I0 = 2 * (10 if big else 5) * pcr / (math.pi * 0.15e-3 ** 2) * 1e-4  # half-way into the collapse
        s.update(band=(0.0, 4.0), nl=(0.0, 3.5), box=u.m(3e-3 if big else 2e-3), dz=u.m(1e-4 if big else 2.5e-4),
                 chi3=u.chi3(1.0, n2), nref=u.cm3(5.4e18), E0=u.field(I0), tau=u.fs(40.0 if big else 35.0),
                 r0=u.m(0.15e-3), ion=(12.07, 0.53))
    # short time windows hold shorter pulses
    window = 2 * math.pi * (n0 if m == "n2_envelope" else n0 - 1) / (s["band"][1] - s["band"][0])
    s["tau"] = min(s["tau"], window / 8)
    s["L"] = case["steps"] * (case["planes"] - 1) * s["dz"]
    s["envelope"] = m == "n2_envelope"
    return s


def _density(case, s):
    """Relative density (x, y, z, r2): uniform, or a jet that varies along z and across the beam."""
    rel, L, r0 = s["rel"], s["L"], s["r0"]
    if not case["jet"]:
        return lambda x, y, z, r2: rel * np.ones(x.shape)
    return lambda x, y, z, r2: rel * (0.7 + 0.3 * np.cos(math.pi * z / L)) * (0.8 + 0.2 * np.exp(-r2 / (9 * r0 ** 2)))


def _volume(case, s):
    vd = {"wave grid": (case["n0"], case["n1"], case["n2"], case["planes"]), "wave coordinates": case["coords"],
          "frequency band": s["band"], "size": (s["box"], s["box"], s["L"]), "subcycles": case["steps"],
          "minimum step": 0.0 if case["adaptive"] else s["dz"], "chi3": s["chi3"], "density reference": s["nref"],
          "window speed": s["vg"], "dispersion inside": s["disp"], "ionizer": None,
          "density lambda": _density(case, s), "precision": case["precision"]}
    if s["nl"] is not None:
        vd["nonlinear band"] = s["nl"]
    if case["coords"] == "cylindrical":
        vd["radial modes"] = case["modes"]
    if case["ion"] != "none" and s["ion"] is not None:
        vd["ionizer"] = _Rate(case["ion"], s["u"].x1 * 2 * math.pi, *s["ion"])
    if s["rot"]:
        vd["rotator"] = Rotator(*_rotor(s["u"]))
    return vd


def _rotor(u):
    """N2: rotational constant, polarizability difference, kT, nuclear degeneracies, dampings, hbar."""
    j = np.arange(32)
    return (2.0 / u.m(1e-2), 4 * math.pi * 6.7e-25 / u.cm3(1.0), u.eV(0.025), 6 - 3 * (j % 2), np.ones(32) / u.fs(1e5),
            _HBAR / u.t1 / u.u1)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _axes(case, s):
    n0, n1, n2 = case["n0"], case["n1"], case["n2"]
    lo, hi = s["band"]
    c, wd = 0.5 * (lo + hi), hi - lo
    w = c + np.linspace(-wd / 2, wd / 2 - wd / n0, n0)
    if case["coords"] == "cartesian":
        x1, x2 = [-s["box"] / 2 + s["box"] / n * (np.arange(n) + 0.5) for n in (n1, n2)]
    else:
        x1 = s["box"] / 2 / n1 * (np.arange(n1) + 0.5)
        x2 = np.array([0.0]) if n2 == 1 else np.linspace(-math.pi, math.pi - 2 * math.pi / n2, n2)
    return w, x1, x2


def _field(case, s, seed):
    """The incoming plane (complex64, on the device): a Gaussian pulse with seeded energy, delay, chirp and
    transverse phase (8 weak gratings; rings and azimuthal lobes on radial grids)."""
    rng = np.random.default_rng(seed)
    w, x1, x2 = _axes(case, s)
    n0, tau, r0 = case["n0"], s["tau"], s["r0"]
    dwn, dw = w[1] - w[0], 2.0 / tau
    energy, delay, chirp = 1 + 0.1 * rng.uniform(-1, 1), rng.uniform(-0.02, 0.02), rng.uniform(-0.2, 0.2)
    E0 = s["E0"] * math.sqrt(energy)
    if s["envelope"]:
        amp = E0 * n0 * dwn / (math.sqrt(math.pi) * dw)
        ph = -(w - w[n0 // 2]) * math.pi / dwn * (1 + delay)
    else:
        amp = E0 * (2 * n0 - 2) / (2.0 * math.sqrt(math.pi) * (dw / dwn))
        ph = w * math.pi / dwn * (1 + delay)
    spec = amp * np.exp(-(w - 1) ** 2 / dw ** 2 + 1j * (ph + chirp * (w - 1) ** 2 / dw ** 2))
    a, b, p = rng.uniform(-3, 3, 8), rng.uniform(-3, 3, 8), rng.uniform(0, 2 * math.pi, 8)
    if case["coords"] == "cartesian":
        r2 = x1[:, None] ** 2 + x2[None, :] ** 2
        arg = [2 * math.pi / s["box"] * (a[i] * x1[:, None] + b[i] * x2[None, :]) for i in range(8)]
    else:
        r2 = x1[:, None] ** 2 + 0 * x2[None, :]
        lobes = min(1.0, 0.25 * case["n2"] - 0.25)
        arg = [2 * math.pi / s["box"] * a[i] * x1[:, None] + lobes * np.cos(x2[None, :] + b[i]) for i in range(8)]
    screen = 0.05 * sum(np.cos(v + q) for v, q in zip(arg, p))
    tr = np.exp(-r2 / r0 ** 2 + 1j * screen)
    dev = _device()
    spec = torch.from_numpy(spec).to(dev).to(torch.complex64)
    tr = torch.from_numpy(tr).to(dev).to(torch.complex64)
    return (spec[:, None, None] * tr[None]).contiguous()


def _cotangent(case, seed):
    """The gradient of a loss on the output field around the pulse's place in the time window: a band of w,
    uneven across the beam."""
    g = torch.Generator(device="cpu").manual_seed(seed + 1)
    tr = (1.0 + 0.5 * torch.randn(case["n1"], case["n2"], 2, generator=g)).to(_device())
    lo, hi = _setup(case)["band"]
    w = lo + (hi - lo) / case["n0"] * torch.arange(case["n0"], device=_device(), dtype=torch.float32)
    k = torch.arange(case["n0"], device=_device())
    env = torch.exp(-((w - 1.0) / 0.2) ** 2) * (1 - 2 * (k % 2))
    return (env[:, None, None] * torch.view_as_complex(tr)[None]).contiguous()


# ---------------------------------------------------------------------------------------------
# The passes
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    s = _setup(case)
    vd = _volume(case, s)
    a = _field(case, s, seed)
    if case["kind"] == "track":
        plane = a.cpu().numpy().astype(np.complex128)
        vd["incoming wave"] = lambda w, x1, x2: plane
        return {"kind": "track", "volume": vd}
    grid = VolumeGrid(vd)
    rates = RateCoefficients(vd["ionizer"]) if vd["ionizer"] is not None else None
    dev = uppe.DeviceGrid(grid, vd, rates, vd["precision"], envelope=s["envelope"])
    dev.set_rotator(vd.get("rotator"))
    chi = np.asarray(s["disp"].chi(grid.w)).astype(np.cdouble)
    st = {"kind": case["kind"], "case": case, "dev": dev, "a": a, "zi": -0.5 * s["L"], "zf": 0.5 * s["L"],
          "dzmin": vd["minimum step"], "envelope": s["envelope"], "dz": s["dz"]}
    if s["envelope"]:
        st["a"] = torch.fft.ifftshift(a, dim=0).contiguous()
        st["mat"] = paraxial.Material(dev, grid, case["coords"], None, chi, s["chi3"], s["nref"],
                                      grid.w[case["n0"] // 2], 1 / s["vg"], 1 / s["vg"], vd["density lambda"])
    else:
        st["mat"] = uppe.Material(dev, grid, case["coords"], None, chi, s["chi3"], s["nref"], s["vg"],
                                  vd["density lambda"])
    if case["kind"] == "grad":
        st["mat"].UpdateMaterial(0.0)
        st["a"].requires_grad_(True)
        st["chi3"] = torch.tensor(s["chi3"] / s["nref"], dtype=torch.float64, requires_grad=True)
        st["g"] = _cotangent(case, seed)
    return st


def run(state):
    if state["kind"] == "track":
        A, J, chi, ne, dom = uppe.track(None, None, None, None, state["volume"])
        return {"A": A, "J": J, "chi": chi, "ne": ne, "domain": dom}
    dev, n = state["dev"], state["case"]["steps"]
    if state["kind"] == "grad":
        A = adjoint.propagate(dev, state["a"], state["chi3"], state["dz"], n)
        ga, gc = torch.autograd.grad(A, (state["a"], state["chi3"]), grad_outputs=state["g"])
        return {"A": A.detach(), "grad_a": ga, "grad_chi3": gc}
    if state["envelope"]:
        A, J, chi, ne, evals = paraxial.propagator(dev, state["mat"], state["a"], n, state["zi"], state["zf"])
    else:
        A, J, chi, ne, evals = uppe.propagator(dev, state["mat"], state["a"], n, state["zi"], state["zf"],
                                               state["dzmin"])
    return {"A": A, "J": J, "chi": chi, "ne": ne, "evaluations": evals}


def work(case):
    """A right-hand-side evaluation crosses the time axis and the transverse axes; each crossing reads its input and
    writes its output once (16 B a point along t; current, operator, two RK states in, one RK state and the next
    field out across the beam: 44 B).  A pass adds its load and its outputs.  The reverse of a step costs
    its four evaluations again and twice their transposes.  Flops: 5 N log2 N a complex transform, 8 a
    complex multiplication, real-matrix Hankel products at 4 a term."""
    n0, n1, n2 = case["n0"], case["n1"], case["n2"]
    P, S = n0 * n1 * n2, n1 * n2
    evals = 4 * case["steps"] * (case["planes"] - 1)
    nt = n0 if case["medium"] == "n2_envelope" else 2 * n0
    transforms = 3 if case["ion"] != "none" else 2
    t_fl = S * transforms * 2.5 * nt * math.log2(nt) * (2 if case["medium"] == "n2_envelope" else 1) + 20 * S * nt
    if case["medium"].startswith("n2"):
        t_fl += S * nt * 30 * 16
    if case["coords"] == "cartesian":
        x_fl = 2 * 5 * P * math.log2(S)
    else:
        x_fl = 4 * P * (n1 + case["modes"]) + (2 * 5 * P * math.log2(n2) if n2 > 1 else 0)
    ev_by, ev_fl = 60 * P, t_fl + x_fl + 60 * P
    if case["kind"] == "grad":
        return {"bytes": int(evals * ev_by * 3 + 8 * 8 * P), "flops": int(evals * ev_fl * 3.5)}
    ends = (case["planes"] - 1) * (16 + 8 + 32)
    if case["kind"] == "track":
        ends += 5 * 16 * case["planes"]
    return {"bytes": int(evals * ev_by + ends * P), "flops": int((evals + 2 * (case["planes"] - 1)) * ev_fl)}


# ---------------------------------------------------------------------------------------------
# The same in FP64, plain torch
# ---------------------------------------------------------------------------------------------
class _Exact:
    def __init__(self, case, s):
        dev = self.dev = _device()
        self.case, self.s = case, s
        n0, n1, n2 = self.N = (case["n0"], case["n1"], case["n2"])
        w, x1, x2 = _axes(case, s)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        self.cart = case["coords"] == "cartesian"
        self.env = s["envelope"]
        self.wn = np.fft.ifftshift(w) if self.env else w
        if self.cart:
            k2 = [(2 - 2 * np.cos(2 * math.pi * np.arange(n) / n)) * (n / s["box"]) ** 2 for n in (n1, n2)]
            self.kr2 = t(k2[0][:, None] + k2[1][None, :])
            self.xy = (x1[:, None] + 0 * x2[None, :], x2[None, :] + 0 * x1[:, None])
        else:
            self._hankel(n1, n2, case["modes"], s["box"] / 2 / n1)
            self.xy = (np.outer(x1, np.cos(x2)), np.outer(x1, np.sin(x2)))
        self.w = t(self.wn)[:, None, None]
        dw = w[1] - w[0]
        if self.env:
            self.dt = 2 * math.pi / ((w[-1] - w[0]) * (1 + 1 / (n0 - 1)))
            self.nt = n0
        else:
            self.dt = math.pi / w[-1]
            self.nt = 2 * n0 - 2
            k = np.arange(n0)
            self.keep = t(((k >= int(s["nl"][0] / dw)) & (k < int(s["nl"][1] / dw))).astype(float))[:, None, None]
            self.cond = t((k >= 4).astype(float))[:, None, None]
            self.window = t(self._window(self.nt))[:, None, None]
        self.chi = np.asarray(s["disp"].chi(self.wn))
        self.red = s["chi3"] / s["nref"]
        self.rate = None
        if case["ion"] != "none" and s["ion"] is not None:
            self._rates(_Rate(case["ion"], s["u"].x1 * 2 * math.pi, *s["ion"]))
        self.raman = self._raman_tables() if s["rot"] else None

    def _hankel(self, nr, nm, nk, dr):
        r = dr * (np.arange(nr) + 0.5)
        inner, outer = 2 * math.pi * (r - dr / 2), 2 * math.pi * (r + dr / 2)
        vol = math.pi * ((r + dr / 2) ** 2 - (r - dr / 2) ** 2)
        lam = np.sqrt(vol)
        H, kr2 = np.zeros((nk, nr, nm)), np.zeros((nr, nm))
        for m in range(nm // 2 + 1):
            d = -(inner + outer) / (dr * vol) - (m / r) ** 2
            d[0] += inner[0] / (dr * vol[0])
            d[-1] -= outer[-1] / (dr * vol[-1])
            up = outer[:-1] / (dr * vol[:-1]) * lam[:-1] / lam[1:]
            val, vec = np.linalg.eigh(np.diag(d) + np.diag(up, 1) + np.diag(up, -1))
            for mm in {m % nm, -m % nm}:
                kr2[:nk, mm] = -val[nr - nk:]
                H[:, :, mm] = vec[:, nr - nk:].T
        dev = self.dev
        self.H, self.kr2 = torch.as_tensor(H, device=dev).to(torch.complex128), torch.as_tensor(kr2, device=dev)
        self.lam = torch.as_tensor(lam, device=dev)[None, :, None]

    @staticmethod
    def _window(n):
        i = np.arange(n)
        d = np.minimum(i, n - 1 - i) - 4
        q = np.clip(d / 64, 0, 1)
        f = 10 * q ** 3 - 15 * q ** 4 + 6 * q ** 5
        if n < 2 * 68:  # both ramps act on every sample they reach
            ramp = lambda e: np.where(e < 64, np.where(e >= 0, (e / 64) ** 3 * (10 - 15 * (e / 64) + 6 * (e / 64) ** 2),
                                                       0.0), 1.0)
            f = ramp(i - 4.0) * ramp(n - 5.0 - i)
        return f

    def _rates(self, model):
        xs = model.get_mks_length()
        ta = _HBAR / (_ME * _C ** 2 * _ALPHA ** 2)
        ea = _ME * _C ** 2 * _ALPHA ** 2 / (_HBAR / (_ME * _C * _ALPHA)) / _E
        conv, rconv = _ME * _C ** 2 / xs / _E / ea, xs / _C / ta
        if model.series:
            E = np.logspace(np.log10(2e-3), 0, 256)
            p = np.polynomial.Polynomial.fit(np.log(E), np.log(model.Rate(E)), 5).convert().coef
            self.rate = lambda e: rconv * torch.exp(sum(float(c) * torch.log(conv * e + 1e-3) ** i for i, c in enumerate(p)))
        else:
            def closed(e):
                em = conv * e + 1e-3
                return rconv * model.pre * em ** model.pow * torch.exp(model.exp / em)
            self.rate = closed

    def _raman_tables(self):
        B, da, kT, dnuc, damp, hbar = _rotor(self.s["u"])
        j = np.arange(len(dnuc))
        wj = 2 * math.pi * B * j * (j + 1)
        X = dnuc * np.exp(-hbar * wj / kT)
        rho = X / np.sum((2 * j + 1) * X)
        return [(complex(wj[i] - wj[i - 2], damp[i]), rho[i] - rho[i - 2], 2.0 * i * (i - 1) / (15 * (2 * i - 1)))
                for i in range(2, len(dnuc))], da, hbar

    def medium(self, z):
        x, y = self.xy
        dens = _density(self.case, self.s)(x, y, np.full(x.shape, z), x * x + y * y)
        chi0 = self.chi * np.where(self.chi > 0, dens.min(), np.where(self.chi < 0, dens.max(), 1.0))
        w = self.wn
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)
        self.ng = t(self.s["nref"] * np.broadcast_to(dens, self.N[1:]).astype(float))[None]
        if self.env:
            ng = 1 / self.s["vg"]
            k0 = w * ng
            self.div = t(k0)[:, None, None]
            self.K = 0.5 * (t(w ** 2 * (1 + chi0 - ng ** 2))[:, None, None] - self.kr2[None]) / self.div
            return
        arg = t(w ** 2 * (1 + chi0))[:, None, None] - self.kr2[None]
        self.kz = torch.where(arg > 0, torch.sqrt(arg.clamp(min=0)), torch.ones_like(arg))
        self.div = self.kz
        self.K = self.kz - self.w / self.s["vg"]

    def kspace(self, a):
        if self.cart:
            return torch.fft.fft2(a, dim=(1, 2))
        b = torch.fft.fft(a, dim=2) * self.lam
        out = torch.einsum("ijm,fjm->fim", self.H, b)
        pad = torch.zeros(b.shape[0], b.shape[1] - out.shape[1], b.shape[2], dtype=b.dtype, device=b.device)
        return torch.cat([out, pad], dim=1) / self.lam

    def rspace(self, a):
        if self.cart:
            return torch.fft.ifft2(a, dim=(1, 2))
        out = torch.einsum("jim,fjm->fim", self.H, (a * self.lam)[:, :self.H.shape[0]]) / self.lam
        return torch.fft.ifft(out, dim=2)

    def density(self, e):
        r = self.rate(e)
        r = torch.cat([r[:-1], torch.zeros_like(r[-1:])], dim=0)
        S = torch.flip(torch.cumsum(torch.flip(0.5 * (r[:-1] + r[1:]) * self.dt, [0]), dim=0), [0])
        return self.ng * -torch.expm1(-torch.cat([S, torch.zeros_like(S[-1:])], dim=0))

    def raman_chi(self, I):
        """Rotational response to the mean square field I (t, x, y): the density-matrix sums, backwards in t."""
        lines, da, hbar = self.raman
        F = torch.flip(0.5 * da / hbar * I, [0])
        n = torch.arange(self.nt, dtype=torch.float64, device=self.dev)[:, None, None]
        chi = 0
        for W, T, S in lines:
            if T == 0.0:
                continue
            a = F * torch.exp(1j * W * self.dt * (n + 0.5))
            rho = -1j * self.dt * (torch.cumsum(a, dim=0) - a)
            term = T * S * W * self.dt * rho * torch.conj(torch.exp(1j * W * self.dt * n))
            chi = chi + 2 * da * torch.cumsum(term.imag, dim=0)
        return torch.flip(chi, [0]) * self.ng

    def current(self, f):
        """J, chi(t), ne(t) from the spectral field E (the envelope solver: from A)."""
        if self.env:
            E, A = torch.fft.ifft(1j * self.w * f, dim=0), torch.fft.ifft(f, dim=0)
            I = E.real ** 2 + E.imag ** 2
            ne = self.density(torch.sqrt(I)) if self.rate else torch.zeros_like(I)
            chi = 0.75 * self.ng * self.red * I + (self.raman_chi(0.5 * I) if self.raman else 0)
            J = -1j * self.w * torch.fft.fft(chi * E, dim=0)
            return J + torch.fft.fft(ne * (0.25 * (A.real ** 2 + A.imag ** 2) - 1) * A, dim=0), chi, ne
        E = torch.fft.irfft(f, n=self.nt, dim=0)
        chi = self.ng * self.red * E * E + (self.raman_chi(E * E) if self.raman else 0)
        J = -1j * self.w * torch.fft.rfft(chi * E, dim=0)
        ne = torch.zeros_like(E)
        if self.rate:
            ne = self.density(torch.abs(E)) * self.window
            J = J + torch.fft.rfft(ne * E, dim=0) / (0.1 - 1j * self.w)
        return J * self.keep, chi, ne

    def real_field(self, q, z):
        return self.rspace(torch.exp(1j * self.K * z) * q)

    def rhs(self, q, z):
        ph = torch.exp(1j * self.K * z)
        J = self.current(self.rspace(ph * q if self.env else 1j * self.kz * ph * q))[0]
        return 0.5j * torch.conj(ph) * self.kspace(J) / self.div

    def step(self, q, z, dz):
        """One RK4 step; dz: the step, or a function of q and its slope."""
        c = 1.0 if self.env else self.cond
        k = self.rhs(q, z)
        h = dz(q, k) if callable(dz) else dz
        qf = q + h / 6 * k
        k = self.rhs((q + h / 2 * k) * c, z + h / 2)
        qf = qf + h / 3 * k
        k = self.rhs((q + h / 2 * k) * c, z + h / 2)
        qf = qf + h / 3 * k
        k = self.rhs((q + h * k) * c, z + h)
        return (qf + h / 6 * k) * c, h

    def interval(self, a, zi, zf):
        case = self.case
        n = case["steps"]
        L = (zf - zi) / n
        q, evals = self.kspace(a), 0
        for i in range(n):
            self.medium(zi + (i + 0.5) * L)
            z = 0.0

            def size(q, k):
                if not case["adaptive"]:
                    return L - z
                den = q.abs() ** 2 + (1e-2 * q.abs().max()) ** 2
                p = torch.conj(q) * k / den
                d = float(torch.min(0.4 / (0.2 / L + p.imag.abs() - p.real.clamp(max=0))))
                return min(d, L - z)
            while z < L and (z - L) ** 2 > (L / 1e6) ** 2:
                q, h = self.step(q, i * L + z, size)
                z += h
                evals += 4
        A = self.real_field(q, zf - zi)
        J, chi, ne = self.current(A if self.env else 1j * self.kz * A)
        rf = torch.fft.fft if self.env else torch.fft.rfft
        return A, J, rf(chi, dim=0), rf(ne, dim=0), evals


def exact(case, seed):
    s = _setup(case)
    x = _Exact(case, s)
    a = _field(case, s, seed).to(torch.complex128)
    if s["envelope"]:
        a = torch.fft.ifftshift(a, dim=0)
    zi, zf = -0.5 * s["L"], 0.5 * s["L"]
    if case["kind"] == "grad":
        x.medium(0.0)
        a.requires_grad_(True)
        chi3 = torch.tensor(s["chi3"] / s["nref"], dtype=torch.float64, device=a.device, requires_grad=True)
        x.red = chi3
        q = x.kspace(a)
        for i in range(case["steps"]):
            q, _ = x.step(q, i * s["dz"], s["dz"])
        A = x.real_field(q, case["steps"] * s["dz"])
        ga, gc = torch.autograd.grad(A, (a, chi3), grad_outputs=_cotangent(case, seed).to(torch.complex128))
        return {"A": A.detach(), "grad_a": ga, "grad_chi3": gc}
    with torch.no_grad():
        if case["kind"] == "track":
            walls = np.linspace(zi, zf, case["planes"])
            zero = torch.zeros_like(a)
            out = [[a], [zero], [zero], [zero]]
            for k in range(case["planes"] - 1):
                planes = x.interval(out[0][-1], walls[k], walls[k + 1])
                for o, p in zip(out, planes):
                    o.append(p)
            A, J, chi, ne = [torch.stack(o, dim=-1) for o in out]
            return {"A": A, "J": J, "chi": chi, "ne": ne, "domain": None}
        A, J, chi, ne, evals = x.interval(a, zi, zf)
        return {"A": A, "J": J, "chi": chi, "ne": ne, "evaluations": evals if not case["adaptive"] else None}
