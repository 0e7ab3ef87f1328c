"""The calls that a simulation spends its time in, over the sizes it runs them at.

Five kinds of call, each through the public entry points and each on state
that stays on the GPU, as a driver's time loop holds it:

* ``leapfrog``:  one ``GaugeConfiguration.Update`` (the long gauge-only
  stretches of modes 1, 2, 3 and 11, and every equilibration).
* ``step``:      one pass of the correlator modes' time loop (3, 31, 32, 33):
  Crank-Nicolson update of the heavy field, leapfrog, norms, correlators.
  ``form`` 0 is the plain FP64 solve, 1 the precision form.
* ``ensemble``:  one coupled step of many sources and two masses in one gauge
  field, as one graph launch.
* ``gluon``:     a copy of the configuration fixed to Coulomb gauge, and its
  transverse correlators (modes 1 and 11).
* ``thermal``:   the Gauss projection of a freshly drawn thermal electric
  field (each initialisation round of modes 11 and 33).

The fields a pass leaves on the GPU are among its outputs; they are read back
when somebody asks for them (``Later``), as a program that goes on stepping
does not.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from nrqcd_b200 import _capi
from nrqcd_b200.batch import CNBatch, Ensemble
from nrqcd_b200.gaugeconfiguration_su3 import GaugeConfiguration
from nrqcd_b200.lattice import Lattice
from nrqcd_b200.nrqcd import NRQCDField

COEFFS = (1.0, 1.0, 1.0, 1.0)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest lattice anybody evolves (a quick check, one MPI job's default): launches only
        dict(name="leapfrog_8", kind="leapfrog", nx=8, ny=8, nz=8, a0=0.1, field="smooth"),
        # extents that are no power of two and no multiple of a warp
        dict(name="leapfrog_30x21x14", kind="leapfrog", nx=30, ny=21, nz=14, a0=0.05, field="thermal"),
        # the benchmark's lattice, before the heavy field is put in
        dict(name="leapfrog_64", kind="leapfrog", nx=64, ny=64, nz=64, a0=0.05, field="smooth"),
        # the thermal correlator run as its template sets it up (12^3, M = pi/2, a_t = 0.1)
        dict(name="step_12", kind="step", nx=12, ny=12, nz=12, a0=0.1, mass=1.570796, tol=1e-10, form=0,
             field="thermal"),
        # an odd box: no stencil that needs whole rows or even extents applies
        dict(name="step_15x21x18", kind="step", nx=15, ny=21, nz=18, a0=0.05, mass=1.0, tol=1e-12, form=0,
             field="smooth"),
        # the mid-size validation run at the heavier mass
        dict(name="step_32", kind="step", nx=32, ny=32, nz=32, a0=0.05, mass=2.0, tol=1e-12, form=0,
             field="smooth"),
        # the headline: one coupled step of the 64^3 lattice at residual 1e-12
        dict(name="step_64", kind="step", nx=64, ny=64, nz=64, a0=0.05, mass=1.0, tol=1e-12, form=0,
             field="smooth"),
        # the precision form at its two production sizes
        dict(name="precision_64", kind="step", nx=64, ny=64, nz=64, a0=0.05, mass=1.0, tol=1e-10, form=1,
             field="smooth"),
        dict(name="precision_96", kind="step", nx=96, ny=96, nz=96, a0=0.05, mass=1.0, tol=1e-10, form=1,
             field="smooth"),
        # one member of the batched ensemble: 16 random sources, masses 1.0 and 1.5
        dict(name="ensemble_24", kind="ensemble", nx=24, ny=24, nz=24, a0=0.05, sources=16, tol=1e-10,
             field="smooth"),
        # the gluon distribution as its template sets it up (16^3, tolerance 1e-10)
        dict(name="gluon_16", kind="gluon", nx=16, ny=16, nz=16, a0=0.1, field="smooth"),
        # one initialisation round's projection to the reference's tolerance
        dict(name="thermal_24", kind="thermal", nx=24, ny=24, nz=24, a0=0.1, tol=1e-3, field="thermal"),
    ]


def _extents(rng, lo, hi):
    """Three extents of a volume spread over its logarithm between lo^3 and hi^3."""
    side = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    shape = rng.choice(("cube", "even", "any"))
    if shape == "cube":
        n = max(lo, min(hi, 2 * round(side / 2)))
        return n, n, n
    n = [max(lo, min(hi, int(side * rng.uniform(0.75, 1.3)))) for _ in range(3)]
    if shape == "even":
        n = [max(lo, v - v % 2) for v in n]
    return tuple(n)


def draw(rng):
    kind = rng.choice(("leapfrog", "step", "step", "precision", "ensemble", "gluon", "thermal"))
    field = rng.choice(("smooth", "thermal"))
    a0 = rng.choice((0.05, 0.1))
    if kind == "leapfrog":
        nx, ny, nz = _extents(rng, 8, 96)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, a0=a0, field=field)
    if kind in ("step", "precision"):
        nx, ny, nz = _extents(rng, 12, 72)
        form = 1 if kind == "precision" else 0
        return dict(kind="step", nx=nx, ny=ny, nz=nz, a0=a0, mass=round(rng.uniform(1.0, 2.5), 3),
                    tol=1e-10 if form else rng.choice((1e-10, 1e-12)), form=form, field=field)
    if kind == "ensemble":
        nx, ny, nz = _extents(rng, 8, 24)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, a0=0.05, sources=rng.randint(2, 16), tol=1e-10, field="smooth")
    if kind == "gluon":
        nx, ny, nz = _extents(rng, 8, 32)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, a0=a0, field="smooth")
    nx, ny, nz = _extents(rng, 8, 24)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, a0=0.1, tol=1e-3, field="thermal")


def _volume(case):
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """What a pass cannot do without, per site: links 432 B, E 192 B, both species' propagators 1152 B, each read
    and written once; one staple force and link update 7.6 kflop; one application of the operator to both species
    22.5 kflop, of which a Crank-Nicolson step needs the right-hand side and, at about 1.5 digits each, the solve's."""
    v = _volume(case)
    gauge = {"bytes": 1248.0 * v, "flops": 7600.0 * v}
    if case["kind"] == "leapfrog":
        return gauge
    if case["kind"] == "step":
        applies = 1 + math.ceil((-math.log10(case["tol"]) - 4) / 1.5)
        return {"bytes": gauge["bytes"] + 2304.0 * v, "flops": gauge["flops"] + 22500.0 * v * applies}
    if case["kind"] == "ensemble":
        fields = 2 * case["sources"]
        return {"bytes": gauge["bytes"] + 2304.0 * v * fields, "flops": gauge["flops"] + 22500.0 * v * 5 * fields}
    if case["kind"] == "gluon":  # the links once per iteration (about a hundred), then the correlators
        return {"bytes": 100.0 * 864 * v + 648.0 * v, "flops": 100.0 * 3000 * v}
    # E once per sweep, about 1e4 sweeps at the reference's step
    return {"bytes": 1e4 * 384.0 * v, "flops": 1e4 * 3300.0 * v}


# ------------------------------------------------------------------ inputs
def _generators(device):
    """The eight SU(3) generators as the reference holds them (its column-major reshape transposes 2, 5 and 7)."""
    t = torch.zeros(8, 3, 3, dtype=torch.complex128)
    for a, (r, c) in ((0, (0, 1)), (3, (0, 2)), (5, (1, 2))):
        t[a, r, c] = t[a, c, r] = 0.5
        t[a + 1, r, c], t[a + 1, c, r] = 0.5j, -0.5j
    t[2] = torch.diag(torch.tensor([0.5, -0.5, 0.0], dtype=t.dtype))
    t[7] = torch.diag(torch.tensor([0.5, 0.5, -1.0], dtype=t.dtype)) / math.sqrt(3.0)
    return t.to(device)


def _mul(a, b):
    return (a.unsqueeze(-1) * b.unsqueeze(-3)).sum(-2)


def _dag(a):
    return a.conj().transpose(-1, -2)


def _algebra(coords):
    """sum_a coords^a T^a"""
    return torch.einsum("...a,arc->...rc", coords.to(torch.complex128), _generators(coords.device))


def _expi(h):
    """exp(i h) of small hermitian matrices: Taylor series of h / 16, squared four times."""
    x = 1j * h / 16
    eye = torch.eye(3, dtype=h.dtype, device=h.device).expand_as(h)
    out = eye.clone()
    for k in range(14, 0, -1):
        out = eye + _mul(x, out) / k
    for _ in range(4):
        out = _mul(out, out)
    return out


def _gauge_inputs(case, seed):
    """Links (nz, ny, nx, 3, 3, 3) [direction, row, column] and E (nz, ny, nx, 3, 8) on the GPU.

    smooth: long-wavelength modes only, as the saturated initial condition occupies them; thermal: white noise, the
    electric field of the reference's thermal draw at beta = 16 (sqrt(4 / beta) a0)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    shape = (case["nz"], case["ny"], case["nx"])
    noise = torch.randn(2, *shape, 3, 8, generator=gen, device="cuda", dtype=torch.float64)
    if case["field"] == "smooth":
        p2 = 0.0
        for k, n in enumerate(shape):
            w = 2 * torch.sin(math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n)
            p2 = p2 + (w * w).reshape([-1 if j == k else 1 for j in range(3)])
        damp = torch.exp(-p2 / 2).reshape(1, *shape, 1, 1)
        noise = torch.fft.ifftn(torch.fft.fftn(noise, dim=(1, 2, 3)) * damp, dim=(1, 2, 3)).real
        noise = noise / noise.square().mean().sqrt()
        angle, electric = 0.1, 0.1
    else:
        angle, electric = 0.12, 0.5
    return _expi(angle * _algebra(noise[0])), electric * case["a0"] * noise[1]


def _site(case, seed, k=0):
    """A source site (0-based, x fastest)."""
    return int(np.random.default_rng((int(seed), k)).integers(0, _volume(case)))


class _State:
    """One lattice with its fields, solver or batch; given back in order when it goes."""

    def __init__(self, case, seed):
        self.kind = case["kind"]
        self.case = case
        self.lat = Lattice((case["nx"], case["ny"], case["nz"]), (case["a0"], 1.0, 1.0, 1.0))
        self.solver = self.ensemble = self.batch = None
        self.fields, self.gauges = [], []
        links, efield = _gauge_inputs(case, seed)
        v = self.lat.V
        gauge = self.new_gauge()
        # the reference's arrays: links [site, direction, column, row]
        gauge.upload(links.reshape(v, 3, 3, 3).transpose(-1, -2).contiguous().cpu().numpy(),
                     efield.reshape(v, 3, 8).cpu().numpy())

    def new_gauge(self):
        self.gauges.append(GaugeConfiguration(lat=self.lat))
        return self.gauges[-1]

    def new_field(self, site):
        field = NRQCDField(lat=self.lat)
        field.InitSinglePoint(site + 1, site + 1)
        self.fields.append(field)

    def close(self):
        lat, self.lat = getattr(self, "lat", None), None
        if lat is None or not lat.is_open:
            return
        for held in (self.ensemble, self.batch, *self.fields):
            if held is not None:
                held.Destructor()
        if self.solver is not None:
            _capi.load().nrq_cn_finalize(self.solver)
        for gauge in self.gauges:
            gauge.Deallocate()
        lat.close()

    __del__ = close


def prepare(case, seed):
    state = _State(case, seed)
    if case["kind"] == "step":
        state.coeffs = _capi.coeffs(COEFFS)
        state.solver = ctypes.c_void_p()
        _capi.check(_capi.load().nrq_cn_init(state.lat.ctx, case["mass"], _capi.dptr(state.coeffs), 1.0, case["tol"],
                                             10000, case["form"], ctypes.byref(state.solver)), state.lat.ctx, "solver")
        state.new_field(_site(case, seed))
    elif case["kind"] == "ensemble":
        for k in range(case["sources"]):
            for _ in range(2):
                state.new_field(_site(case, seed, k))
        state.batch = CNBatch(state.fields, [1.0, 1.5] * case["sources"], case["tol"], lat=state.lat)
        state.ensemble = Ensemble([state.batch], state.gauges)
    elif case["kind"] in ("gluon", "thermal"):
        state.new_gauge()  # the copy that is worked on
    return state


# ------------------------------------------------------------------ one pass
class Later(dict):
    """Fields on the GPU by name: a name's array is read back when it is asked for."""

    def __getitem__(self, name):
        return super().__getitem__(name)()


def _read_links(state, gauge):
    return lambda: state.gauges[gauge].download()[0]


def _read_efield(state, gauge):
    return lambda: state.gauges[gauge].download()[1]


def _read_field(state, k):
    return lambda: np.stack(state.fields[k].download())


def _on_gpu(state, gauge=0):
    out = {"links": _read_links(state, gauge), "efield": _read_efield(state, gauge)}
    out.update({"field%02d" % k: _read_field(state, k) for k in range(len(state.fields))})
    return Later(out)


def run(state):
    gauge = state.gauges[0]
    if state.kind == "leapfrog":
        gauge.Update(1.0)
        return {"gpu": _on_gpu(state)}
    if state.kind == "step":
        field = state.fields[0]
        _capi.check(_capi.load().nrq_heavy_update_cn(state.solver, field.handle, gauge.handle, state.case["mass"],
                                                     _capi.dptr(state.coeffs), 1.0, None), state.lat.ctx, "update")
        gauge.Update(1.0)
        norms = np.array([field.GetNorm_Quark(), field.GetNorm_AntiQ()])
        mesons = field.GetMesoncorrelators()
        return {"gpu": _on_gpu(state), "norms": norms, "mesons": np.array([mesons[k] for k in sorted(mesons)])}
    if state.kind == "ensemble":
        state.ensemble.Step(COEFFS, 1.0)
        return {"gpu": _on_gpu(state)}
    copy = state.gauges[1]
    copy.assign(gauge)
    if state.kind == "gluon":
        iterations, deviations = copy.CoulombGaugefixing(1e-10, 0.08, 100000, verbose=False)
        aa, ee, momenta = copy.GetTransverseCorrelators()
        return {"gpu": _on_gpu(state, 1), "iterations": iterations, "deviations": deviations, "aa": aa, "ee": ee,
                "momenta": momenta}
    sweeps, deviation = copy.GaussProjection(state.case["tol"])
    return {"gpu": _on_gpu(state, 1), "sweeps": sweeps, "deviation": deviation}


# ------------------------------------------------------------------ the same in plain 64-bit torch
def _up(x, i, n=1):
    """The field at the neighbour n steps along direction i (x, y, z = dims 2, 1, 0)."""
    return torch.roll(x, -n, dims=2 - i)


def _coords(m):
    """2 Tr(T^a m)"""
    return 2 * torch.einsum("arc,...cr->...a", _generators(m.device), m)


def _exact_leapfrog(u, e, a0):
    u = _mul(_expi(_algebra(e)), u)
    new = []
    for i in range(3):
        staples = 0
        for k in range(3):
            if k == i:
                continue
            ui, uk = u[..., i, :, :], u[..., k, :, :]
            above = _mul(_mul(_up(uk, i), _dag(_up(ui, k))), _dag(uk))
            below = _mul(_mul(_dag(_up(_up(uk, i), k, -1)), _dag(_up(ui, k, -1))), _up(uk, k, -1))
            staples = staples + a0 ** 2 * (above + below)
        new.append(e[..., i, :] - _coords(_mul(u[..., i, :, :], staples)).imag)
    return u, torch.stack(new, -2)


def _log_angle(p):
    """The hermitian H of p = exp(i H), eigenphases inside the principal branch."""
    k = (p - _dag(p)) / 2j
    s = torch.cat([torch.linalg.eigh(part)[1] for part in k.reshape(-1, 3, 3).split(16384)]).reshape(k.shape)
    theta = torch.angle(torch.diagonal(_mul(_mul(_dag(s), p), s), dim1=-2, dim2=-1))
    return _mul(s * theta.unsqueeze(-2), _dag(s))


class _Operator:
    """A = 1 + sum_t alpha_t G_t of one species, blocks transposed as PETSc assembles them (row index 2 colour + spin)."""

    def __init__(self, u, e, a0, mass, sign):
        c = torch.complex128
        dev = u.device
        m = sign * mass
        kappa = -0.5j * a0
        eye2 = torch.eye(2, dtype=c, device=dev)
        sigma = torch.tensor([[[0, 1], [1, 0]], [[0, 1j], [-1j, 0]], [[1, 0], [0, -1]]], dtype=c, device=dev)

        def kron(a, s):
            return torch.einsum("...ij,st->...isjt", a, s).reshape(*a.shape[:-2], 6, 6)

        ef = -_algebra(e).real.to(c) / a0
        link = [u[..., i, :, :] for i in range(3)]
        el = [ef[..., j, :, :] for j in range(3)]
        darwin, magnetic = 0, 0
        for i in range(3):
            j, k = (i + 1) % 3, (i + 2) % 3
            darwin = darwin + (_mul(_mul(link[i], _up(el[i], i)), _dag(link[i]))
                               - _up(_mul(_mul(_dag(link[i]), el[i]), link[i]), i, -1)) / 2
            plaq = _mul(_mul(link[j], _up(link[k], j)), _dag(_mul(link[k], _up(link[j], k))))
            magnetic = magnetic + _log_angle(plaq).real.to(c)
        diag = kron(darwin, eye2) * (-kappa / (8 * m * m)) + kron(magnetic, eye2) * (-kappa / (2 * m))
        diag = diag + torch.eye(6, dtype=c, device=dev) * (1 + 3 * kappa / m)
        self.diag = diag.transpose(-1, -2)
        self.hop = []
        for i in range(3):
            j, k = (i + 1) % 3, (i + 2) % 3
            w = kron(link[i], eye2) * (-kappa / (2 * m))
            for jj, kk, eps in ((j, k, 1.0), (k, j, -1.0)):
                de = (_mul(el[jj], link[i]) + _mul(link[i], _up(el[jj], i))) / 2
                w = w + kron(de, sigma[kk]) * (-1j * kappa * eps / (8 * m * m))
            self.hop.append(w.transpose(-1, -2))

    def apply(self, psi, herm=False):
        """Real coefficients: the backward block is -(forward block at the neighbour)^H, and A^H = 2 - A."""
        out = torch.matmul(self.diag, psi)
        for i in range(3):
            out += torch.matmul(self.hop[i], _up(psi, i))
            out -= _up(torch.matmul(_dag(self.hop[i]), psi), i, -1)
        return 2 * psi - out if herm else out

    def step(self, psi, centre):
        """A^H x = A psi by Richardson steps about the spectrum's centre, to rounding."""
        b = self.apply(psi)
        x = 2 * b - psi
        norm, best = b.norm(), math.inf
        for _ in range(200):
            r = b - self.apply(x, True)
            now = float(r.norm() / norm)
            if now < 3e-16 or now > 0.7 * best:
                break
            best = now
            x = x + r / (1 + 1j * centre)
        return x


def _point(case, sites):
    """(nz, ny, nx, 6, 6 len(sites)) point sources, columns of one source together."""
    psi = torch.zeros(_volume(case), 6, len(sites), 6, dtype=torch.complex128, device="cuda")
    for k, s in enumerate(sites):
        psi[s, :, k, :] = torch.eye(6, dtype=psi.dtype, device=psi.device) / math.sqrt(6.0)
    return psi.reshape(case["nz"], case["ny"], case["nx"], 6, 6 * len(sites))


def _exact_fields(case, u, e, mass, sites):
    """Both species of every source after one step: (2, V, 6, 6) [species, site, column, row] each."""
    species = []
    for sign in (1.0, -1.0):
        x = _Operator(u, e, case["a0"], mass, sign).step(_point(case, sites), sign * 3 * case["a0"] / (2 * mass))
        species.append(x.reshape(-1, 6, len(sites), 6).permute(2, 0, 3, 1).contiguous())
    return torch.stack(species, 1)


def _exact_mesons(prop):
    """O1(1S0), O1(3S1), O8(1S0), O8(3S1) of one field (2, V, 6, 6)."""
    q, a = prop[0].transpose(-1, -2), prop[1].transpose(-1, -2)
    t = _generators(prop.device)
    sigma = torch.tensor([[[0, 1], [1, 0]], [[0, 1j], [-1j, 0]], [[1, 0], [0, -1]]], dtype=t.dtype, device=t.device)
    eye2, eye3 = (torch.eye(n, dtype=t.dtype, device=t.device) for n in (2, 3))
    colours, spins = list(t), list(sigma)

    def total(pairs, weight):
        out = 0
        for colour, spin in pairs:
            g = torch.kron(colour, spin)
            out = out + torch.einsum("xji,jk,xkl,li->", a.conj(), g, q, g)
        return 1j * weight * out

    return torch.stack([total([(eye3, eye2)], 1.0), total([(eye3, s) for s in spins], 1 / 3),
                        total([(c, eye2) for c in colours], 6 / 8),
                        total([(c, s) for s in spins for c in colours], 6 / 24)])


def _exact_gauge(u, e):
    v = u.shape[0] * u.shape[1] * u.shape[2]
    return {"links": u.reshape(v, 3, 3, 3).transpose(-1, -2).contiguous(), "efield": e.reshape(v, 3, 8)}


def _exact_gluon(case, u, e):
    dims = (0, 1, 2)
    momentum = []
    for i in range(3):
        n = u.shape[2 - i]
        ph = math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n
        p = 2 * torch.sin(ph) * torch.exp(-1j * ph)
        momentum.append(p.reshape([-1 if 2 - i == d else 1 for d in range(3)]).expand(u.shape[:3]))
    pn = sum(p.abs() ** 2 for p in momentum).sqrt()
    accelerate = torch.where(pn > 1e-12, (pn.max() / pn.clamp_min(1e-12)) ** 2, torch.ones_like(pn))
    deviations, count = [], 0
    for count in range(1, 100001):
        d = sum(_up(u[..., i, :, :], i, -1) - u[..., i, :, :] for i in range(3))
        d = (d - _dag(d)) / 2
        deviations.append(float(d.abs().square().sum((-1, -2)).sqrt().max() / 9))
        if not deviations[-1] > 1e-10:
            break
        d = torch.fft.ifftn(torch.fft.fftn(d, dim=dims) * accelerate[..., None, None], dim=dims)
        g = _expi(-0.08j * d)
        u = torch.stack([_mul(_mul(g, u[..., i, :, :]), _dag(_up(g, i))) for i in range(3)], -3)
    out = {"iterations": count, "deviations": np.array(deviations), "momenta": pn.reshape(-1)}
    p = torch.stack(momentum, -1)
    unit = torch.where(pn > 1e-12, 1 / pn.clamp_min(1e-12), torch.zeros_like(pn))[..., None]
    project = (torch.eye(3, device="cuda") - (p.conj().unsqueeze(-1) * p.unsqueeze(-2)).real
               * (unit * unit).unsqueeze(-1)) / 2
    project = torch.where((pn < 1e-12)[..., None, None], torch.zeros_like(project), project).to(torch.complex128)
    a = _coords(_log_angle(u)).real
    for name, field in (("aa", a), ("ee", e / case["a0"])):
        f = torch.fft.fftn(field.to(torch.complex128), dim=dims)
        out[name] = (torch.einsum("...ia,...ij,...ja->...", f, project, f.conj()).real / (8 * _volume(case))).reshape(-1)
    return dict(out, gpu=_exact_gauge(u, e))


def _exact_thermal(case, u, e):
    a0 = case["a0"]
    ud = _dag(u)
    sweeps = 0
    while True:
        m = _algebra(e)
        back = _mul(_mul(ud, m), u)
        g = sum(m[..., i, :, :] - _up(back[..., i, :, :], i, -1) for i in range(3)) / a0
        deviation = float(_coords(g).abs().max())
        if not deviation > case["tol"]:
            return {"gpu": _exact_gauge(u, e), "sweeps": sweeps, "deviation": deviation}
        sweeps += 1
        ahead = torch.stack([_up(g, i) for i in range(3)], -3)
        here = g.unsqueeze(-3)
        e = _coords(0.01 * a0 * (_mul(_mul(_mul(u, here), ud), ahead) - here) + m).real


def exact(case, seed):
    if _volume(case) > 72 ** 3:
        return None  # takes over about 20 seconds
    u, e = _gauge_inputs(case, seed)
    if case["kind"] == "gluon":
        return _exact_gluon(case, u, e)
    if case["kind"] == "thermal":
        return _exact_thermal(case, u, e)
    fields = {}
    if case["kind"] == "step":
        field = _exact_fields(case, u, e, case["mass"], [_site(case, seed)])[0]
        fields["field00"] = field
    elif case["kind"] == "ensemble":
        sites = [_site(case, seed, k) for k in range(case["sources"])]
        for which, mass in enumerate((1.0, 1.5)):
            for k, field in enumerate(_exact_fields(case, u, e, mass, sites)):
                fields["field%02d" % (2 * k + which)] = field
    out = {"gpu": dict(_exact_gauge(*_exact_leapfrog(u, e, case["a0"])), **fields)}
    if case["kind"] == "step":
        out["norms"] = field.abs().square().sum((1, 2, 3)).sqrt()
        out["mesons"] = _exact_mesons(field)
    return out
