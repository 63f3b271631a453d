"""The work that programs have this package do, as cases that can be timed and checked.

A case is a dict of plain values.  ``prepare`` makes on the GPU what a program holds before the call (fields from the
seed, in the distributions of ``pelelmex_b200.workloads``; the reactor and the surrogate a program keeps for its whole
run are made once per process), ``run`` is one pass through the public entry points, ``exact`` the same result from
plain torch in 64 bits: the reaction ODE solved by a three-stage Radau IIA method with steps far below what its error
needs, the rates and the network's gradients evaluated directly.

Fields are the flame-like and box-list fields of the workloads module: H2/air at random temperatures, a CH4/air tanh
flame, dodecane mixing boxes and a dodecane random-field flame.  Tolerances of the reactor are the parity settings
(rtol 1e-8, atol 1e-12, order 5) unless a case sets the usual input-file ones (rtol 1e-6, atol 1e-5 on typical values).
"""
import functools
import math
from pathlib import Path

import numpy as np
import torch

from pelelmex_b200 import mechanism as mechmod
from pelelmex_b200 import perfmodel
from pelelmex_b200.reactor import Box, ReactorB200
from pelelmex_b200.surrogate import Ensemble, HybridReactor, MLPSurrogate, fit_normalisation

DEV = "cuda:0"
MECHS = {"h2": "synth_h2_9", "ch4": "synth_ch4_21", "c12": "synth_c12_53"}
RU, PATM = mechmod.R_CGS, mechmod.P_ATM_CGS
SURROGATE = Path(mechmod.__file__).parent / "surrogates" / "synth_ch4_21.b2s"
# right-hand sides and Jacobians a cell needs on the way (measured means of the fields at dt 1e-6; a longer step needs
# more by about the fourth root), for the operation counts only
RHS_PER_CELL = {"h2": 45.0, "ch4": 36.0, "c12_boxes": 30.0, "c12_grf": 200.0}


def listed():
    return [
        # one AMR box of the smallest blocking factor: launches and latency are all there is
        dict(name="h2_box_8", kind="react", field="h2", nx=8, ny=8, nz=8, ghost=1, dt=1e-6, boxes=True),
        # the CPU-runnable H2/air batch, flat arrays
        dict(name="h2_flat_32", kind="react", field="h2", nx=32, ny=32, nz=32, ghost=0, dt=1e-6, boxes=False),
        # one ragged CH4 box with ghost cells and the longer of the two chemistry steps
        dict(name="ch4_box_61x43x37_dt1e-5", kind="react", field="ch4", nx=61, ny=43, nz=37, ghost=2, dt=1e-5, boxes=True),
        # the headline field: 128^3 CH4 flame, dt 1e-6
        dict(name="ch4_flat_128", kind="react", field="ch4", nx=128, ny=128, nz=128, ghost=0, dt=1e-6, boxes=False),
        # Newton solves in 64 bits throughout, the option of parity runs
        dict(name="ch4_fp64_32", kind="react", field="ch4", nx=32, ny=32, nz=32, ghost=0, dt=1e-6, boxes=False, lu_fp64=True),
        # one level's step: forcing from the advection-diffusion update, then the chemistry advance of its box list
        # (mask, one covered box), at the tolerances of the input files
        dict(name="ch4_level_7_boxes", kind="level", nbox=7, e0=20, e1=48, ghost=1, dt=1e-6),
        # surrogate first, at the headline size and at a ragged ordinary one with the longer step
        dict(name="hybrid_128", kind="hybrid", nx=128, ny=128, nz=128, dt=1e-6),
        dict(name="hybrid_57x40x33_dt1e-5", kind="hybrid", nx=57, ny=40, nz=33, dt=1e-5),
        # dodecane box list, half cold and half igniting
        dict(name="c12_boxes_6", kind="boxes", nbox=6, e0=16, e1=48, dt=1e-6),
        # dodecane random-field flame: few cells with thousands of right-hand sides set the length
        dict(name="c12_grf_20", kind="react", field="c12_grf", nx=20, ny=20, nz=20, ghost=0, dt=5e-6, boxes=False),
        # derived fields of a plotfile: T from (h, Y), rates and heat release
        dict(name="rates_ch4_96", kind="rates", field="ch4", nx=96, ny=96, nz=96),
        # one training step of a network of the ensemble
        dict(name="train_16384", kind="train", batch=16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["react", "react", "react", "react", "level", "hybrid", "boxes", "rates", "train"])
    if kind == "react":
        field = rng.choice(["h2", "ch4", "ch4", "c12_grf"])
        dt = math.exp(rng.uniform(math.log(2e-7), math.log(1e-5)))
        hi = {"h2": 1_000_000, "ch4": 1_000_000 if dt < 2e-6 else 500_000, "c12_grf": 6000}[field]
        nx, ny, nz = _shape(rng, 64, hi)
        return dict(kind=kind, field=field, nx=nx, ny=ny, nz=nz, ghost=rng.choice([0, 1, 2]), dt=dt,
                    boxes=rng.random() < 0.5, lu_fp64=field != "c12_grf" and nx * ny * nz < 50_000 and rng.random() < 0.2)
    if kind == "level":
        return dict(kind=kind, nbox=rng.randint(1, 9), e0=rng.randint(8, 24), e1=rng.randint(25, 56), ghost=rng.choice([1, 2]),
                    dt=math.exp(rng.uniform(math.log(2e-7), math.log(4e-6))))
    if kind == "hybrid":
        nx, ny, nz = _shape(rng, 1000, 1_200_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dt=rng.choice([1e-6, 1e-5]))
    if kind == "boxes":
        return dict(kind=kind, nbox=rng.randint(2, 8), e0=rng.randint(8, 20), e1=rng.randint(21, 44),
                    dt=math.exp(rng.uniform(math.log(3e-7), math.log(1.5e-6))))
    if kind == "rates":
        field = rng.choice(["h2", "ch4", "c12_grf"])
        nx, ny, nz = _shape(rng, 1000, 200_000 if field == "c12_grf" else 1_500_000)
        return dict(kind=kind, field=field, nx=nx, ny=ny, nz=nz)
    return dict(kind="train", batch=128 * _log_int(rng, 4, 256))


def _shape(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    nx = max(3, int(round(n ** (1 / 3) * rng.uniform(0.8, 1.6))))
    ny = max(3, int(round(math.sqrt(n / nx) * rng.uniform(0.8, 1.25))))
    return nx, ny, max(2, n // (nx * ny))


# ------------------------------------------------------------------- mechanism tables and formulas, FP64 torch
class _Mech:
    def __init__(self, key, dev=DEV):
        self.mech = mechmod.builtin(MECHS[key])
        f = mechmod.flatten(self.mech)
        a = f.arrays
        self.N, self.R, self.names = f.n_species, f.n_reactions, self.mech.names
        t = lambda v: torch.tensor(np.asarray(v, np.float64), device=dev)  # noqa: E731
        self.mw, self.nasa = t(a["mw"]), t(a["nasa"])
        self.arr, self.arr_lo, self.arr_rev, self.troe = t(a["arr"]), t(a["arr_lo"]), t(a["arr_rev"]), t(a["troe"])
        sp, nu = np.asarray(a["sp"]).reshape(self.R, 8), np.asarray(a["nu"]).reshape(self.R, 8)
        net, eff = np.zeros((self.R, self.N)), np.ones((self.R, self.N))
        for j in range(self.R):
            for s in range(8):
                if sp[j, s] >= 0:
                    net[j, sp[j, s]] += nu[j, s] if s >= 4 else -nu[j, s]
            for q in range(a["eff_ptr"][j], a["eff_ptr"][j + 1]):
                eff[j, a["eff_sp"][q]] = a["eff_val"][q]
        self.net, self.eff = t(net), t(eff)
        self.sp = torch.tensor(np.where(sp < 0, self.N, sp), device=dev)
        self.nu = t(np.where(sp < 0, 0, nu))
        kind, flags = torch.tensor(np.asarray(a["rtype"]), device=dev), torch.tensor(np.asarray(a["rflags"]), device=dev)
        self.third, self.fall, self.is_troe = kind == 1, kind >= 2, kind == 3
        self.rev, self.exp_rev, self.t2 = (flags & 1) != 0, (flags & 2) != 0, (flags & 4) != 0

    def thermo(self, T):
        """cp/R, h/RT, s/R of every species, [..., N], for T [...]."""
        T = T[..., None]
        a = torch.where((T < self.nasa[:, 0])[..., None], self.nasa[:, 1:8], self.nasa[:, 8:15])
        a0, a1, a2, a3, a4, a5, a6 = a.unbind(-1)
        cp = a0 + T * (a1 + T * (a2 + T * (a3 + T * a4)))
        h = a0 + T * (a1 / 2 + T * (a2 / 3 + T * (a3 / 4 + T * a4 / 5))) + a5 / T
        s = a0 * torch.log(T) + T * (a1 + T * (a2 / 2 + T * (a3 / 3 + T * a4 / 4))) + a6
        return cp, h, s

    def wdot(self, C, T, g):
        """Molar production rates for concentrations C [..., N], temperature T [...] and g/RT [..., N]."""
        T = T[..., None]
        ln, inv = torch.log(T), 1.0 / T
        arr = lambda p: torch.exp(p[:, 0] + p[:, 1] * ln - p[:, 2] * inv)  # noqa: E731
        kinf, k0 = arr(self.arr), arr(self.arr_lo)
        M = C @ self.eff.T
        pr = k0 * M / kinf
        al, t3, t1, t2 = self.troe.unbind(-1)
        safe = lambda v: torch.where(self.is_troe, v, 1.0)  # noqa: E731
        fc = (1 - al) * torch.exp(-T / safe(t3)) + al * torch.exp(-T / safe(t1)) + torch.where(self.t2, torch.exp(-t2 * inv), 0.0)
        lf = torch.log10(torch.where(self.is_troe, fc, 1.0).clamp_min(1e-300))
        u = torch.log10(pr.clamp_min(1e-300)) - 0.4 - 0.67 * lf
        f1 = u / (0.75 - 1.27 * lf - 0.14 * u)
        F = torch.where(self.is_troe, 10.0 ** (lf / (1 + f1 * f1)), 1.0)
        kf = torch.where(self.fall, kinf * pr / (1 + pr) * F, kinf)
        kc = torch.exp(torch.where(self.rev, g @ self.net.T - self.net.sum(1) * torch.log(PATM / (RU * T)), 0.0))
        kr = torch.where(self.exp_rev, arr(self.arr_rev), torch.where(self.rev, kf * kc, 0.0))
        slots = torch.cat([C, torch.ones_like(C[..., :1])], -1)[..., self.sp] ** self.nu
        q = kf * slots[..., :4].prod(-1) - kr * slots[..., 4:].prod(-1)
        return torch.where(self.third, q * M, q) @ self.net

    def rhs(self, y, F):
        """d(rhoY, T)/dt of the constant-pressure system, [..., N + 1], for the forcing F (extF_rhoY, extF_rhoH)."""
        N, T = self.N, y[..., self.N]
        cp, h, s = self.thermo(T)
        C = y[..., :N] / self.mw
        yd = self.wdot(C, T, h - s) * self.mw + F[..., :N]
        hs = (h * (RU * T)[..., None] / self.mw * yd).sum(-1)
        return torch.cat([yd, ((F[..., N] - hs) / (cp * C * RU).sum(-1))[..., None]], -1)

    def density_enthalpy(self, Y, T):
        """rho [...] at 1 atm and h [...] per mass (CGS)."""
        _, h, _ = self.thermo(T)
        return PATM / (RU * T * (Y / self.mw).sum(-1)), (Y * h * (RU * T)[..., None] / self.mw).sum(-1)

    def mass(self, **moles):
        """Mass fractions [n, N] of a mixture given by moles per species name."""
        n = max(v.numel() for v in moles.values())
        X = torch.zeros((n, self.N), dtype=torch.float64, device=self.mw.device)
        for k, v in moles.items():
            X[:, self.names.index(k)] = v
        X *= self.mw
        return X / X.sum(1, keepdim=True)


@functools.lru_cache(maxsize=None)
def _mech(key):
    return _Mech(key)


def _rand(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device=DEV, generator=g)


def _noisy(g, Y, share):
    Y = Y * (1.0 + share * (2.0 * torch.rand(Y.shape, dtype=torch.float64, device=DEV, generator=g) - 1.0))
    return Y / Y.sum(1, keepdim=True)


def _field(field, g, nx, ny, nz):
    """(mechanism, Y [cells, N], T [cells]) of one box, i fastest."""
    n = nx * ny * nz
    if field == "h2":
        m = _mech("h2")
        Y = m.mass(H2=torch.full((n,), 2.0), O2=torch.tensor([1.0]), N2=torch.tensor([3.76]))
        return m, _noisy(g, Y, 0.05), _rand(g, n, 1000.0, 2000.0)
    if field == "ch4":
        m = _mech("ch4")
        col = torch.arange(n, device=DEV) // nx
        x = (torch.arange(n, device=DEV) % nx).double()
        s = 0.5 * (1.0 + torch.tanh((x - nx / 2) / (nx / 16)))
        Tu, phi, Tb = (_rand(g, ny * nz, a, b) for a, b in ((300.0, 800.0), (0.7, 1.3), (1500.0, 2300.0)))
        Yu = m.mass(CH4=phi, O2=torch.tensor([2.0]), N2=torch.tensor([7.52]))
        # burnt: complete products with a little dissociation; rich columns leave CO and H2
        o2 = 2.0 / phi - 2.0
        lack = (-2.0 * o2).clamp_min(0.0)
        co = (lack / 2).clamp_max(1.0)
        h2 = (lack - co).clamp_max(2.0)
        co2, h2o = 1.0 - co, 2.0 - h2
        Yb = m.mass(CO2=0.95 * co2, CO=co + 0.05 * co2, H2O=0.98 * h2o, OH=0.02 * h2o, H2=h2 + 0.01 * h2o,
                    O2=o2.clamp_min(0.0) + 0.025 * co2, N2=7.52 / phi)
        Y = (1.0 - s)[:, None] * Yu[col] + s[:, None] * Yb[col]
        for sp, amp in (("H", 4e-4), ("O", 1e-3), ("OH", 3e-3), ("HO2", 2e-4), ("CH3", 1e-3), ("CH2O", 1.5e-3), ("HCO", 5e-5)):
            Y[:, m.names.index(sp)] += amp * 4.0 * s * (1.0 - s) * _rand(g, ny * nz, 0.5, 1.5)[col]
        return m, _noisy(g, Y, 0.02), (1.0 - s) * Tu[col] + s * Tb[col]
    m = _mech("c12")
    air = m.mass(O2=torch.ones(n), N2=torch.tensor([3.76]))
    i = m.names.index
    if field in ("c12_cold", "c12_ignite"):
        fa = _rand(g, n, 0.5, 2.0) * m.mw[i("NC12H26")] / (18.5 * (m.mw[i("O2")] + 3.76 * m.mw[i("N2")]))
        Z = fa / (1.0 + fa)
        Y = (1.0 - Z)[:, None] * air
        Y[:, i("NC12H26")] += Z
        return m, _noisy(g, Y, 0.02), _rand(g, n, *((300.0, 600.0) if field == "c12_cold" else (900.0, 1400.0)))
    # random-field flame: smooth Gaussian fields for T and the mixture fraction, through the normal CDF
    c = torch.arange(n, device=DEV)
    xyz = torch.stack([c % nx, (c // nx) % ny, c // (nx * ny)], 1).double()

    def smooth():
        k = torch.randn((3, 64), dtype=torch.float64, device=DEV, generator=g) / (max(nx, ny, nz) / 16.0)
        f = torch.cos(xyz @ k + 2 * math.pi * _rand(g, 64)).sum(1) * math.sqrt(2.0 / 64)
        return 0.5 * (1.0 + torch.erf(f / math.sqrt(2.0)))
    prog, Z = smooth(), smooth()
    mix = (1.0 - Z)[:, None] * air
    mix[:, i("NC12H26")] += Z
    nf, no2 = mix[:, i("NC12H26")] / m.mw[i("NC12H26")], mix[:, i("O2")] / m.mw[i("O2")]
    burn = torch.minimum(nf, no2 / 12.5)
    left = no2 - 12.5 * burn
    co2 = torch.minimum(12.0 * burn, 2.0 * left)
    prod = m.mass(NC12H26=nf - burn, CO2=co2, CO=12.0 * burn - co2, H2O=13.0 * burn, O2=left - 0.5 * co2,
                  N2=mix[:, i("N2")] / m.mw[i("N2")])
    Y = ((1.0 - prog)[:, None] * mix + prog[:, None] * prod).clamp_min(0.0)
    return m, Y / Y.sum(1, keepdim=True), 300.0 + 2100.0 * prog


def _state(field, g, nx, ny, nz):
    """(mechanism, rhoY [N, cells], T, rhoH) in CGS."""
    m, Y, T = _field(field, g, nx, ny, nz)
    rho, h = m.density_enthalpy(Y, T)
    return m, (rho[:, None] * Y).t().contiguous(), T, rho * h


# ------------------------------------------------------------------------------------------- what a program keeps
@functools.lru_cache(maxsize=None)
def _reactor(key, lu_fp64=False, inputs=False):
    """The reactor of a program's run: parity settings, or the input files' with typical values."""
    if not inputs:
        return ReactorB200(MECHS[key], rtol=1e-8, atol=1e-12, max_order=5, lu_fp64=lu_fp64).init(2, 1)
    r = ReactorB200(MECHS[key], rtol=1e-6, atol=1e-5, max_order=5).init(2, 1)
    r.set_typ_vals_ode([1e-4] * r.N + [2000.0])  # partial densities ~1e-4 g/cm^3, burnt temperature
    return r


@functools.lru_cache(maxsize=None)
def _hybrid():
    return HybridReactor(_reactor("ch4"), Ensemble.load(SURROGATE, MECHS["ch4"], DEV))


def _key(field):
    return field.split("_")[0]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _fab(v, nx, ny, nz, ghost, fill=0.0):
    """[ncomp, cells] (or [cells]) values of a box as a fab with ghost cells."""
    v = v.reshape(-1, nz, ny, nx)
    f = torch.full((v.shape[0], nz + 2 * ghost, ny + 2 * ghost, nx + 2 * ghost), fill, dtype=v.dtype, device=v.device)
    f[:, ghost:ghost + nz, ghost:ghost + ny, ghost:ghost + nx] = v
    return f


def _box_dims(case):
    """Edges of the boxes of a list: e0 and e1 in turn with odd ones between, placed side by side along x."""
    out, x0 = [], 0
    for b in range(case["nbox"]):
        f = [0.0, 1.0, 0.35, 0.7, 0.15, 0.85, 0.5][b % 7]
        e = int(round(case["e0"] + f * (case["e1"] - case["e0"])))
        out.append((Box((x0, 0, 0), (x0 + e - 1, e + b % 3 - 1, e - 1)), e, e + b % 3, e))
        x0 += e
    return out


def _fields_of(case):
    """[(field, nx, ny, nz)] of the boxes of a case."""
    if case["kind"] in ("level", "boxes"):  # cold and igniting boxes of a dodecane list alternate
        return [("ch4" if case["kind"] == "level" else ("c12_cold" if b % 2 else "c12_ignite"), nx, ny, nz)
                for b, (_, nx, ny, nz) in enumerate(_box_dims(case))]
    if case["kind"] == "train":
        return []
    return [(case.get("field", "ch4"), case["nx"], case["ny"], case["nz"])]


# --------------------------------------------------------------------------------------------------- the interface
def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, g, seed)
    states = [_state(f, g, nx, ny, nz) for f, nx, ny, nz in _fields_of(case)]
    s = {"case": case}
    if kind in ("react", "hybrid"):
        m, rhoY, T, rhoH = states[0]
        n = T.numel()
        # the advection-diffusion forcing moves a cell by about 1e-5 of its content in a step; the hybrid field has none
        amp = 0.0 if kind == "hybrid" else 1e-5 / case["dt"]
        fY = rhoY * amp * torch.randn(rhoY.shape, dtype=torch.float64, device=DEV, generator=g)
        fH = rhoH.abs() * amp * torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
        if kind == "hybrid":
            s["r"] = _hybrid()
            s["r"]._handle()  # the networks are on the device before the first step
        else:
            s["r"] = _reactor(_key(case["field"]), bool(case.get("lu_fp64")))
        arrays = [rhoY, T, rhoH, fY, fH, torch.zeros_like(T)]
        if case.get("boxes"):
            dims = (case["nx"], case["ny"], case["nz"])
            gh = case["ghost"]
            arrays = [_fab(v, *dims, gh) for v in arrays]
            s["box"] = Box((0, 0, 0), tuple(d - 1 for d in dims))
            s["lo"] = (-gh, -gh, -gh)
        s["rhoY0"], s["T0"], s["rhoH0"], s["fY"], s["fH"], s["fct"] = arrays
        s["rhoY"], s["T"], s["rhoH"] = (torch.empty_like(v) for v in arrays[:3])
        return s
    if kind == "boxes":
        s["r"] = _reactor("c12")
        s["old"], s["items"] = [], []
        for (m, rhoY, T, rhoH), (box, nx, ny, nz) in zip(states, _box_dims(case)):
            old = [_fab(v, nx, ny, nz, 0) for v in (rhoY, T, rhoH)]
            new = [torch.empty_like(v) for v in old]
            s["old"].append((old, new))
            s["items"].append((box, new[0], torch.zeros_like(old[0]), new[1], new[2], torch.zeros_like(old[1]),
                               torch.zeros_like(old[1]), None, box.lo))
        return s
    if kind == "level":
        s["r"] = _reactor("ch4", inputs=True)
        gh = case["ghost"]
        s["force"], s["adv"] = [], []
        for b, ((m, rhoY, T, rhoH), (box, nx, ny, nz)) in enumerate(zip(states, _box_dims(case))):
            fab = lambda v: _fab(v, nx, ny, nz, gh)  # noqa: E731
            lo = tuple(v - gh for v in box.lo)
            old = [fab(rhoY * 1e3), fab(rhoH * 0.1), fab(T)]  # MKS
            noise = lambda v: v * (1.0 + 1e-5 * torch.randn(v.shape, dtype=torch.float64, device=DEV, generator=g))  # noqa: E731
            adv = [noise(old[0]), noise(old[1])]
            ir_old = old[0] * (0.05 / case["dt"]) * 1e-3 * torch.randn(old[0].shape, dtype=torch.float64, device=DEV, generator=g)
            fY, fH = torch.zeros_like(old[0]), torch.zeros_like(old[1])
            new = [torch.zeros_like(v) for v in old]
            mask = (torch.rand((1,) + old[2].shape[1:], device=DEV, generator=g) < 0.97).to(torch.int32)
            s["force"].append((box, old[0], old[1], adv[0], adv[1], ir_old, fY, fH, lo))
            s["adv"].append((box, old[0], old[1], old[2], new[0], new[1], new[2], fY, fH, torch.zeros_like(fH), mask,
                             torch.zeros_like(old[0]), lo))
        s["skip"] = [b == 2 for b in range(case["nbox"])]  # one box covered by a finer level
        return s
    m, rhoY, T, rhoH = states[0]  # rates: MKS state and the previous temperature as the first guess
    s["r"] = _reactor(_key(case["field"]))
    s["rhoY"], s["rhoH"] = rhoY * 1e3, rhoH * 0.1
    s["T0"] = T * (1.0 + 0.01 * torch.randn(T.shape, dtype=torch.float64, device=DEV, generator=g))
    s["T"] = torch.empty_like(T)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind in ("react", "hybrid"):
        for k in ("rhoY", "T", "rhoH"):  # new state <- old state, as a step begins
            s[k].copy_(s[k + "0"])
        dt = s["case"]["dt"]
        if "box" in s:
            s["r"].react(s["box"], s["rhoY"], s["fY"], s["T"], s["rhoH"], s["fH"], s["fct"], None, dt, fab_lo=s["lo"])
        else:
            s["r"].react_flat(s["rhoY"], s["fY"], s["T"], s["rhoH"], s["fH"], s["fct"], dt_react=dt)
        return [s["rhoY"], s["T"], s["rhoH"]]
    if kind == "boxes":
        for old, new in s["old"]:
            for a, b in zip(old, new):
                b.copy_(a)
        s["r"].react_boxes(s["items"], s["case"]["dt"])
        return [new for _, new in s["old"]]
    if kind == "level":
        dt = s["case"]["dt"]
        s["r"].react_force(s["force"], dt)
        s["r"].advance_chemistry(s["adv"], dt, skip_react=s["skip"])
        return [[it[4], it[5], it[6], it[11]] for it in s["adv"]]
    if kind == "rates":
        s["T"].copy_(s["T0"])
        w = s["r"].inst_rr(s["rhoY"], s["rhoH"], s["T"])
        return [s["T"], w, s["r"].heat_release(s["T"], w)]
    net = s["net"]
    loss, dW, db = net.loss_and_grads(s["x"], s["y"], s["w"])
    net.adam_step(dW, db, 2e-4)
    return [loss, dW, db, net.W, net.b]


def _prepare_train(case, g, seed):
    """A network part-way through its training's life: random weights, a batch of flame states as inputs and changes of
    the size a step of 1e-6 s makes as targets."""
    n = case["batch"]
    m, Y, T = _field("ch4", g, 64, 32, max(1, -(-n // 2048)))
    rho, _ = m.density_enthalpy(Y, T)
    pick = torch.randperm(T.numel(), device=DEV, generator=g)[:n]
    rhoY, T = (rho[:, None] * Y)[pick].t().contiguous(), T[pick].contiguous()
    dy = torch.cat([T[None] * 1e-3, (rhoY / rhoY.sum(0)) * 1e-2]).t()
    dy = (dy * torch.randn(dy.shape, dtype=torch.float64, device=DEV, generator=g)).contiguous()
    net = MLPSurrogate(MECHS["ch4"], seed=seed % (1 << 31), device=DEV)
    torch.manual_seed(seed)
    fit_normalisation(net, net.raw_features(rhoY, T, 1e-6), dy)
    x = net.features(_reactor("ch4"), rhoY, T, 1e-6, (n + 127) // 128 * 128)
    w = torch.ones(net.nout, device=DEV)
    w[0] = float(net.N)
    return {"case": case, "net": net, "x": x[:n], "y": net.encode(dy), "w": w}


def work(case):
    if case["kind"] == "train":
        n = case["batch"]
        macs = 32 * 256 + 2 * 256 * 256 + 256 * 32
        weights = macs + 3 * 256 + 32
        return {"bytes": n * (2 * 64 + 4 * 22) + 4 * weights * 7, "flops": 2.0 * n * macs * 4}
    total = {"bytes": 0.0, "flops": 0.0}
    for f, nx, ny, nz in _fields_of(case):
        key, cells = _key(f), float(nx * ny * nz)
        N = {"h2": 9, "ch4": 21, "c12": 53}[key]
        c = _counts(key)
        if case["kind"] == "rates":
            total["bytes"] += 8 * cells * (2 * N + 4)
            total["flops"] += cells * (c["rhs"] + 4 * 20 * N)
            continue
        nfe = RHS_PER_CELL.get("c12_grf" if f == "c12_grf" else "c12_boxes" if key == "c12" else key)
        nfe *= (case["dt"] / (5e-6 if f == "c12_grf" else 1e-6)) ** 0.25
        if f == "c12_cold":
            nfe /= 3
        if case["kind"] == "hybrid":
            nfe *= 0.45 if case["dt"] < 3e-6 else 0.7
            total["flops"] += cells * 8 * 4 * (32 * 256 + 2 * 256 * 256 + 256 * 32)  # two-term inputs
        total["flops"] += cells * perfmodel.flops_per_cell(c, nfe, 1.1, nfe / 4.5, nfe - 2, nfe / 1.5)
        total["bytes"] += 8 * cells * (3 * N + 8 + (5 * N + 4 if case["kind"] == "level" else 0))
    return total


@functools.lru_cache(maxsize=None)
def _counts(key):
    return perfmodel.op_counts(mechmod.flatten(mechmod.builtin(MECHS[key])))


def tolerance(case):
    if case["kind"] == "train":
        return {"rel": 2e-2, "max": 0.5}   # BF16 activations and gradients
    if case["kind"] == "rates":
        return {"rel": 1e-10, "max": 1e-8}  # 64 bits; rates are differences of large terms
    if case["kind"] == "hybrid":
        return {"rel": 1e-6, "max": 1e-3}  # cells at the edge of the acceptance rule may fall to the other side
    if case["kind"] == "level":
        return {"rel": 1e-5, "max": 1e-2}  # the reaction term is a difference over dt, at rtol 1e-6
    # step-size decisions that flip at round-off move a cell within the integrator's own error
    return {"rel": 1e-6, "max": 1e-4} if "c12" in case.get("field", "c12") else {"rel": 1e-8, "max": 1e-6}


# ------------------------------------------------------------------------------------------------- 64-bit results
def _radau(m, y, F, dt, steps=120):
    """y(dt) of every cell by the three-stage Radau IIA method (order 5) on a graded grid, full Jacobians."""
    r6 = math.sqrt(6.0)
    A = torch.tensor([[(88 - 7 * r6) / 360, (296 - 169 * r6) / 1800, (-2 + 3 * r6) / 225],
                      [(296 + 169 * r6) / 1800, (88 + 7 * r6) / 360, (-2 - 3 * r6) / 225],
                      [(16 - r6) / 36, (16 + r6) / 36, 1.0 / 9]], dtype=torch.float64, device=y.device)
    n = y.shape[1]
    eye = torch.eye(3 * n, dtype=torch.float64, device=y.device)
    jac = torch.func.vmap(torch.func.jacfwd(m.rhs))
    t = [dt * (i / steps) ** 4 for i in range(steps + 1)]
    for i in range(steps):
        h = t[i + 1] - t[i]
        J = jac(y, F)
        big = eye - h * (A[:, None, :, None] * J[:, None, :, None, :]).reshape(-1, 3 * n, 3 * n)
        lu = torch.linalg.lu_factor(big)
        Z = torch.zeros((y.shape[0], 3, n), dtype=torch.float64, device=y.device)
        for _ in range(8):
            f = m.rhs(y[:, None] + Z, F[:, None].expand_as(Z))
            res = Z - h * torch.einsum("ij,bjk->bik", A, f)
            Z = Z - torch.linalg.lu_solve(*lu, res.reshape(-1, 3 * n, 1)).reshape_as(Z)
        y = y + Z[:, 2]
    return y


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "rates":
        s = prepare(case, seed)
        m = _mech(_key(case["field"]))
        T, w, hr = torch.empty_like(s["T0"]), torch.empty_like(s["rhoY"]), torch.empty_like(s["T0"])
        for a in range(0, T.numel(), 65536):
            b = slice(a, a + 65536)
            rhoY, t = s["rhoY"][:, b].t() * 1e-3, s["T0"][b]
            rho = rhoY.sum(1)
            Y, h1 = rhoY / rho[:, None], s["rhoH"][b] * 10.0 / rho
            for _ in range(30):
                cp, h, sr = m.thermo(t)
                t = t + (h1 - (Y * h / m.mw).sum(1) * RU * t) / ((Y * cp / m.mw).sum(1) * RU)
            cp, h, sr = m.thermo(t)
            wd = m.wdot(rhoY / m.mw, t, h - sr) * m.mw
            T[b], w[:, b] = t, wd.t() * 1e3
            hr[b] = -(h * (RU * t)[:, None] / m.mw * 1e-4 * wd * 1e3).sum(1)
        return [T, w, hr]
    if case["kind"] != "react":
        return None  # networks and an acceptance rule, or box lists of too many cells for a plain solve
    n = {"h2": 10, "ch4": 22, "c12": 54}[_key(case["field"])]
    if case["nx"] * case["ny"] * case["nz"] * n * n > 3_500_000:
        return None  # too long for a plain solve
    s = prepare(dict(case, boxes=False), seed)
    m = _mech(_key(case["field"]))
    y0 = torch.cat([s["rhoY0"], s["T0"][None]]).t().contiguous()
    F = torch.cat([s["fY"], s["fH"][None]]).t().contiguous()
    out = torch.cat([_radau(m, y0[a:a + 4096], F[a:a + 4096], case["dt"]) for a in range(0, y0.shape[0], 4096)])
    res = [out[:, :-1].t().contiguous(), out[:, -1].contiguous(), s["rhoH0"] + case["dt"] * s["fH"]]
    if not case.get("boxes"):
        return res
    return [_fab(v, case["nx"], case["ny"], case["nz"], case["ghost"]) for v in res]


def _exact_train(case, seed):
    """The gradients of the same loss in FP64: the BF16 weights and inputs the state holds, everything after in 64 bits.
    The updated weights have no value of that kind (Adam's first step is the sign of the gradient)."""
    s = prepare(case, seed)
    net = s["net"]
    W = [v.double().requires_grad_() for v in net.Wb]
    b = [v.double().requires_grad_() for v in net.b]
    h = s["x"].double()
    h = h[:, :net.kin] + h[:, net.kin:]
    for li in range(4):
        h = h @ W[li].t() + b[li]
        if li < 3:
            h = torch.nn.functional.gelu(h, approximate="tanh")  # the network's activation is the tanh form
    loss = ((h[:, :net.nout] - s["y"].double()) ** 2 * s["w"].double()).sum() / h.shape[0]
    grads = torch.autograd.grad(loss, W + b)
    return [loss.detach(), list(grads[:4]), list(grads[4:]), None, None]
