"""The work that a user of droplet_gb300 has it do, as cases to be timed.

Each case is one pass through the public entry points: a stretch of time steps
that ends with the state or the fields in the caller's hands, a gradient, the
diagnostics of a field, the labels of its droplets, a restart with its
checkpoint. ``listed()`` gives the cases themselves, ``draw()`` others of the
same ranges; sizes and parameters are those of ``droplet_gb300.configs`` (or
generic ones where it has none).

Outputs of the two-phase FP32 form are its device state (``dl_save_state``);
those of the FP16 and single-phase forms are single-precision snapshots of the
fields, as a visualisation or an analysis in FP32 takes them; the FP64 form
returns its FP64 fields.
"""
import ctypes
import math

import numpy as np
import torch

from droplet_gb300.adjoint import CheckpointedRun
from droplet_gb300.ensemble import Ensemble
from droplet_gb300.params import Params, kappag_from_sigma
from droplet_gb300.solver import (Droplet, FORCE_NONE, FORCE_SPECTRAL, FORCE_STATIC, FORM_FP16, FORM_FP32,
                                  FORM_FP64)

CX = (0, 1, 0, 0, -1, 0, 0, 1, -1, 1, 1, -1, 1, -1, -1)
CY = (0, 0, 1, 0, 0, -1, 0, 1, 1, -1, 1, -1, -1, 1, -1)
CZ = (0, 0, 0, 1, 0, 0, -1, 1, 1, 1, -1, -1, -1, -1, 1)
E = (2.0 / 9.0,) + (1.0 / 9.0,) * 6 + (1.0 / 72.0,) * 8
F = (-7.0 / 3.0,) + (1.0 / 3.0,) * 6 + (1.0 / 24.0,) * 8
C = tuple(zip(CX, CY, CZ))
Q = 15
FORMS = {"fp64": FORM_FP64, "fp32": FORM_FP32, "fp16": FORM_FP16, "single32": FORM_FP32}
POP_BYTES = {"fp64": 8, "fp32": 4, "fp16": 2, "single32": 4}
MEMBER_SIZES = (48, 64, 96)
WEBERS = (2.0, 5.0, 10.0, 20.0)


def listed():
    def steps(name, form, flow, nx, ny, nz, n, drops=1):
        return dict(name=name, kind="steps", form=form, flow=flow, nx=nx, ny=ny, nz=nz, steps=n, drops=drops)

    return [
        # a small shear droplet stepped interactively: launches and latency
        steps("shear_32_fp32", "fp32", "shear", 32, 32, 32, 10),
        # the sheared droplet in the plain form, which the other forms are checked against
        steps("shear_64_fp64", "fp64", "shear", 64, 64, 64, 20),
        # the reference run of the forced turbulence in the plain form
        steps("turbulence_128_fp64", "fp64", "turbulence", 128, 128, 128, 5),
        # the same flow in production: FP32, LES, band forcing
        steps("turbulence_128_fp32", "fp32", "turbulence", 128, 128, 128, 20),
        # the vortex-forced droplet at a viscosity ratio (static force), on a box of odd sides
        steps("vortex_150x101x77_fp32", "fp32", "vortex", 150, 101, 77, 20),
        # eight droplets in a large box, FP16 storage
        steps("turbulence_256_fp16", "fp16", "turbulence", 256, 256, 256, 50, drops=8),
        # the precursor turbulence (single phase) at its full size
        steps("precursor_256_fp32", "single32", "turbulence", 256, 256, 256, 50),
        # uneven members stepped together
        dict(name="ensemble_16_fp32", kind="ensemble", members=16, steps=20),
        # gradient of the deformation: forward with every state kept, then the reverse pass
        dict(name="adjoint_96_fp32", kind="adjoint", nx=96, ny=96, nz=96, steps=40),
        # in-situ monitoring of a production run: conservation sums, dissipation, spectrum, free energy
        dict(name="diagnostics_128_fp32", kind="diagnostics", form="fp32", nx=128, ny=128, nz=128, drops=1),
        # droplet statistics of a large box with the label field
        dict(name="labels_256_fp32", kind="labels", form="fp32", nx=256, ny=256, nz=256, drops=24),
        # a restart from a checkpoint and the writing of the next one
        dict(name="checkpoint_96_fp32", kind="checkpoint", form="fp32", nx=96, ny=96, nz=96, drops=1),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi):
        return dict(nx=side(lo, hi), ny=side(lo, hi), nz=side(lo, hi))

    kind = rng.choice(("steps",) * 5 + ("ensemble", "adjoint", "diagnostics", "labels", "checkpoint"))
    if kind == "steps":
        form, flow, top = rng.choice((("fp64", "shear", 96), ("fp64", "turbulence", 128), ("fp32", "shear", 160),
                                      ("fp32", "turbulence", 200), ("fp32", "vortex", 160),
                                      ("fp16", "turbulence", 200), ("single32", "turbulence", 240)))
        return dict(kind=kind, form=form, flow=flow, **box(24, top), drops=rng.randint(1, 4),
                    steps=rng.randint(3, 10) if form == "fp64" else rng.randint(8, 32))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(4, 20), steps=rng.randint(8, 24))
    if kind == "adjoint":
        # near-cubic: the deformation is that of a droplet which fills a fair part of the box
        n = side(32, 96)
        return dict(kind=kind, **box(0.9 * n, 1.1 * n), steps=rng.randint(10, 40))
    if kind == "checkpoint":
        return dict(kind=kind, form=rng.choice(("fp64", "fp32", "fp16")), **box(24, 96), drops=rng.randint(1, 3))
    return dict(kind=kind, form=rng.choice(("fp64", "fp32", "fp16")), **(box(32, 160) if kind == "diagnostics" else box(64, 256)),
                drops=rng.randint(1, 12))


# ---- inputs -------------------------------------------------------------------
def _axes(shape, dev):
    nx, ny, nz = shape
    r = [torch.arange(n, dtype=torch.float64, device=dev) for n in (nx, ny, nz)]
    return r[0].view(1, 1, nx), r[1].view(1, ny, 1), r[2].view(nz, 1, 1)


def _droplets(P, shape, drops, radius, rng, dev, spread=0.0, width=2.0):
    """phi of tanh-profile droplets at seeded places (one: near the centre)."""
    n = shape
    axes = _axes(shape, dev)
    pt = torch.full((n[2], n[1], n[0]), -1.0, dtype=torch.float64, device=dev)
    m = 1
    while m ** 3 < drops:
        m += 1
    if m > 1:  # one droplet per cell of an m^3 grid, none touching its neighbour
        radius = min(radius, 0.34 / (1.0 + spread) * min(n) / m)
    for cell in rng.permutation(m ** 3)[:drops]:
        at = np.array([cell % m, cell // m % m, cell // m ** 2])
        off = rng.uniform(-2.0, 2.0, 3) if m == 1 else ((at + 0.5) / m - 0.5 + rng.uniform(-0.08, 0.08, 3) / m) * n
        r = radius * (1.0 + spread * rng.uniform(-1.0, 1.0))
        d2 = 0.0
        for a, v, o in zip(axes, n, off):
            d = (a - ((v - 1) / 2.0 + o)).abs()
            d = torch.minimum(d, v - d)
            d2 = d2 + d * d
        pt = torch.maximum(pt, torch.tanh((r - d2.sqrt()) / width))
    return P.phi1 + (P.phi2 - P.phi1) * (pt + 1.0) / 2.0


def _turbulence(shape, urms, rng, dev):
    """Random-phase solenoidal velocity on 1 <= |k| <= 2, scaled to urms per component."""
    n = shape
    axes = _axes(shape, dev)
    u = [torch.zeros((n[2], n[1], n[0]), dtype=torch.float64, device=dev) for _ in range(3)]
    for kx in range(-2, 3):
        for ky in range(-2, 3):
            for kz in range(0, 3):
                kk = kx * kx + ky * ky + kz * kz
                if not 1 <= kk <= 4 or (kz == 0 and (ky < 0 or (ky == 0 and kx < 0))):
                    continue
                k = np.array([kx / n[0], ky / n[1], kz / n[2]])
                a, b = rng.standard_normal(3), rng.standard_normal(3)
                a, b = a - k * (k @ a) / (k @ k), b - k * (k @ b) / (k @ k)
                ph = 2.0 * math.pi * (k[0] * axes[0] + k[1] * axes[1] + k[2] * axes[2])
                c, s = torch.cos(ph), torch.sin(ph)
                for q in range(3):
                    u[q] += a[q] * c + b[q] * s
    rms = math.sqrt(sum(float((v * v).mean()) for v in u) / 3.0)
    return [v * (urms / rms) for v in u]


def _physics(case, rng):
    """Parameters and force mode of a case's flow."""
    flow = case.get("flow") or {"adjoint": "shear"}.get(case["kind"], "turbulence")
    P = Params.lbm_drop_xy().replace(kappaf=0.01)
    small = min(case["nx"], case["ny"], case["nz"])
    radius = 0.1875 * small if case.get("drops", 1) == 1 else max(5.0, 0.0625 * small)
    if flow == "shear":  # moving walls, tau_g = 0.8, Ca = 0.3
        nu, U = 0.1, 0.05
        P = P.replace(tauf=1.0, nu1=nu, nu2=nu, walls=True, wall_u=(U, 0.0, 0.0),
                      kappag=kappag_from_sigma(2.0 * U / (case["nz"] - 1) * nu * radius / 0.3))
        return P, FORCE_NONE, radius
    if flow == "vortex":  # static force, dispersed phase half as viscous, range from the previous step
        P = P.replace(tauf=0.7, nu1=0.1, nu2=0.05, kappag=2e-3)
        return P, FORCE_STATIC, radius
    if case.get("form") == "single32":  # precursor: nu = 0.001
        P = P.replace(nu1=0.001, nu2=0.001, kappaf=0.0, kappag=0.0, eps=1e-9, kc=3, visc_mode=1)
        return P, FORCE_SPECTRAL, radius
    nu = 0.02 / 3.0  # LES, band forcing
    we = case.get("we", 5.0)
    P = P.replace(tauf=0.7, nu1=nu, nu2=nu, les=True, Cs=0.1, delta=1.0, eps=2e-7, kc=3,
                  kappag=kappag_from_sigma(1e-4 * 2.0 * radius / we))
    return P, FORCE_SPECTRAL, radius


def _inputs(case, seed):
    """(params, shape, force mode, force arrays, phi, u, p): FP64 tensors on the GPU where there is one."""
    rng = np.random.default_rng([int(seed), 77])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    shape = (case["nx"], case["ny"], case["nz"])
    P, mode, radius = _physics(case, rng)
    many = case["kind"] == "labels"
    phi = _droplets(P, shape, case.get("drops", 1), radius, rng, dev, spread=0.5 if many else 0.0)
    if case.get("form") == "single32":
        phi = torch.full_like(phi, P.phi1)
    u = _turbulence(shape, 1e-4 if case.get("form") == "single32" else (2e-3 if mode != FORCE_SPECTRAL else 1e-2), rng,
                    dev)
    if case["kind"] == "diagnostics":  # a mean drift: the momentum sums are then not rounding alone
        u = [v + 2e-3 * rng.uniform(0.5, 1.5) for v in u]
    if P.walls:  # the linear profile between the walls
        z = torch.arange(shape[2], dtype=torch.float64, device=dev).view(-1, 1, 1)
        u[0] = u[0] + P.wall_u[0] * (2.0 * z / (shape[2] - 1) - 1.0)
    p = 1.0 / 3.0 + 1e-5 * torch.cos(2.0 * math.pi * _axes(shape, dev)[0] / shape[0]) + torch.zeros_like(phi)
    force = None
    if mode == FORCE_STATIC:  # externalforce of the vortex program: one cell over the box
        x, _, z = _axes(shape, dev)
        kx, kz, amp = 2.0 * math.pi / shape[0], 2.0 * math.pi / shape[2], 2e-6
        force = [amp * torch.sin(kx * x) * torch.cos(kz * z) + torch.zeros_like(phi), torch.zeros_like(phi),
                 -amp * torch.cos(kx * x) * torch.sin(kz * z) + torch.zeros_like(phi)]
    return P, shape, mode, force, phi, u, p


def _host(t):
    return t.cpu().numpy()


def _start(sim, inp):
    _, _, mode, force, phi, u, p = inp
    sim.set_fields(_host(phi), *[_host(v) for v in u], _host(p))
    sim.init_equilibrium()
    sim.set_force(mode, *([_host(v) for v in force] if force else []))


def _members(case, seed):
    """One case per member: size, Weber number and seed drawn from the case's own."""
    rng = np.random.default_rng(4)
    out = []
    for m in range(case["members"]):
        n, we = int(rng.choice(MEMBER_SIZES)), float(rng.choice(WEBERS))
        out.append((dict(kind="steps", form="fp32", flow="turbulence", nx=n, ny=n, nz=n, drops=1, we=we),
                    int(seed) * 1000 + m))
    return out


class _State:
    """Device copy of a two-phase FP32 state (dl_save_state), as its parts."""

    def __init__(self, sim):
        n = ctypes.c_int64()
        sim._call("state_floats", ctypes.byref(n))
        self.buf = torch.empty(int(n.value), dtype=torch.float32, device="cuda")
        s = sim.shape3
        pops = Q * sim.n_sites
        self.parts = {"f": self.buf[:pops].view(Q, *s), "g": self.buf[pops:2 * pops].view(Q, *s),
                      "fields": self.buf[2 * pops:].view(5, *s)}

    def save(self, sim):
        sim._call("save_state", ctypes.c_void_p(self.buf.data_ptr()))
        return self.parts


class _Snapshot:
    """Page-locked FP64 fields of the caller, and their copy in single precision."""

    def __init__(self, sim, single):
        self.f64 = torch.empty((5,) + sim.shape3, dtype=torch.float64, pin_memory=True)
        self.f32 = torch.empty_like(self.f64, dtype=torch.float32) if single else None
        self.into = dict(zip(("phi", "u1", "u2", "u3", "p"), self.f64.numpy()))

    def save(self, sim):
        sim.get_fields_into(self.into)
        if self.f32 is not None:
            self.f32.copy_(self.f64)
        v = self.f64 if self.f32 is None else self.f32
        return {"phi": v[0], "u": v[1:4], "p": v[4]}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        inps = [_inputs(c, s) for c, s in _members(case, seed)]
        ens = Ensemble([i[0] for i in inps], [i[1] for i in inps], FORM_FP32)
        for sim, inp in zip(ens.members, inps):
            _start(sim, inp)
        return dict(case=case, ens=ens, out=[_State(m) for m in ens.members])
    inp = _inputs(case, seed)
    P, shape, _, _, phi, u, p = inp
    if kind == "adjoint":
        run_ = CheckpointedRun(P, shape, [_host(v) for v in u], _host(p), case["steps"])
        return dict(case=case, run=run_, phi0=_host(phi))
    form = case["form"]
    sim = Droplet(P, shape, FORMS[form], single_phase=form == "single32")
    _start(sim, inp)
    st = dict(case=case, sim=sim)
    if kind == "steps":
        st["out"] = _State(sim) if form == "fp32" else _Snapshot(sim, form != "fp64")
    elif kind == "checkpoint":
        # the record of a run three steps in, as the restarted program reads it
        sim.step(3)
        st["f"], st["g"] = sim.get_populations()
    return st


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        return [o.save(m) for o, m in zip(state["out"], state["ens"].members)]
    if kind == "adjoint":
        r = state["run"]
        D = r.forward(state["phi0"])
        return {"D": D, "grads": r.backward(download=False)}
    sim = state["sim"]
    if kind == "steps":
        sim.step(case["steps"])
        return state["out"].save(sim)
    if kind == "diagnostics":
        return {"sums": sim.reduce(), "energy": sim.energy()}
    if kind == "labels":
        volumes, labels = sim.label_droplets(14, labels=True)
        return {"volumes": volumes, "labels": labels}
    sim.set_populations(state["f"], state["g"])
    f, g = sim.get_populations()
    return {"f": f, "g": g}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        ws = [work(dict(c, steps=case["steps"])) for c, _ in _members(case, 0)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "adjoint":
        # forward: 30 populations read and written, 20 values of state kept; reverse: 30 adjoints read and
        # written, the state read
        return {"bytes": 4.0 * n * case["steps"] * (60 + 20 + 60 + 20), "flops": 1200.0 * n * case["steps"]}
    form = case["form"]
    b = POP_BYTES[form]
    if kind == "steps":
        pops = 15 if form == "single32" else 30
        out = {"fp64": 40, "fp32": 140, "fp16": 40, "single32": 40}[form]  # the result, written once
        flops = 200 if form == "single32" else 450 + (200 if case["flow"] == "turbulence" else 0)
        return {"bytes": float(n) * (2 * pops * b * case["steps"] + out), "flops": float(n) * flops * case["steps"]}
    field = 8 if form == "fp64" else 4
    if kind == "diagnostics":  # five fields read; three real transforms
        return {"bytes": 5.0 * field * n, "flops": n * (150.0 + 3 * 2.5 * math.log2(n))}
    if kind == "labels":
        return {"bytes": n * (field + 4.0), "flops": 30.0 * n}
    return {"bytes": n * 30 * (8.0 + b + b + 8.0), "flops": 60.0 * n}


# ---- the same in 64 bits, with plain torch --------------------------------------
def _at(a, i, s=1):
    """a at x + s c_i (periodic); a: (..., nz, ny, nx)."""
    return a if i == 0 else torch.roll(a, (-s * CZ[i], -s * CY[i], -s * CX[i]), (-3, -2, -1))


def _grad(a, P):
    out = []
    shifted = [None] + [_at(a, i) for i in range(1, Q)]
    for q in range(3):
        out.append(sum(C[i][q] * shifted[i] for i in range(1, Q) if C[i][q]) / (10.0 * P.ds))
    return out, (sum(shifted[1:]) - 14.0 * a) / (5.0 * P.ds ** 2)


def _dot(c, v):
    return sum(k * w for k, w in zip(c, v) if k) if any(c) else torch.zeros_like(v[0])


def _equilibria(P, phi, u, p, single, kf, kg):
    g = []
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    if single:
        for i in range(Q):
            cu = _dot(C[i], u)
            g.append(E[i] * (3.0 * p + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq))
        return None, g
    gr, lap = _grad(phi, P)
    gsq = gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2]
    A = phi * P.T / (1.0 - P.b * phi) - P.a * phi * phi - kf * phi * lap - kf / 6.0 * gsq
    f = []
    for i in range(Q):
        cu, cg = _dot(C[i], u), _dot(C[i], gr)
        G = 4.5 * cg * cg - 1.5 * sum(k * k for k in C[i]) * gsq
        f.append((phi if i == 0 else 0.0) + F[i] * A + 3.0 * E[i] * phi * cu + E[i] * kf * G)
        g.append(E[i] * (3.0 * p + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq) + E[i] * kg * G)
    return f, g


def _moments(f, g, phi):
    return (phi if f is None else sum(f), [sum(C[i][q] * g[i] for i in range(Q) if C[i][q]) for q in range(3)],
            sum(g) / 3.0)


def _tau(P, phi, u, rng):
    nu = (phi - rng[0]) / (rng[1] - rng[0]) * (P.nu2 - P.nu1) + P.nu1
    if P.les:
        d = [_grad(v, P)[0] for v in u]
        ss = sum((0.5 * (d[a][b] + d[b][a])) ** 2 for a in range(3) for b in range(3))
        nu = nu + (P.Cs * P.delta) ** 2 * torch.sqrt(2.0 * ss)
    return 0.5 + 3.0 * nu / P.ds


def _band_force(P, u):
    nz, ny, nx = u[0].shape
    k = [torch.fft.fftfreq(n, 1.0 / n, device=u[0].device, dtype=torch.float64) for n in (nz, ny, nx)]
    kk = k[0].view(-1, 1, 1) ** 2 + k[1].view(1, -1, 1) ** 2 + k[2].view(1, 1, -1) ** 2
    band = ((kk >= 1) & (kk < P.kc ** 2)).to(torch.float64)
    n = nx * ny * nz
    h = [torch.fft.fftn(v) / n * band for v in u]
    en = 0.5 * sum((v.real ** 2 + v.imag ** 2).sum() for v in h)
    return [torch.fft.ifftn(v).real * (n * 0.5 * P.eps / en) for v in h]


def _walls(g, step, P, U):
    on = 1.0 if step >= P.wall_start else 0.0
    for pairs, plane, sign in (((3, 6), (7, 11), (8, 12), (9, 13), (14, 10)), 0, -1.0), \
            (((6, 3), (10, 14), (11, 7), (12, 8), (13, 9)), -1, 1.0):
        src = [g[j] for _, j in pairs]
        for (i, j), s in zip(pairs, src):
            w = 6.0 * E[j] * sign * on * sum(U[q] * C[j][q] for q in range(3))
            keep = s[plane] - w
            g[i] = torch.cat([keep[None], g[i][1:]]) if plane == 0 else torch.cat([g[i][:-1], keep[None]])
    return g


def _steps(P, single, mode, force, phi, u, p, n, kf=None, kg=None, tauf=None, U=None):
    """f, g, phi, u, p after n steps from equilibrium."""
    kf = P.kappaf if kf is None else kf
    kg = P.kappag if kg is None else kg
    tauf = P.tauf if tauf is None else tauf
    U = P.wall_u if U is None else (U, 0.0, 0.0)
    f, g = _equilibria(P, phi, u, p, single, kf, kg)
    rng = (P.phi1, P.phi2)
    phi, u, p = _moments(f, g, phi)
    for s in range(1, n + 1):
        fe, ge = _equilibria(P, phi, u, p, single, kf, kg)
        tau = _tau(P, phi, u, rng)
        Fv = _band_force(P, u) if mode == FORCE_SPECTRAL else force
        gn = []
        for i in range(Q):
            v = g[i] - (g[i] - ge[i]) / tau
            if Fv is not None and i:
                v = v + 3.0 * P.ds * E[i] * _dot(C[i], Fv)
            gn.append(_at(v, i, -1))
        g = _walls(gn, s, P, U) if P.walls else gn
        if f is not None:
            f = [_at(f[i] - (f[i] - fe[i]) / tauf, i, -1) for i in range(Q)]
        phi, u, p = _moments(f, g, phi)
        if P.nu1 != P.nu2 and not P.visc_mode:
            rng = (min(P.phi2, float(phi.min())), max(P.phi1, float(phi.max())))
    return f, g, phi, u, p


def _state64(P, f, g, phi, u, p):
    p0 = P.phi1 * P.T / (1.0 - P.b * P.phi1) - P.a * P.phi1 ** 2
    return {"f": torch.stack([f[i] - ((P.phi1 if i == 0 else 0.0) + F[i] * p0) for i in range(Q)]),
            "g": torch.stack([g[i] - E[i] for i in range(Q)]),
            "fields": torch.stack([phi - P.phi1, *u, p - 1.0 / 3.0])}


def _deformation(P, phi):
    x, y, z = _axes(phi.shape[::-1], phi.device)
    w = (phi - P.phi1) / (P.phi2 - P.phi1)
    W = w.sum()
    m = [(w * a).sum() / W for a in (x, y, z)]
    S = torch.stack([torch.stack([(w * (a - ma) * (b - mb)).sum() / W for b, mb in zip((x, y, z), m)])
                     for a, ma in zip((x, y, z), m)])
    lam = torch.linalg.eigvalsh(S)
    a, b = lam[-1].sqrt(), lam[0].sqrt()
    return (a - b) / (a + b)


def _sums64(P, phi, u, p):
    x, y, z = _axes(phi.shape[::-1], phi.device)
    w = (phi - P.phi1) / (P.phi2 - P.phi1)
    d = [_grad(v, P)[0] for v in u]
    ss = sum((0.5 * (d[a][b] + d[b][a])) ** 2 for a in range(3) for b in range(3))
    inside, outside = w > 0.95, w < 0.05
    r = {"phi_sum": phi.sum(), "p_sum": p.sum(), "mom": [v.sum() for v in u],
         "ke": 0.5 * sum((v * v).sum() for v in u),
         "diss": (2.0 * (P.nu1 + w * (P.nu2 - P.nu1)) * ss).sum(),
         "vol_count": (phi > 0.5 * (P.phi1 + P.phi2)).sum(), "vol_smooth": w.sum(),
         "phi_min": phi.min(), "phi_max": phi.max(), "p_in": p[inside].sum(), "n_in": inside.sum(),
         "p_out": p[outside].sum(), "n_out": outside.sum(), "w_sum": w.sum(),
         "w_x": [(w * a).sum() for a in (x, y, z)],
         "w_xx": [(w * a * b).sum() for a, b in ((x, x), (y, y), (z, z), (x, y), (x, z), (y, z))]}
    return {k: [float(e) for e in v] if isinstance(v, list) else float(v) for k, v in r.items()}


def _energy64(P, phi, u):
    nz, ny, nx = phi.shape
    nb = nx // 2 + 1
    e2 = sum(torch.fft.fftn(v).abs() ** 2 for v in u)[: nz // 2 + 1] / float(nx * ny * nz) ** 2

    def signed(n, m):
        k = torch.arange(m, device=phi.device)
        return torch.where(k >= n // 2 + 1, k - n, k)

    k = signed(nz, nz // 2 + 1).view(-1, 1, 1) ** 2 + signed(ny, ny).view(1, -1, 1) ** 2 + signed(nx, nx).view(1, 1, -1) ** 2
    b = k.double().sqrt().long()
    e2 = 0.5 * e2 * 2.0
    e2[0] *= 0.5
    ok = b < nb
    spec = torch.zeros(nb, dtype=torch.float64, device=phi.device).index_add_(0, b[ok], e2[ok])
    gr, lap = _grad(phi, P)
    lg, omb = torch.log(phi / (1.0 - P.b * phi)), 1.0 - P.b * phi
    return {"psi_sum": float((phi * P.T * lg - P.a * phi * phi).sum()),
            "mu_sum": float((P.T * lg + P.T / omb - 2.0 * P.a * phi - P.kappag * lap).sum()),
            "grad_sq_sum": float((gr[0] ** 2 + gr[1] ** 2 + gr[2] ** 2).sum()), "spectrum_sum": float(spec.sum()),
            "spectrum": spec}


def exact(case, seed):
    kind = case["kind"]
    if kind == "labels":
        return None  # whole numbers only
    if kind == "ensemble":
        return [exact(dict(c, steps=case["steps"]), s) for c, s in _members(case, seed)]
    P, _, mode, force, phi, u, p = _inputs(case, seed)
    if kind == "adjoint":
        leaf = [torch.tensor(v, dtype=torch.float64, device=phi.device, requires_grad=True)
                for v in (P.kappaf, P.kappag, P.tauf, P.wall_u[0])]
        phi.requires_grad_(True)
        D = _deformation(P, _steps(P, False, mode, None, phi, u, p, case["steps"], *leaf)[2])
        D.backward()
        g = [float(v.grad) for v in leaf]
        return {"D": float(D.detach()), "grads": {"dphi0": phi.grad, "dkappaf": g[0], "dkappag": g[1], "dtauf": g[2],
                                         "dmobility": g[2] / P.ds, "dU": g[3]}}
    with torch.no_grad():
        if kind == "diagnostics":
            return {"sums": _sums64(P, phi, u, p), "energy": _energy64(P, phi, u)}
        if kind == "checkpoint":
            f, g, *_ = _steps(P, False, mode, force, phi, u, p, 3)
            return {"f": torch.stack(f, -1), "g": torch.stack(g, -1)}
        f, g, phi, u, p = _steps(P, case["form"] == "single32", mode, force, phi, u, p, case["steps"])
        if case["form"] == "fp32":
            return _state64(P, f, g, phi, u, p)
        return {"phi": phi, "u": torch.stack(u), "p": p}
