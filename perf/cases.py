"""Timed cases of the time step and the operators around it, through the public entry points (``Box``, ``Ensemble``).

A case is a dict: ``kind`` says which call is timed, ``nx, ny, nz`` the grid (``nbox`` boxes of each size for an
ensemble), ``precision`` the form, and the rest are options of that call.  Inputs are seeded synthetic velocity fields
(white noise shaped to E(k) ~ k^4 exp(-2 k^2 / k0^2), solenoidal, dealiased, kinetic energy 0.5) built with torch
alone; ``exact`` is the same mathematics in 64-bit torch.
"""
import math

import numpy as np
import torch

from dnsbox_b200.ensemble import Ensemble
from dnsbox_b200.ops import Box

SIZES = (16, 24, 32, 48, 64, 96, 128, 192, 256, 512)
PRECISION_BYTES = {"fp64": 16, "fp32": 8, "tc_split": 8}   # of a complex value


def _case(kind, n, precision, **kw):
    nx, ny, nz = n if isinstance(n, tuple) else (n, n, n)
    return dict({"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision}, **kw)


def listed():
    step = dict(stepper="heun", cfl=True, bandlim=True, nu=2e-3, tune=False, records=False)
    return [
        # a small box between two outputs of a parameter study: launches and latency count
        _case("step", 32, "fp32", name="step_32_fp32", **dict(step, nsteps=10, nu=1e-2)),
        # a double-precision validation run with its step records (Ekin.dat rows) read back
        _case("step", 64, "fp64", name="step_64_fp64_ab2", **dict(step, stepper="ab2", nsteps=8, nu=5e-3, records=True)),
        # an anisotropic box on a ragged grid (no two axes alike, none a power of two)
        _case("step", (192, 48, 96), "fp32", name="step_192x48x96_fp32", alpha_x=0.5, alpha_y=2.0, alpha_z=1.0,
              **dict(step, nsteps=4, nu=5e-3)),
        # the forced-turbulence workload of the benchmark, tuned as its program does
        _case("step", 256, "tc_split", name="step_256_tc", **dict(step, nsteps=4, tune=True)),
        # the same in double precision, with the step records
        _case("step", 256, "fp64", name="step_256_fp64", **dict(step, nsteps=2, tune=True, records=True)),
        # the benchmark's larger box
        _case("step", 512, "fp32", name="step_512_fp32", **dict(step, nsteps=1, nu=8e-4, tune=True)),
        # 96 decaying boxes (32 each of 32^3, 64^3, 96^3) advanced together
        _case("ensemble", 96, "fp32", name="ensemble_32_64_96", nbox=32, nsteps=2),
        # one right-hand side as an operator (torch code around it): the full, unpruned passes
        _case("rhs", 128, "fp32", name="rhs_128_fp32", bandlim=True),
        # objective and gradient of the steady-state search: a forward and a transposed right-hand side
        _case("residual_grad", 64, "fp64", name="residual_grad_64_fp64", bandlim=False, nu=2.5e-2),
        # the backward pass of a time horizon, as in the periodic-orbit search
        _case("horizon_grad", 96, "fp32", name="horizon_grad_96_fp32", bandlim=False, nu=2.5e-2, nsteps=16, every=8),
        # the transforms alone: one field to physical space, one back
        _case("fft", 256, "fp32", name="fft_256_fp32"),
        # what a run saves between steps: spectrum, energy, dissipation, Courant number, divergence
        _case("diagnostics", 128, "fp64", name="diagnostics_128_fp64"),
    ]


def _points(c):
    return c["nx"] * c["ny"] * c["nz"]


def _grid(rng, most):
    """Three axis lengths, the geometric mean spread over the range, at most `most` points; half of them cubic."""
    while True:
        i = rng.randrange(len(SIZES))
        if rng.random() < 0.5:
            n = (SIZES[i],) * 3
        else:
            n = tuple(SIZES[min(len(SIZES) - 1, max(0, i + rng.choice((-2, -1, 0, 0, 1, 2))))] for _ in range(3))
        if n[0] * n[1] * n[2] <= most:
            return n


def draw(rng):
    kind = rng.choice(("step",) * 6 + ("ensemble", "rhs", "vjp", "residual_grad", "horizon_grad", "fft", "diagnostics"))
    nu = round(10 ** rng.uniform(-3, -1.5), 6)
    precision = rng.choice(("fp32", "fp32", "fp64"))
    if kind == "step":
        n = _grid(rng, 256 ** 3 if precision == "fp64" else 512 * 512 * 256)
        cubic = n[0] == n[1] == n[2]
        if cubic and n[0] in (128, 256) and precision == "fp32" and rng.random() < 0.5:
            precision = "tc_split"
        c = _case(kind, n, precision, stepper=rng.choice(("heun", "heun", "ab2")), cfl=rng.random() < 0.7,
                  bandlim=rng.random() < 0.7, nu=nu, tune=cubic and n[0] >= 128,
                  records=precision == "fp64" and rng.random() < 0.5, spherical=rng.random() < 0.15)
        if not cubic and rng.random() < 0.5:
            c.update(alpha_x=rng.choice((0.5, 1.0)), alpha_y=rng.choice((1.0, 2.0)), alpha_z=1.0)
        c["nsteps"] = max(1, min(rng.randint(1, 10), int(1.0e8 / (_points(c) * (2 if precision == "fp64" else 1)))))
        return c
    if kind == "ensemble":
        return _case(kind, rng.choice((48, 64, 96)), "fp32", nbox=rng.randint(2, 32), nsteps=rng.randint(1, 2))
    if kind == "rhs":
        return _case(kind, _grid(rng, 256 ** 3), precision, bandlim=rng.random() < 0.5)
    if kind == "vjp":
        return _case(kind, _grid(rng, 128 ** 3), precision, bandlim=False)
    if kind == "residual_grad":
        return _case(kind, _grid(rng, 128 ** 3), "fp64", bandlim=False, nu=nu)
    if kind == "horizon_grad":
        n = _grid(rng, 64 ** 3 if precision == "fp64" else 96 ** 3)
        return _case(kind, n, precision, bandlim=False, nu=nu, nsteps=rng.randint(2, 16),
                     every=rng.choice((1, 4, 8, 32)))
    if kind == "fft":
        return _case(kind, _grid(rng, 256 ** 3), precision)
    return _case("diagnostics", _grid(rng, 256 ** 3), "fp64")


# ------------------------------------------------------------------ inputs
def _alpha(c):
    return c.get("alpha_x", 1.0), c.get("alpha_y", 1.0), c.get("alpha_z", 1.0)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Grid:
    """Wavenumbers (Nyquist entry 0), masks and transforms of one box in 64 bits."""

    def __init__(self, nx, ny, nz, alpha=(1.0, 1.0, 1.0), spherical=False):
        d = _device()
        self.n, self.alpha, self.spherical = (nx, ny, nz), alpha, spherical
        self.s = 1.0 / float(nx * ny * nz)

        def full(n, a):
            k = torch.arange(n, dtype=torch.float64, device=d)
            k = torch.where(k < n // 2, k, k - n) * a
            k[n // 2] = 0.0
            return k
        kx = torch.arange(nx // 2 + 1, dtype=torch.float64, device=d) * alpha[0]
        kx[nx // 2] = 0.0
        self.kx, self.ky, self.kz = kx, full(ny, alpha[1])[:, None], full(nz, alpha[2])[:, None, None]
        self.k2 = self.kx ** 2 + self.ky ** 2 + self.kz ** 2
        self.zero = self.k2 == 0
        self.k2s = torch.where(self.zero, 1.0, self.k2)
        cut = [(m / 2.0) * (2.0 * a / 3.0) for m, a in zip(self.n, alpha)]
        self.mask = (self.kx.abs() >= cut[0]) | (self.ky.abs() >= cut[1]) | (self.kz.abs() >= cut[2]) | self.zero
        if spherical:
            self.mask = self.mask | (self.k2 >= ((nx / 2.0) * 0.5 * alpha[0]) ** 2)
        self.w = torch.where(self.kx == 0, 1.0, 2.0).to(torch.float64)   # half-spectrum multiplicity

    def c2r(self, f):
        nx, ny, nz = self.n
        return torch.fft.irfftn(f, s=(nz, ny, nx), dim=(-3, -2, -1), norm="forward")

    def r2c(self, f):
        return torch.fft.rfftn(f, dim=(-3, -2, -1))

    def curl(self, u):
        kx, ky, kz = self.kx, self.ky, self.kz
        return 1j * (ky * u[2] - kz * u[1]), 1j * (kz * u[0] - kx * u[2]), 1j * (kx * u[1] - ky * u[0])

    def project(self, n):
        q = (self.kx * n[0] + self.ky * n[1] + self.kz * n[2]) / self.k2s
        return torch.stack([n[0] - self.kx * q, n[1] - self.ky * q, n[2] - self.kz * q])

    def energy(self, u):
        """Kinetic energy per box (the kx = 0 plane half weighted)."""
        return ((u.abs() ** 2).sum(0) * (0.5 * self.w)).sum((-3, -2, -1)) * self.s ** 2


def _field(g, gen, k0=3.0, boxes=None, solenoidal=True):
    """Velocity with E(k) ~ k^4 exp(-2 k^2 / k0^2) in expectation and energy 0.5, complex128 (3[, boxes], nz, ny, nxh)."""
    nx, ny, nz = g.n
    shape = (3,) if boxes is None else (3, boxes)
    noise = torch.randn(shape + (nz, ny, nx), generator=gen, device=_device(), dtype=torch.float64)
    u = g.r2c(noise)
    del noise
    amp = torch.sqrt(g.k2) * torch.exp(-g.k2 / (k0 * k0))
    u *= torch.where(g.mask, 0.0, amp)
    u[..., nx // 2] = 0
    u[..., ny // 2, :] = 0
    u[..., nz // 2, :, :] = 0
    if solenoidal:
        u = g.project(u)
    e = g.energy(u)
    u *= torch.sqrt(0.5 / e)[..., None, None, None]
    return u


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _case_grid(c):
    return _Grid(c["nx"], c["ny"], c["nz"], _alpha(c), c.get("spherical", False))


def _cdtype(c):
    return torch.complex128 if c["precision"] == "fp64" else torch.complex64


def _inputs(c, seed):
    """The tensors a program has before the call, in the precision of the form."""
    gen, g = _generator(seed), _case_grid(c)
    kind = c["kind"]
    if kind == "fft":
        spec = _field(g, gen)[0]
        phys = torch.randn(c["nz"], c["ny"], c["nx"], generator=gen, device=_device(), dtype=torch.float64)
        cd = _cdtype(c)
        return {"spec": spec.to(cd).contiguous(), "phys": phys.to(cd.to_real())}
    u = _field(g, gen, solenoidal=kind != "diagnostics")
    out = {"u": u.to(_cdtype(c)).contiguous()}
    if kind in ("vjp", "horizon_grad"):
        out["g"] = _field(g, gen, k0=6.0).to(_cdtype(c)).contiguous()
    return out


def _ensemble_sizes(c):
    return tuple(n for n in (32, 64, 96) if n <= c["nx"]) if c["nx"] == 96 else (32, c["nx"])


def _ensemble_inputs(c, seed):
    gen = _generator(seed)
    out = []
    for n in _ensemble_sizes(c):
        nus = np.exp(np.random.Generator(np.random.PCG64(seed + n)).uniform(math.log(5e-3), math.log(5e-2), c["nbox"]))
        u = _field(_Grid(n, n, n), gen, boxes=c["nbox"])
        out.append((n, nus, u.to(_cdtype(c)).contiguous()))
    return out


DT, DT_MAX, COURANT, KCUT, PIN = 1e-3, 1e-2, 0.5, 2.5, 0.1


def _box(c, **kw):
    return Box(nx=c["nx"], ny=c["ny"], nz=c["nz"], precision=c["precision"], alpha=_alpha(c), kCutOff=KCUT, Pin=PIN,
               bandlim=c.get("bandlim", True), spherical=c.get("spherical", False), nu=c.get("nu", 5e-3), dt=DT,
               courant_min=COURANT, courant_max=COURANT, dt_max=DT_MAX, tstep_fix=not c.get("cfl", False), **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        groups = []
        for n, nus, u in _ensemble_inputs(case, seed):
            box = Box(n, precision=case["precision"], nbatch=case["nbox"], nu=float(np.mean(nus)), bandlim=False,
                      tstep_fix=True, dt=DT)
            box.set_batch_nu(nus)
            groups.append((box, u))
        return {"case": case, "groups": groups, "ens": Ensemble(groups)}
    state = _inputs(case, seed)
    if kind == "step":
        box = _box(case, stepper=case["stepper"], ab2="standard")
        if case["tune"]:
            box.autotune(state["u"])
    else:
        box = _box(case)
    return dict(state, case=case, box=box)


def _records(recs):
    cols = ("t", "dt", "ekin", "dissipation", "injected_power", "courant", "eband")
    return dict({k: np.array([r[k] for r in recs]) for k in cols}, umax=np.array([r["umax"] for r in recs]))


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "ensemble":
        state["ens"].run(c["nsteps"])
        return [u for _, u in state["groups"]]
    box = state["box"]
    if kind == "step":
        recs = box.step(state["u"], c["nsteps"], diag=c["records"])
        return {"u": state["u"], "records": _records(recs)} if c["records"] else {"u": state["u"]}
    if kind == "rhs":
        return box.rhs_nonlinear(state["u"], want_eband=False)[0]
    if kind == "vjp":
        return box.rhs_nonlinear_vjp(state["u"], state["g"])
    if kind == "residual_grad":
        return box.residual_grad(state["u"])
    if kind == "horizon_grad":
        return box.heun_steps_vjp(state["u"], c["nsteps"], state["g"], every=c["every"], want_uT=True)
    if kind == "fft":
        return box.c2r(state["spec"]), box.r2c(state["phys"])
    return {"spectrum": box.spectrum(state["u"]), "kinetic": box.kinetic(state["u"]),
            "dissipation": box.dissipation(state["u"]), "courant": box.courant(state["u"], DT),
            "divergence": box.divergence(state["u"])}


# ------------------------------------------------------------------ what a pass cannot do without
def _fft_flops(p):
    return 2.5 * p * math.log2(p)   # one real 3D transform


def _step_work(points, nxh_points, cbytes, rhs):
    state = 3 * nxh_points * cbytes
    return 2 * state, rhs * (9 * _fft_flops(points) + 15 * points + 90 * nxh_points) + 30 * nxh_points


def work(case):
    c, kind = case, case["kind"]
    cb = PRECISION_BYTES[c["precision"]]
    if kind == "ensemble":
        b = f = 0.0
        for n in _ensemble_sizes(c):
            sb, sf = _step_work(n ** 3, n * n * (n // 2 + 1), cb, 2)
            b, f = b + c["nbox"] * c["nsteps"] * sb, f + c["nbox"] * c["nsteps"] * sf
        return {"bytes": b, "flops": f}
    p, h = _points(c), c["nz"] * c["ny"] * (c["nx"] // 2 + 1)
    fwd_bytes, fwd = _step_work(p, h, cb, 1)
    adj = 15 * _fft_flops(p) + 30 * p + 120 * h    # one transposed right-hand side
    if kind == "step":
        ab2 = c["stepper"] == "ab2"
        b, f = _step_work(p, h, cb, 1 if ab2 else 2)
        b += 2 * 3 * h * cb if ab2 else 0           # the previous nonlinear term, read and written
        return {"bytes": b * c["nsteps"], "flops": f * c["nsteps"]}
    if kind == "rhs":
        return {"bytes": fwd_bytes, "flops": fwd}
    if kind == "vjp":
        return {"bytes": 9 * h * cb, "flops": adj}
    if kind == "residual_grad":
        return {"bytes": fwd_bytes, "flops": fwd + adj}
    if kind == "horizon_grad":                      # per step: the forward step, one more right-hand side, two transposes
        return {"bytes": c["nsteps"] * 12 * h * cb, "flops": c["nsteps"] * (3 * fwd + 2 * adj)}
    if kind == "fft":
        return {"bytes": 2 * (h * cb + p * cb // 2), "flops": 2 * _fft_flops(p)}
    return {"bytes": 3 * h * cb, "flops": 4 * _fft_flops(p) + 100 * h}


# ------------------------------------------------------------------ the same in 64 bits
def _rhs(g, u, band):
    """Nonlinear term (rotational form, 2/3 rule, projection, band forcing) and the band energy; u may have a box axis."""
    om = [g.c2r(w) * g.s for w in g.curl(u)]
    v = [g.c2r(u[i]) for i in range(3)]
    n = torch.stack([g.r2c((om[1] * v[2] - om[2] * v[1]) * g.s), g.r2c((om[2] * v[0] - om[0] * v[2]) * g.s),
                     g.r2c((om[0] * v[1] - om[1] * v[0]) * g.s)])
    umax = [x.abs().amax() * g.s for x in v]
    del om, v
    n = -g.project(n)
    eband = 0.0
    if band:
        inband = torch.sqrt(g.k2) <= KCUT
        eband = float(((u.abs() ** 2).sum(0) * (0.5 * g.w) * inband).sum()) * g.s ** 2
        n = n + (PIN / (2.0 * eband)) * (inband * u)
    return torch.where(g.mask, 0.0, n), eband, umax


def _vjp(g, u, go):
    """Transpose of the linearised nonlinear term (no band forcing), Euclidean on the parts of the half spectrum."""
    h = -g.project(torch.where(g.mask, 0.0, go))
    phi = [g.c2r(h[i] / g.w) for i in range(3)]
    v = [g.c2r(u[i]) * g.s for i in range(3)]
    om = [g.c2r(w) * g.s for w in g.curl(u)]

    def cross(a, b):
        return a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]
    psi = [g.s * g.w * g.r2c(x) for x in cross(v, phi)]
    gu = [g.s * g.w * g.r2c(x) for x in cross(phi, om)]
    return torch.stack([a + b for a, b in zip(g.curl(psi), gu)])


def _heun(g, u, nu, dt, band, n1=None):
    e = torch.exp(-nu * g.k2 * dt)
    if n1 is None:
        n1 = _rhs(g, u, band)[0]
    n2 = _rhs(g, e * (u + dt * n1), band)[0]
    return e * (u + 0.5 * dt * n1) + 0.5 * dt * n2


def _exact_step(c, u):
    g, band, nu = _case_grid(c), c["bandlim"], c["nu"]
    dx = [2 * math.pi / a / n for a, n in zip(g.alpha, g.n)]
    dt, t, recs, nold, h = DT, 0.0, [], None, 0.0
    for i in range(c["nsteps"]):
        n1, eband, umax = _rhs(g, u, band)
        umax = [float(x) for x in umax]
        cfl = sum(m * dt / d for m, d in zip(umax, dx))
        if c["cfl"] and (i == 0 or cfl > COURANT or (cfl < COURANT and dt < DT_MAX)):
            new = min((COURANT + COURANT) / (2.0 * cfl) * dt, DT_MAX)
            cfl, dt = cfl * new / dt, new
        if c["stepper"] == "heun" or i == 0:
            u = _heun(g, u, nu, dt, band, n1)
        else:
            c1, c2 = dt * (1.0 + dt / (2.0 * h)), -dt * dt / (2.0 * h)
            u = (torch.exp(-nu * g.k2 * dt) * (u + c1 * n1) + c2 * torch.exp(-nu * g.k2 * (dt + h)) * nold)
        nold, h, t = n1, dt, t + dt
        recs.append({"t": t, "dt": dt, "ekin": float(g.energy(u)), "courant": cfl, "eband": eband, "umax": umax,
                     "dissipation": nu * float(((u.abs() ** 2).sum(0) * g.w * g.k2).sum()) * g.s ** 2,
                     "injected_power": PIN if band else 0.0})
    return {"u": u, "records": _records(recs)} if c["records"] else {"u": u}


def _exact_diagnostics(g, u, nu):
    absk = torch.sqrt(g.k2)
    e2 = (u.abs() ** 2).sum(0)
    nspec = int(math.sqrt(sum(((n / 2.0) * (2.0 * a / 3.0)) ** 2 for n, a in zip(g.n, g.alpha)))) - 1
    base = torch.floor(absk)
    nk = torch.where(absk < base + 0.5, base, base + 1).to(torch.int64)
    es = torch.bincount(nk.reshape(-1), weights=e2.reshape(-1), minlength=nspec)[1:nspec] * g.s ** 2
    es = torch.cat([es, es.new_zeros(1)])            # the last shell is not filled
    e0, e1, eq = (float(e2[m].sum()) for m in (absk == 0, absk == 1.0, absk - math.sqrt(2.0) < 1e-9))
    umax = [float(g.c2r(u[i]).abs().amax()) * g.s for i in range(3)]
    dx = [2 * math.pi / a / n for a, n in zip(g.alpha, g.n)]
    div = g.c2r(1j * (g.kx * u[0] + g.ky * u[1] + g.kz * u[2])) * g.s
    return {"spectrum": (es.cpu().numpy(), e0, e1, eq), "kinetic": float(g.energy(u)),
            "dissipation": nu * float((e2 * g.w * g.k2).sum()) * g.s ** 2,
            "courant": (sum(m * DT / d for m, d in zip(umax, dx)), tuple(umax)), "divergence": float(div.amax())}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "ensemble":
        out = []
        for n, nus, u in _ensemble_inputs(c, seed):
            g, u = _Grid(n, n, n), u.to(torch.complex128)
            nu = torch.from_numpy(nus).to(u.device)[:, None, None, None]
            for _ in range(1 + c["nsteps"]):   # building an Ensemble advances its boxes by one step
                u = _heun(g, u, nu, DT, False)
            out.append(u)
        return out
    g, x = _case_grid(c), _inputs(c, seed)
    if kind == "fft":
        return g.c2r(x["spec"].to(torch.complex128)), g.r2c(x["phys"].to(torch.float64))
    u = x["u"].to(torch.complex128)
    if kind == "step":
        return _exact_step(c, u)
    if kind == "rhs":
        return _rhs(g, u, c["bandlim"])[0]
    if kind == "vjp":
        return _vjp(g, u, x["g"].to(torch.complex128))
    if kind == "residual_grad":
        lin, hm = -c["nu"] * g.k2, 1.0 / (1.0 + g.k2)
        r = lin * u + _rhs(g, u, False)[0]
        ge = g.s ** 2 * g.w * hm * r
        return 0.5 * g.s ** 2 * float((g.w * hm * r.abs() ** 2).sum()), _vjp(g, u, ge) + lin * ge
    if kind == "horizon_grad":
        go, dt, nu, states = x["g"].to(torch.complex128), DT, c["nu"], [u]
        for _ in range(c["nsteps"]):
            states.append(_heun(g, states[-1], nu, dt, False))
        e = torch.exp(-nu * g.k2 * dt)
        for v in reversed(states[:-1]):
            a = _vjp(g, e * (v + dt * _rhs(g, v, False)[0]), 0.5 * dt * go)
            go = e * (go + a) + _vjp(g, v, e * (0.5 * dt * go + dt * a))
        return go, states[-1]
    return _exact_diagnostics(g, u, c.get("nu", 5e-3))
