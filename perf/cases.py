"""The workloads this library's speed is measured on, through its public entry points.

A case is one stretch of a run as a driver makes it: the conserved state that the host holds goes
to the device (``Shark.upload_ptr`` from pinned memory), a number of steps run
(``Shark.run_steps``), and the state comes back for an output (``Shark.download_ptr``).  Charging
alone (``Shark.charge`` from a cold start) is a case of its own, as a run's first step and a
restart have it.  Sizes are those of the repository's configurations, tests and benchmark.

The mixed path holds its state in FP32 and the download widens it; those cases hand the fields
back in FP32, which loses nothing.  FP64 cases hand them back in FP64.
"""
import functools
import math

import numpy as np
import torch

from shark_gb300 import config as K
from shark_gb300 import setups
from shark_gb300.solver import Shark

DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # the 1D shock tube, the smallest problem users run: every step is launch latency
        dict(name="sod_1000_fp64", setup="sod", nx=1000, ny=1, ndust=0, fp64=True, slope=1, solver=2, steps=100),
        # the 1D dusty wave of the convergence tests: four species, implicit drag, FP64
        dict(name="dustywave_2048x4_fp64", setup="dustywave", nx=2048, ny=1, ndust=4, fp64=True, slope=2, solver=2,
             steps=100),
        # a small streaming-instability box, the size of parameter sweeps
        dict(name="si_128x8_mixed", setup="si", nx=128, ny=128, ndust=8, fp64=False, slope=3, solver=2, steps=100),
        # the benchmark's streaming-instability box
        dict(name="si_1024x8_mixed", setup="si", nx=1024, ny=1024, ndust=8, fp64=False, slope=3, solver=2, steps=100),
        # the same physics in FP64, the precision a reference run is made in
        dict(name="si_256x8_fp64", setup="si", nx=256, ny=256, ndust=8, fp64=True, slope=3, solver=2, steps=20),
        # adiabatic dusty shear layer on a ragged grid: HLLC with an energy equation, Epstein drag
        dict(name="kh_500x301x4_mixed", setup="kh", nx=500, ny=301, ndust=4, fp64=False, slope=1, solver=2, steps=50),
        # gas-only blast wave
        dict(name="sedov_1000_mixed", setup="sedov", nx=1000, ny=1000, ndust=0, fp64=False, slope=1, solver=2, steps=50),
        # Cartesian disk with softened gravity, viscosity and buffers
        dict(name="disk_cart_512x4_mixed", setup="disk_cart", nx=512, ny=512, ndust=4, fp64=False, slope=3, solver=2,
             steps=50),
        # polar disk at full size: FARGO, growth and charging every step
        dict(name="disk_polar_512x1024x16_mixed", setup="disk_polar", nx=512, ny=1024, ndust=16, fp64=False, slope=1,
             solver=2, steps=10, growth=True, charging=True),
        # the same in FP64 on a coarser grid
        dict(name="disk_polar_128x256x16_fp64", setup="disk_polar", nx=128, ny=256, ndust=16, fp64=True, slope=1,
             solver=2, steps=5, growth=True, charging=True),
        # driven dusty turbulence, the largest: 32 species, forcing, growth and charging every step
        dict(name="turb_768x32_mixed", setup="dusty_turb", nx=768, ny=768, ndust=32, fp64=False, slope=1, solver=2,
             steps=10, growth=True, charging=True),
        # charging alone from a cold start, as at the first step and after a restart
        dict(name="charge_384x32_fp64", setup="charge", nx=384, ny=384, ndust=32, fp64=True, slope=1, solver=2, steps=1,
             charging=True),
    ]


def draw(rng):
    def span(lo, hi):   # log-uniform whole number
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    setup = rng.choice(["sod", "dustywave", "si", "si", "kh", "sedov", "disk_cart", "disk_polar", "dusty_turb", "charge"])
    c = dict(setup=setup, ny=1, fp64=False, slope=rng.choice([1, 2, 3]), solver=rng.choice([0, 1, 2, 2]))
    if setup == "sod":
        c.update(nx=span(100, 4000), ndust=rng.choice([0, 0, 1, 3]), fp64=rng.random() < 0.7, steps=100)
    elif setup == "dustywave":
        c.update(nx=span(200, 8000), ndust=rng.randint(1, 10), fp64=rng.random() < 0.7, steps=100)
    elif setup == "si":
        c["fp64"] = rng.random() < 0.4
        n = span(48, 256 if c["fp64"] else 1024)
        c.update(nx=n, ny=n, ndust=rng.choice([1, 2, 3, 4, 6, 8, 8, 12]) if n < 800 else rng.choice([2, 4, 8]),
                 steps=20 if c["fp64"] else 50)
    elif setup == "kh":
        c["fp64"] = rng.random() < 0.3
        top = 256 if c["fp64"] else 1000
        c.update(nx=span(60, top), ny=span(60, top), ndust=rng.choice([0, 1, 3, 4, 5]), steps=20 if c["fp64"] else 50)
    elif setup == "sedov":
        c["fp64"] = rng.random() < 0.3
        n = span(64, 300 if c["fp64"] else 1000)
        c.update(nx=n, ny=n, ndust=0, steps=20 if c["fp64"] else 50)
    elif setup == "disk_cart":
        c["fp64"] = rng.random() < 0.3
        n = span(64, 160 if c["fp64"] else 512)
        c.update(nx=n, ny=n, ndust=rng.choice([1, 3, 4, 7]), steps=20 if c["fp64"] else 50)
    elif setup == "disk_polar":
        c["fp64"] = rng.random() < 0.3
        c.update(nx=span(48, 100 if c["fp64"] else 500), ny=span(64, 200 if c["fp64"] else 1000),
                 ndust=rng.choice([5, 8, 12, 16]), steps=5, growth=rng.random() < 0.7, charging=rng.random() < 0.7)
    elif setup == "dusty_turb":
        c["fp64"] = rng.random() < 0.2
        n = span(48, 96 if c["fp64"] else 512)
        c.update(nx=n, ny=n, ndust=rng.choice([8, 16, 20, 32]), steps=4, growth=rng.random() < 0.8,
                 charging=rng.random() < 0.7)
    else:
        n = span(48, 300)
        c.update(nx=n, ny=n, ndust=rng.choice([4, 10, 16, 32]), fp64=rng.random() < 0.5, steps=1, charging=True)
    return c


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _base(setup, nx, ny, ndust, fp64, slope, solver, growth, charging):
    """(config, unperturbed state on the device), from the repository's setup builders."""
    prec = K.PREC_FP64 if fp64 else K.PREC_MIXED
    if setup == "sod":
        cfg, u = setups.sod(nx=nx, ndust=ndust, slope_type=slope, solver=solver, precision=prec)
    elif setup == "dustywave":
        cfg, u = setups.dustywave(nx=nx, ndust=ndust, eps=np.full(ndust, 1.0 / ndust), slope_type=slope, precision=prec)
    elif setup == "si":
        cfg, u = setups.si(n=nx, ndust=ndust, noise=0.0, slope_type=slope, precision=prec)
    elif setup == "kh":
        # the namelist's values: the builder's defaults are dense enough to leave FP32's range
        cfg, u = setups.kh(n=nx, ny=ny, ndust=ndust, precision=prec, **dict(setups.KH_NML, slope_type=slope))
    elif setup == "sedov":
        cfg, u = setups.sedov(n=nx, slope_type=slope, precision=prec)
    elif setup == "disk_cart":
        cfg, u = setups.disk_cart(n=nx, ndust=ndust, slope_type=slope, precision=prec)
    elif setup == "disk_polar":
        cfg, u = setups.disk_polar_au(nr=nx, nphi=ny, ndust=ndust, growth=growth, charging=charging, noise=0.0,
                                      slope_type=slope, precision=prec)
    else:   # dusty_turb, charge
        cfg, u = setups.dusty_turb(n=nx, ndust=ndust, forcing=setup == "dusty_turb", charging=charging, growth=growth,
                                   slope_type=slope, precision=prec)
    cfg.solver = solver
    return cfg, torch.from_numpy(u).to(DEV)


def _inputs(case, seed):
    """(config, FP64 state on the device) of one seed: the setup's state with the structure a run
    has.  The boxes of the turbulence get smooth lognormal densities (gas, and every species its
    own on top), the SI box the noise on the dust velocities that its configuration states, the
    others white noise on the densities."""
    cfg, base = _base(case["setup"], case["nx"], case["ny"], case["ndust"], case["fp64"], case["slope"], case["solver"],
                      case.get("growth", False), case.get("charging", False))
    gen = torch.Generator(device=DEV).manual_seed(seed)
    N, g = cfg.ndust, cfg.nghost
    full = base.clone()
    u = full.view(cfg.nvar, cfg.ny_max, cfg.nx_max)[:, (g if cfg.ny > 1 else 0):(g + cfg.ny if cfg.ny > 1 else 1), g:g + cfg.nx]

    def uniform(*shape):
        return 2.0 * torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64) - 1.0

    ny, nx, setup = cfg.ny, cfg.nx, case["setup"]
    if setup == "si":
        for c in (1, 2, 3):
            u[5 + c * N:5 + (c + 1) * N] += u[5:5 + N] * (1e-3 * cfg.cs0) * uniform(N, ny, nx)
    elif setup == "sedov":
        u[0] *= 1.0 + 1e-2 * uniform(ny, nx)
    elif setup in ("dusty_turb", "charge"):
        x = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5) * (2.0 * math.pi / nx)
        y = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * (2.0 * math.pi / ny)
        modes = [(1, 0), (0, 1), (1, 1), (2, -1), (1, 2), (3, 1)]
        waves = torch.stack([torch.cos(kx * x[None, :] + ky * y[:, None] + math.pi * uniform(1))
                             for kx, ky in modes])
        own = uniform(1 + N, len(modes))
        f = torch.exp(0.35 * torch.einsum("m,myx->yx", own[0], waves))
        u[:5] *= f
        for k in range(N):
            fk = f * torch.exp(0.1 * torch.einsum("m,myx->yx", own[1 + k], waves))
            for c in range(4):
                u[5 + c * N + k] *= fk
    else:
        f = 1.0 + (1e-5 if setup == "dustywave" else 1e-3) * uniform(ny, nx)
        if setup == "sod":
            u[0] *= f
        else:
            u *= f
    return cfg, full


def prepare(case, seed):
    """A run's handle, its initial state in pinned host memory and the buffers the fields come back in."""
    cfg, full = _inputs(case, seed)
    u0 = torch.empty(full.shape, dtype=torch.float64, pin_memory=DEV == "cuda")
    u0.copy_(full)
    shark = Shark(cfg)
    state = dict(case=case, cfg=cfg, shark=shark, u0=u0)
    if case["setup"] == "charge":
        shark.upload_ptr(u0.data_ptr())
    else:
        state["host"] = torch.empty_like(u0, pin_memory=DEV == "cuda")
        if not case["fp64"]:
            state["out"] = torch.empty(u0.shape, dtype=torch.float32)
    return state


def run(state):
    g = state["shark"]
    if state["case"]["setup"] == "charge":
        g.charge_reset()
        g.charge()
        ch = g.download_charge()
        out = dict(psi=ch["psi"], zd=ch["zd"], ni=ch["ni"], ne=ch["ne"], eta=ch["eta"], gamma_d=ch["gamma_d"])
        if not state["case"]["fp64"]:
            out = {k: v if k == "psi" else v.astype(np.float32) for k, v in out.items()}
        return out
    host = state["host"]
    g.upload_ptr(state["u0"].data_ptr())
    g.run_steps(state["case"]["steps"])
    g.download_ptr(host.data_ptr())
    if not state["case"]["fp64"]:
        host = state["out"].copy_(host)
    return _fields(state["cfg"], host)


def _fields(cfg, u):
    """The state's fields by their kind (each kind has units and a size of its own)."""
    u = u.view(cfg.nvar, cfg.ncells)
    N = cfg.ndust
    out = dict(rho=u[0], momentum=u[1:4], energy=u[4])
    if N > 0:
        out.update(rho_dust=u[5:5 + N], momentum_dust=u[5 + N:])
    return out


def work(case):
    """Each step reads and writes the state once; the copies to and from the host move it in FP64.
    Operations: about 250 for a species' fluxes, limiters and update in a cell; growth N(N+1)/2
    pairs at 20 for one sub-step, charging some 40 for a species in an iteration."""
    cfg_n, cells = case["ndust"], case["nx"] * case["ny"]
    nvar, elem, steps = 5 + 4 * cfg_n, 8 if case["fp64"] else 4, case["steps"]
    if case["setup"] == "charge":
        return {"bytes": cells * (elem * (1 + cfg_n) + elem * (5 + 2 * cfg_n) + 8 * (6 + 2 * cfg_n)),
                "flops": cells * 20 * 40 * cfg_n}
    flops = cells * steps * 250.0 * (1 + cfg_n)
    if case.get("growth"):
        flops += cells * steps * 20.0 * cfg_n * (cfg_n + 1) / 2
    if case.get("charging"):
        flops += cells * steps * 3 * 40.0 * cfg_n
    return {"bytes": float(cells * nvar * (2 * 8 + steps * 2 * elem)), "flops": flops}


# ---------------------------------------------------------------------------------------------
# the same steps in plain FP64 torch (Cartesian grids without growth and charging)
# ---------------------------------------------------------------------------------------------
def exact(case, seed):
    if case["setup"] in ("disk_cart", "disk_polar", "dusty_turb", "charge"):
        return None
    cfg, full = _inputs(case, seed)
    u = full.view(cfg.nvar, cfg.ny_max, cfg.nx_max)
    step = _Step(cfg)
    step.ghosts(u)
    for _ in range(case["steps"]):
        u = step(u)
    return {k: v.clone() for k, v in _fields(cfg, u.reshape(-1)).items()}


class _Step:
    """One step of the Godunov scheme: predictor and limited slopes, HLLC / HLL / LLF gas and
    upwind dust fluxes, force kick, drag heating, implicit drag, on a uniform grid.  Fields are
    (variable, y, x) with two ghost cells on every side that has neighbours."""

    def __init__(self, cfg):
        self.c, self.N, self.two_d = cfg, cfg.ndust, cfg.ny > 1
        self.iso = cfg.iso_cs == 1
        self.dx = cfg.box_l / cfg.nx
        self.dy = cfg.box_l_y / cfg.ny if self.two_d else math.inf
        self.ya = slice(2, 2 + cfg.ny) if self.two_d else slice(0, 1)   # active rows
        self.yp = slice(1, 3 + cfg.ny) if self.two_d else slice(0, 1)   # rows that are predicted
        self.xa, self.xp = slice(2, 2 + cfg.nx), slice(1, 3 + cfg.nx)
        self.x = (torch.arange(cfg.nx, device=DEV, dtype=torch.float64) + 0.5) * self.dx
        self.kick = bool(cfg.flags & K.FLAG_FORCE_KICK)
        self.per_species = lambda a: torch.tensor(list(a)[:self.N], device=DEV, dtype=torch.float64).view(-1, 1, 1)

    def ghosts(self, u):
        c, nx, ny, N = self.c, self.c.nx, self.c.ny, self.N
        if c.setup == K.SETUP_SOD:
            for cells, rho, p in ((slice(0, 2), c.sod_rho_l, c.sod_P_l), (slice(2 + nx, 4 + nx), c.sod_rho_r, c.sod_P_r)):
                u[0, :, cells], u[1:4, :, cells], u[4, :, cells] = rho, 0.0, p / (c.gamma - 1.0)
            return
        if self.two_d:
            u[:, :2, self.xa], u[:, 2 + ny:, self.xa] = u[:, ny:ny + 2, self.xa].clone(), u[:, 2:4, self.xa].clone()
        u[:, :, :2], u[:, :, 2 + nx:] = u[:, :, nx:nx + 2].clone(), u[:, :, 2:4].clone()
        if c.setup == K.SETUP_SI:
            shift = c.si_q_shear * c.si_omega * c.box_l
            for iz, ir in [(3, 0)] + [(5 + 3 * N + k, 5 + k) for k in range(N)]:
                u[iz, :, :2] -= u[ir, :, :2] * shift
                u[iz, :, 2 + nx:] += u[ir, :, 2 + nx:] * shift

    def limit(self, a, b):
        t = self.c.slope_type
        if t == 1:
            r = torch.where(b.abs() < a.abs(), b, a)
            return torch.where(a * b < 0.0, 0.0, r)
        if t == 2:
            return torch.where(a * b <= 0.0, 0.0, 2.0 * a * b / (a + b))
        cen = 0.5 * (a + b)
        lim = torch.where(a * b <= 0.0, 0.0, 1.5 * torch.minimum(a.abs(), b.abs()))
        return torch.copysign(torch.minimum(lim, cen.abs()), cen)

    def slopes(self, q):
        x, y = slice(1, -1), slice(1, -1) if self.two_d else slice(0, 1)
        mid = q[..., y, x]
        sx = self.limit((mid - q[..., y, :-2]) / self.dx, (q[..., y, 2:] - mid) / self.dx)
        if not self.two_d:
            return sx, torch.zeros_like(sx)
        return sx, self.limit((mid - q[..., :-2, x]) / self.dy, (q[..., 2:, x] - mid) / self.dy)

    def gas_flux(self, l, r):
        """l, r: (rho, normal, transverse and z velocity, P) of the two sides of the faces."""
        gm1 = self.c.gamma - 1.0
        cs = [self.cs0 if self.iso else torch.sqrt(self.c.gamma * s[4] / s[0]) for s in (l, r)]
        E = [s[4] / gm1 + 0.5 * s[0] * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2) for s in (l, r)]
        U = [torch.stack((s[0], s[0] * s[1], s[0] * s[2], s[0] * s[3], e)) for s, e in zip((l, r), E)]
        F = [torch.stack((s[0] * s[1], s[0] * s[1] ** 2 + s[4], s[0] * s[1] * s[2], s[0] * s[1] * s[3], (e + s[4]) * s[1]))
             for s, e in zip((l, r), E)]
        ul, ur = l[1], r[1]
        if self.c.solver == 0:
            lam = torch.maximum(ul.abs() + cs[0], ur.abs() + cs[1])
            return 0.5 * (F[0] + F[1]) - 0.5 * lam * (U[1] - U[0])
        top = max(cs) if self.iso else torch.maximum(*cs)
        sl = torch.clamp(torch.minimum(ul, ur) - top, max=0.0)
        sr = torch.clamp(torch.maximum(ul, ur) + top, min=0.0)
        if self.c.solver == 1:
            return (sr * F[0] - sl * F[1] + sr * sl * (U[1] - U[0])) / (sr - sl)
        hl, hr = l[0] * (ul - sl), r[0] * (sr - ur)
        us = (hr * ur + hl * ul + (l[4] - r[4])) / (hr + hl)
        ps = (hr * l[4] + hl * r[4] + hl * hr * (ul - ur)) / (hr + hl)
        left = us > 0.0
        s, S, e = torch.where(left, l, r), torch.where(left, sl, sr), torch.where(left, E[0], E[1])
        rs = s[0] * (S - s[1]) / (S - us)
        es = ((S - s[1]) * e - s[4] * s[1] + ps * us) / (S - us)
        outer = torch.where(left, sl > 0.0, sr <= 0.0)   # a supersonic face takes its own side's state
        ro, uo = torch.where(outer, s[0], rs), torch.where(outer, s[1], us)
        po, eo = torch.where(outer, s[4], ps), torch.where(outer, e, es)
        return torch.stack((ro * uo, ro * uo * uo + po, ro * uo * s[2], ro * uo * s[3], (eo + po) * uo))

    @staticmethod
    def dust_flux(l, r):
        """Huang & Bai: each side's flux where its velocity points through the face."""
        def one(s):
            return torch.stack((s[0] * s[1], s[0] * s[1] ** 2, s[0] * s[1] * s[2], s[0] * s[1] * s[3]))
        ul, ur = l[1], r[1]
        from_l = (ul > 0.0) & (ur != 0.0)
        from_r = (ur < 0.0) & (ul != 0.0)
        return one(l) * from_l + one(r) * from_r

    def __call__(self, u):
        c, N, gamma = self.c, self.N, self.c.gamma
        A = (Ellipsis, self.ya, self.xa)
        gas, dust = u[:5], u[5:].view(4, N, u.shape[1], u.shape[2])
        rho = gas[0]
        q = torch.empty_like(gas)
        q[0], q[1:4] = rho, gas[1:4] / rho
        q[4] = torch.clamp((gamma - 1.0) * (gas[4] - 0.5 * rho * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)), min=c.smallp)
        cs = c.cs0 if self.iso else torch.sqrt(gamma * q[4] / q[0])
        self.cs0 = cs
        if self.iso:
            q[4] = rho * cs ** 2
        qd = torch.cat((dust[:1], dust[1:] / dust[:1])) if N else dust
        # explicit forces of the shearing box, on the active cells
        f, fd = torch.zeros_like(q[1:4]), torch.zeros_like(qd[1:4])
        if self.kick:
            q_om, om = c.si_q_shear, c.si_omega
            tide = 2.0 * q_om * om ** 2 * (self.x - 0.5 * c.box_l)
            f[0][A] = tide - 2.0 * om * q[3][A] - 2.0 * c.si_rad0 * om * c.si_eta_stream
            f[2][A] = 2.0 * om * q[1][A]
            fd[0][A] = tide - 2.0 * om * qd[3][A]
            fd[2][A] = 2.0 * om * qd[1][A]
        ts = self.stopping_times(q, qd, cs, A)
        dt = self.courant(q, qd, cs, f, fd, A)
        new = u.clone()
        ng, nd = new[:5], new[5:].view_as(dust)
        if self.kick:
            ra = rho[A]
            old = 0.5 * (ng[1:4][A] ** 2).sum(0) / ra
            ng[1:4][A] += ra * dt * f[A]
            ng[4][A] += 0.5 * (ng[1:4][A] ** 2).sum(0) / ra - old
            nd[1:4][A] += dust[0][A] * dt * fd[A]
        self.update(ng, self.faces(q, f, dt, cs, True), dt, A)
        if N:
            self.update(nd, self.faces(qd, fd, dt, cs, False), dt, A)
        drag, back = bool(c.flags & K.FLAG_DRAG), bool(c.flags & K.FLAG_BACK_REACTION)
        if N and back and not self.iso:   # drag heating
            v = q[1:4].unsqueeze(1)
            ng[4][A] += (dt * (v * (v - qd[1:4]))[A].sum(0) / ts).sum(0)
        if N and drag:
            a = dt / ts
            w = a / (1.0 + a)
            p = ng[1:4][A] + (w * nd[1:4][A]).sum(1)
            rn = ng[0][A] + (w * nd[0][A]).sum(0)
            nd[1:4][A] = nd[1:4][A] / (1.0 + a) + w * (p / rn).unsqueeze(1) * nd[0][A]
            if back:
                ng[1:4][A] = p / rn * ng[0][A]
            nd[0][A] = torch.maximum(ng[0][A] * c.dust_ratio_min, nd[0][A])
        self.ghosts(new)
        return new

    def stopping_times(self, q, qd, cs, A):
        c = self.c
        if not self.N:
            return None
        if c.setup == K.SETUP_SI:
            return self.per_species(c.dust_tstop).expand(qd[0][A].shape)
        if c.setup == K.SETUP_DUSTYWAVE:
            return qd[0][A] / self.per_species(c.dust_K)
        return math.sqrt(math.pi * c.gamma / 8.0) * c.rhograin * self.per_species(c.dust_size) / (q[0][A] * cs[A])

    def courant(self, q, qd, cs, f, fd, A):
        c = self.c
        d = min(self.dx, self.dy)
        vv = q[1:4][A].abs().sum(0)
        vmax = (cs if self.iso else cs[A]) + vv
        force = torch.sqrt((f[A] ** 2).sum(0))
        if self.N:
            vd = qd[1:4][A].abs().sum(0)
            vmax = torch.maximum(vmax, vd.amax(0))
            force = torch.maximum(force, torch.sqrt((fd[A] ** 2).sum(0)).amax(0))
            vv = vd[-1]
        dt = c.cfl * d / vmax.max()
        if self.kick:
            ratio = torch.clamp(force * d / vv ** 2, min=1e-3)
            lim = c.cfl * d / vv * (torch.sqrt(1.0 + 2.0 * c.cfl * ratio) - 1.0) / ratio
            dt = torch.minimum(dt, torch.where(vv != 0.0, lim, math.inf).min())
        return dt

    def faces(self, q, f, dt, cs, gas):
        """Fluxes through the x and y faces of the active cells, as (x faces, y faces or None)."""
        c, h = self.c, 0.5 * dt
        sx, sy = self.slopes(q)
        P = (Ellipsis, self.yp, self.xp)
        q0, v = q[P], q[1:4][P] + h * f[P] if self.kick else q[1:4][P]
        rho, uu, vv, ww = q0[0], v[0], v[1], v[2]
        div = sx[1] + sy[2]
        half = [rho + h * (-uu * sx[0] - vv * sy[0] - div * rho)]
        press_x = press_y = 0.0
        if gas:
            p, px, py = q0[4], sx[4], sy[4]
            if self.iso:
                px, py = sx[0] * cs ** 2, sy[0] * cs ** 2
            press_x, press_y = px / rho, py / rho
        half.append(uu + h * (-uu * sx[1] - vv * sy[1] - press_x))
        half.append(vv + h * (-uu * sx[2] - vv * sy[2] - press_y))
        half.append(ww + h * (-uu * sx[3] - vv * sy[3]))
        if gas:
            half.append(p + h * (-uu * px - vv * py - div * c.gamma * p))
            sx, sy = torch.cat((sx[:4], px[None])), torch.cat((sy[:4], py[None]))
        half = torch.stack(half)

        def sides(s, d):
            m, p_ = half + 0.5 * s * d, half - 0.5 * s * d
            if gas:
                for w in (m, p_):
                    w[4] = cs ** 2 * w[0] if self.iso else torch.clamp(w[4], min=c.smallp)
            return m, p_

        flux = self.gas_flux if gas else self.dust_flux
        m, p_ = sides(sx, self.dx)
        ya = slice(1, -1) if self.two_d else slice(0, 1)
        fx = flux(m[..., ya, :-1], p_[..., ya, 1:])
        if not self.two_d:
            return fx, None
        m, p_ = sides(sy, self.dy)
        swap = [0, 2, 1, 3] + ([4] if gas else [])
        fy = flux(m[swap][..., :-1, 1:-1], p_[swap][..., 1:, 1:-1])
        return fx, fy[swap]

    def update(self, u, faces, dt, A):
        fx, fy = faces
        # the x faces' area is dx and the y faces' dy, which is exact for square cells only
        vol = self.dx * self.dy if self.two_d else self.dx
        new = u[A] + (fx[..., :-1] - fx[..., 1:]) * (self.dx if self.two_d else 1.0) / vol * dt
        if self.two_d:
            new = new + (fy[..., :-1, :] - fy[..., 1:, :]) * self.dy / vol * dt
        u[A] = new

