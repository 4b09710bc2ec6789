"""The workloads this framework's speed is measured on.

A case is a plain dict: what is run ("kind"), the grid and the options.  The
kinds are the framework's public entry points as a user's program calls them:

  step       one composed moist RK3 large step (gm1b_moist_large_step through
             NativeMoistLargeStep): what a simulation spends its time in
  dry        one dry RK3 step of the doubly periodic trajectory
  acoustic   one split-explicit acoustic RK stage
  scalar     the fifth-order / WENO5 tendency of one scalar
  momentum   the fifth-order momentum advection with its mass fluxes
  tke        one advection / RK stage of the subgrid TKE
  gradient   one forward step of the differentiable warm-rain transport and
             its reverse

"column" is "uniform" (the terrain operator family on flat metrics) or
"stretched" (the flat family on a stretch_z = 1 column, 20 m at the ground to
500 m aloft).  The inputs are a Weisman-Klemp column and hodograph with warm,
cloudy, raining bubbles, smooth wind perturbations and grid-scale noise, all
made on the GPU from the seed.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gm1_b200.adjoint import FrozenFlow, StageCheckpointedAdjoint, WarmRainTransport
from gm1_b200.advection import (StretchedColumn, launch_cuda_gm1_child_stretched_scalar_advection5,
                                launch_cuda_scalar_advection5)
from gm1_b200.initial_state import DryBubbleCase, dry_periodic_state
from gm1_b200.momentum import (StretchedMomentumColumn, launch_cuda_gm1_child_stretched_momentum5,
                               launch_cuda_terrain_open_momentum_advection5)
from gm1_b200.moist_step import (MOIST_STATE_DTYPES, MoistStepConfig, NativeMoistLargeStep, StretchedColumnSpec,
                                 moist_state_shapes, weisman_klemp_initial_state)
from gm1_b200.periodic import launch_cuda_psolver3_trajectory, sound3_stage_schedule_f32
from gm1_b200.terrain_open import (ALL_ARRAY_NAMES, COLUMN_DIAGNOSTIC_NAMES, TERRAIN_STATIC_REQUIRED,
                                   compile_cuda_psolver3_terrain_open, launch_cuda_gm1_child_psolver3_open_stage,
                                   launch_cuda_psolver3_terrain_open_stage, terrain_open_sound_shapes,
                                   terrain_static_shapes)
from gm1_b200.tke_evolution import launch_cuda_flat_tke_rk_stage, launch_cuda_tke_rk_stage

NG = 3
OPEN = (2, 2, 2, 2)
THETA_WEPS = float(np.float32(10.0) * np.float32(1.0e-18))
Q_WEPS = float(np.float32(1.0e-2) * np.float32(1.0e-18))


def _case(name, kind, ni, nj, nk, column="uniform", **more):
    return dict(name=name, kind=kind, ni=ni, nj=nj, nk=nk, column=column, **more)


def listed():
    return [
        # the headline run: a 39 M cell supercell at 100 m on the stretched column
        _case("step-640x768x80-stretched", "step", 640, 768, 80, "stretched", nsound=8, closure=False),
        # the ordinary run: the 1 km supercell benchmark on the uniform column
        _case("step-256x256x80-uniform", "step", 256, 256, 80, nsound=10, closure=False),
        # a ragged domain with the closure's held tendencies (SGS stress and
        # scalar diffusion, Rayleigh damping, dissipative heating) switched on
        _case("step-189x131x64-held", "step", 189, 131, 64, "stretched", nsound=6, closure=True),
        # the smallest member of an ensemble: launches and latency
        _case("step-53x48x40-member", "step", 53, 48, 40, nsound=10, closure=False),
        # the dry warm-bubble benchmark, one large step per call
        _case("dry-64x64x40", "dry", 64, 64, 40, nsound=6),
        # the acoustic stage on both columns, for a host model that calls the
        # operators one by one
        _case("acoustic-256x256x80-uniform", "acoustic", 256, 256, 80, nrk=3, nsound=10),
        _case("acoustic-333x271x72-stretched", "acoustic", 333, 271, 72, "stretched", nrk=3, nsound=8),
        # final-stage WENO5 of one scalar, and a small fifth-order one
        _case("scalar-weno-320x384x80-stretched", "scalar", 320, 384, 80, "stretched", nrk=3),
        _case("scalar-fifth-67x61x45-uniform", "scalar", 67, 61, 45, nrk=1),
        _case("momentum-320x384x80-stretched", "momentum", 320, 384, 80, "stretched"),
        _case("tke-256x250x80-stretched", "tke", 256, 250, 80, "stretched", nrk=2),
        # one step of a gradient: forward keeping the stages, then the reverse
        _case("gradient-96x96x48", "gradient", 96, 96, 48),
    ]


KINDS = ("step", "step", "dry", "acoustic", "acoustic", "scalar", "scalar", "momentum", "momentum", "tke", "gradient")
# the largest plane a drawn case of each kind takes (cells)
MOST_CELLS = {"step": 12_000_000, "dry": 1_500_000, "acoustic": 20_000_000, "scalar": 30_000_000,
              "momentum": 20_000_000, "tke": 25_000_000, "gradient": 1_500_000}


def draw(rng):
    kind = rng.choice(KINDS)
    nk = rng.randint(24, 96)
    if kind in ("dry", "gradient"):
        nk = rng.randint(24, 64)
    most = min(700.0, math.sqrt(MOST_CELLS[kind] / nk))

    def size():
        return int(round(math.exp(rng.uniform(math.log(24.0), math.log(most)))))

    c = dict(kind=kind, ni=size(), nj=size(), nk=nk, column=rng.choice(("uniform", "stretched")))
    if kind in ("dry", "gradient"):
        c["column"] = "uniform"
    if kind in ("step", "dry", "acoustic"):
        c["nsound"] = rng.choice((6, 8, 10))
    if kind in ("acoustic", "scalar", "tke"):
        c["nrk"] = rng.randint(1, 3)
    if kind == "step":
        c["closure"] = rng.random() < 0.4
    return c


# --------------------------------------------------------------- the inputs


def _config(c):
    nk = c["nk"]
    closure = dict(sgs_diffusion=True, rayleigh=True, dissipative_heating=True) if c.get("closure") else {}
    if c["column"] == "uniform":
        return MoistStepConfig(c["ni"], c["nj"], nk, 1000.0, 1000.0, 20000.0 / nk, 5.0, c.get("nsound", 10), **closure)
    n1 = n3 = nk // 8
    bot = 20.0 * n1
    top = bot + 260.0 * (nk - n1 - n3)
    spec = StretchedColumnSpec(top + 500.0 * n3, bot, top, 20.0, 500.0)
    return MoistStepConfig(c["ni"], c["nj"], nk, 100.0, 100.0, 100.0, 0.6, c.get("nsound", 8), column=spec, **closure)


@functools.lru_cache(maxsize=8)
def _column(cfg):
    """State and metrics of the undisturbed column (an 8 x 8 plane of it)."""
    import dataclasses

    small = dataclasses.replace(cfg, ni=8, nj=8)
    return weisman_klemp_initial_state(small, bubble_k=0.0, noise_k=0.0)


def _spread(a, shape, dtype=None):
    """The column array `a` over the whole plane of `shape`, on the GPU."""
    t = torch.from_numpy(np.ascontiguousarray(a))
    if t.ndim >= 3:
        t = t[..., 4, 4][..., None, None].expand(*shape)
    elif t.ndim == 2:
        t = t[4:5, 4:5].expand(*shape)
    elif tuple(t.shape) != tuple(shape):
        t = t[:1].expand(*shape)
    if t.ndim >= 3:
        return t[..., :1, :1].contiguous().cuda().expand(*shape).contiguous()
    return t.contiguous().cuda()


def _metrics(cfg, names=None):
    _, m = _column(cfg)
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    shapes = dict(terrain_static_shapes(ni=ni, nj=nj, nk=nk), rho0_padded=(nk + 2, nj + 6, ni + 6))
    return {n: _spread(a, shapes.get(n, a.shape)) for n, a in m.items() if names is None or n in names}


class _Air:
    """The disturbed fields: theta', the moisture, the winds and TKE, smooth
    structure from a few bubbles and waves plus grid-scale noise."""

    def __init__(self, cfg, seed):
        self.cfg = cfg
        self.col, _ = _column(cfg)
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))
        ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
        zh = _column(cfg)[1]["zh"][:, 4, 4]
        k = torch.from_numpy(zh.copy()).cuda().view(nk, 1, 1)
        j = ((torch.arange(nj, device="cuda") + 0.5) / nj).view(1, nj, 1)
        i = ((torch.arange(ni, device="cuda") + 0.5) / ni).view(1, 1, ni)
        host = np.random.default_rng(int(seed))
        bubble = torch.zeros((nk, nj, ni), device="cuda")
        for _ in range(4):
            x, y, z = host.uniform(0.25, 0.75, 2).tolist() + [host.uniform(1200.0, 6000.0)]
            r = torch.sqrt(((i - x) / 0.2) ** 2 + ((j - y) / 0.2) ** 2 + ((k - z) / 1500.0) ** 2)
            bubble += torch.where(r < 1.0, torch.cos(0.5 * math.pi * r) ** 2, torch.zeros_like(r))
        self.bubble = bubble
        px, py = host.uniform(0.0, 2.0 * math.pi, 2).tolist()
        ramp = 1.0 - torch.exp(-k / 2000.0)
        # zero within a few cells of the lateral edges: the open sides see
        # the undisturbed flow
        wi = torch.clamp((torch.minimum(i, 1.0 - i) * ni - 4.0) / 4.0, 0.0, 1.0)
        wj = torch.clamp((torch.minimum(j, 1.0 - j) * nj - 4.0) / 4.0, 0.0, 1.0)
        self.wave_u = 3.0 * torch.sin(6.0 * math.pi * i + px) * torch.cos(4.0 * math.pi * j + py) * ramp * wi * wj
        self.wave_v = 3.0 * torch.cos(4.0 * math.pi * i + py) * torch.sin(6.0 * math.pi * j + px) * ramp * wi * wj
        self.window = wi * wj

    def noise(self, amp, shape=None):
        c = self.cfg
        n = torch.rand((c.nk, c.nj, c.ni) if shape is None else shape, device="cuda", generator=self.g)
        return (2.0 * amp) * n.sub_(0.5)

    def theta(self):
        return (2.0 * self.bubble + self.noise(0.1)).float()

    def moisture(self):
        qv0 = torch.from_numpy(self.col["qv0"].copy()).cuda().view(-1, 1, 1)
        core = torch.clamp(self.bubble - 0.3, min=0.0)
        qv = qv0 * (1.0 + 0.3 * self.bubble) + torch.zeros_like(self.bubble)
        return qv, 2.0e-3 * core, 1.0e-3 * core * (1.0 + self.noise(0.2))

    def winds(self, u, v, w):
        """The column's wind plus the disturbance into the padded u, v, w."""
        c = self.cfg
        ni, nj, nk = c.ni, c.nj, c.nk
        u += _spread(self.col["u3d"], u.shape)
        v += _spread(self.col["v3d"], v.shape)
        u[1:nk + 1, NG:NG + nj, NG:NG + ni] += self.wave_u + self.noise(0.3) * self.window
        v[1:nk + 1, NG:NG + nj, NG:NG + ni] += self.wave_v + self.noise(0.3) * self.window
        up = (4.0 * self.bubble + self.noise(0.1)) * self.window
        w[2:nk + 1, NG:NG + nj, NG:NG + ni] += 0.5 * (up[:-1] + up[1:])

    def tke(self):
        c = self.cfg
        t = torch.zeros((c.nk + 1, c.nj, c.ni), device="cuda")
        t[1:c.nk] = 1.0e-4 + torch.clamp(self.bubble + 0.05 * self.noise(1.0), min=0.0)[1:]
        return t


def _storm(cfg, seed):
    """The composed step's device state and metrics."""
    s0, _ = _column(cfg)
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    s = {}
    for n, shape in moist_state_shapes(ni, nj, nk).items():
        dt = MOIST_STATE_DTYPES.get(n, np.float32)
        a = s0[n]
        s[n] = _spread(a, shape) if a.any() and n not in ("u3d", "v3d", "ua", "va") else \
            torch.zeros(shape, dtype=torch.from_numpy(np.zeros(1, dt)).dtype, device="cuda")
    m = _metrics(cfg)
    air = _Air(cfg, seed)
    s["th3d"].copy_(air.theta())
    for r, q in enumerate(air.moisture()):
        s["q3d"][r].copy_(q)
    air.winds(s["u3d"], s["v3d"], s["w3d"])
    s["tke3d"].copy_(air.tke())
    # the start's density from its pi, theta and qv
    pi, theta = s["pi0_3d"], s["th0_3d"] + s["th3d"]
    s["prs"].copy_(100000.0 * pi ** (1005.7 / 287.04))
    s["rho"].copy_(s["prs"] / (theta * pi * (287.04 + 461.5 * s["q3d"][0])))
    s["rr"].copy_(1.0 / s["rho"])
    rho, rf = s["rho"], s["rf"]
    rf[1:nk] = m["c1"][1:nk] * rho[:-1] + m["c2"][1:nk] * rho[1:]
    rf[0] = 1.875 * rho[0] - 1.25 * rho[1] + 0.375 * rho[2]
    rf[nk] = 1.875 * rho[nk - 1] - 1.25 * rho[nk - 2] + 0.375 * rho[nk - 3]
    for cur, base in (("ua", "u3d"), ("va", "v3d"), ("wa", "w3d"), ("tha", "th3d"), ("qa", "q3d"), ("tkea", "tke3d")):
        s[cur].copy_(s[base])
    return s, m


def _flow(cfg, air, m):
    """Mass fluxes rru, rrv, rrw of the disturbed winds and their divergence."""
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    u = torch.zeros((nk + 2, nj + 6, ni + 7), device="cuda")
    v = torch.zeros((nk + 2, nj + 7, ni + 6), device="cuda")
    w = torch.zeros((nk + 3, nj + 6, ni + 6), device="cuda")
    air.winds(u, v, w)
    rho = torch.zeros(nk + 2, device="cuda")
    rho[1:nk + 1] = m["rho0_3d"][:, 0, 0]
    rf = torch.zeros(nk + 3, device="cuda")
    rf[1:nk + 2] = m["rf0"][:, 0, 0]
    rru, rrv, rrw = u * rho.view(-1, 1, 1), v * rho.view(-1, 1, 1), w * rf.view(-1, 1, 1)
    _, rdsf = _levels(cfg, m)
    js, is_ = slice(NG, NG + nj), slice(NG, NG + ni)
    div = (rru[1:nk + 1, js, NG + 1:NG + ni + 1] - rru[1:nk + 1, js, is_]) / cfg.dx
    div += (rrv[1:nk + 1, NG + 1:NG + nj + 1, is_] - rrv[1:nk + 1, js, is_]) / cfg.dy
    div += (rrw[2:nk + 2, js, is_] - rrw[1:nk + 1, js, is_]) * rdsf.view(-1, 1, 1)
    return rru, rrv, rrw, div


def _rdz(cfg):
    return float(np.float32(np.float32(1.0) / np.float32(cfg.dz)))


def _levels(cfg, m):
    """1/dz between mass levels (at the nk+1 w levels) and at the nk mass levels."""
    if cfg.column is None:
        one = torch.full((cfg.nk + 1,), 1.0 / cfg.dz, device="cuda")
        return one, one[:cfg.nk].clone()
    return _rdz(cfg) * m["mf"][:, 0, 0], _rdz(cfg) * m["mh"][:, 0, 0]


def _acoustic_arrays(cfg, seed, m):
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    shapes = terrain_open_sound_shapes(ni, nj, nk)
    shapes.update({n: (1,) for n in COLUMN_DIAGNOSTIC_NAMES})
    a = {n: torch.zeros(shapes[n], device="cuda") for n in ALL_ARRAY_NAMES}
    air = _Air(cfg, seed)
    air.winds(a["ua"], a["va"], a["wa"])
    for n in ("u", "v", "w"):
        a[n + "3d"].copy_(a[n + "a"])
        a[n + "ten"].copy_(air.noise(1.0e-3, a[n + "ten"].shape))
    for n in ("uh", "vh", "ruf", "rvf"):
        a[n].fill_(1.0)

    def padded(x):
        p = torch.nn.functional.pad(x[None, None], (1, 1, 1, 1, 1, 1), mode="replicate")
        return p[0, 0]

    pi0, th0 = (_spread(_column(cfg)[0][n], (nk, nj, ni)) for n in ("pi0_3d", "th0_3d"))
    pp = 1.0e-5 * air.bubble + air.noise(2.0e-6)
    qv = air.moisture()[0]
    a["ppi"].copy_(padded(pp))
    a["pp3d"].copy_(a["ppi"])
    a["ppx"].copy_(padded(air.noise(1.0e-7)))
    a["piadv"].copy_(padded(pi0 + pp))
    a["ppterm"].copy_(padded(0.4 * (pi0 + pp)))
    a["thv"].copy_(padded((th0 + air.theta()) * (1.0 + 0.61 * qv)))
    a["ppten"].copy_(padded(air.noise(1.0e-8)))
    a["scalar"].copy_(air.noise(1.0, a["scalar"].shape))
    for n, side, shape in (("radbcw", -1, (nk + 2, nj + 6)), ("radbce", 1, (nk + 2, nj + 6)),
                           ("radbcs", -1, (nk + 2, ni + 6)), ("radbcn", 1, (nk + 2, ni + 6))):
        a[n].copy_(side * (15.0 + air.noise(10.0, shape)))
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dry":
        b = DryBubbleCase(ni=case["ni"], nj=case["nj"], nk=case["nk"], dz=20000.0 / case["nk"], seed=int(seed) % (1 << 31),
                          u0=5.0, v0=-3.0, wind_perturbation=2.0)
        arrays = {n: torch.from_numpy(a).cuda() for n, a in dry_periodic_state(b).items()}
        return dict(kind=kind, case=b, a=arrays, nsound=case["nsound"])
    cfg = _config(case)
    grid = dict(ni=cfg.ni, nj=cfg.nj, nk=cfg.nk)
    if kind == "step":
        s, m = _storm(cfg, seed)
        return dict(kind=kind, s=s, step=NativeMoistLargeStep(cfg, s, m))
    if kind == "acoustic":
        m = _metrics(cfg, TERRAIN_STATIC_REQUIRED + ("rho0_padded", "mh_profile", "mf_profile"))
        return dict(kind=kind, cfg=cfg, grid=grid, m=m, nrk=case["nrk"], a=_acoustic_arrays(cfg, seed, m),
                    compiled=compile_cuda_psolver3_terrain_open(retain_column_diagnostics=False))
    m = _metrics(cfg)
    air = _Air(cfg, seed)
    if kind == "momentum":
        a = {}
        for n, shape in (("u", (cfg.nk + 2, cfg.nj + 6, cfg.ni + 7)), ("v", (cfg.nk + 2, cfg.nj + 7, cfg.ni + 6)),
                         ("w", (cfg.nk + 3, cfg.nj + 6, cfg.ni + 6))):
            for f in (n + "3d", n + "ten", "rr" + n):
                a[f] = torch.zeros(shape, device="cuda")
        air.winds(a["u3d"], a["v3d"], a["w3d"])
        a["uh"] = torch.ones(cfg.ni + 6, device="cuda")
        a["vh"] = torch.ones(cfg.nj + 6, device="cuda")
        return dict(kind=kind, cfg=cfg, grid=grid, m=m, a=a,
                    divx=torch.zeros((cfg.nk, cfg.nj, cfg.ni), device="cuda"))
    rru, rrv, rrw, divx = _flow(cfg, air, m)
    if kind == "scalar":
        th0 = _spread(_column(cfg)[0]["th0_3d"], (cfg.nk, cfg.nj, cfg.ni))
        scalar = torch.zeros((cfg.nk + 2, cfg.nj + 6, cfg.ni + 6), device="cuda")
        scalar[1:cfg.nk + 1] = torch.nn.functional.pad((th0 - 300.0 + air.theta())[None], (3, 3, 3, 3),
                                                       mode="replicate")[0]
        return dict(kind=kind, cfg=cfg, grid=grid, m=m, scalar=scalar, flux=dict(rru=rru, rrv=rrv, rrw=rrw),
                    divx=divx, out=torch.zeros((cfg.nk, cfg.nj, cfg.ni), device="cuda"), nrk=case["nrk"])
    if kind == "tke":
        t = air.tke()
        a = dict(tkea=t, tke3d=t.clone(), tketen=torch.zeros_like(t), rru=rru, rrv=rrv, rrw=rrw, divx=divx,
                 **{n: m[n] for n in ("c1", "c2", "rrf0", "mh", "mf", "gz", "rgz", "rgzu", "rgzv")})
        a["tketen"][1:cfg.nk] = 1.0e-4 * air.noise(1.0)[1:]
        for n in ("kmh", "kmv"):
            a[n] = torch.ones_like(t)
        a["rho"], a["rf"] = m["rho0_3d"], m["rf0"].clone()
        return dict(kind=kind, cfg=cfg, grid=grid, m=m, a=a, ws=torch.empty_like(t), nrk=case["nrk"])
    assert kind == "gradient", kind
    col = _column(cfg)[0]
    shape = (cfg.nk, cfg.nj, cfg.ni)
    fields = dict(rru=rru, rrv=rrv, rrw=rrw, divx=divx, c1=m["c1"], c2=m["c2"], rr0=m["rr0"], gz=m["gz"],
                  th0=_spread(col["th0_3d"], shape), pi0=_spread(col["pi0_3d"], shape),
                  prs=_spread(col["prs"], shape), pp3d=1.0e-5 * air.bubble)
    flow = FrozenFlow(cfg.ni, cfg.nj, cfg.nk, cfg.dx, cfg.dy, cfg.dz, THETA_WEPS, fields)
    model = WarmRainTransport(flow, cfg.dt, weps={"th3d": THETA_WEPS, "qv": Q_WEPS, "qc": Q_WEPS, "qr": Q_WEPS})
    qv, qc, qr = air.moisture()
    # a thin haze everywhere keeps the water off the limiters' kinks at zero,
    # where the derivative is a matter of convention
    qc, qr = qc + 1.0e-4 * (1.0 + air.noise(0.2)), qr + 1.0e-5 * (1.0 + air.noise(0.2))
    state = (air.theta(), qv.contiguous(), qc, qr)
    lam = tuple(air.noise(1.0) for _ in range(4))
    return dict(kind=kind, cfg=cfg, fields=fields, state=state, lam=lam, adj=StageCheckpointedAdjoint(model, streams=2))


STEP_OUTPUTS = ("u3d", "v3d", "w3d", "th3d", "pp3d", "q3d", "tke3d", "rho", "prs", "rain", "ppx")
ACOUSTIC_OUTPUTS = ("u3d", "v3d", "w3d", "pp3d", "ppd", "rru", "rrv", "rrw", "radbcw", "radbce", "radbcs", "radbcn")


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["step"].step()
        return {n: state["s"][n] for n in STEP_OUTPUTS}
    if kind == "dry":
        b, a = state["case"], state["a"]
        launch_cuda_psolver3_trajectory(a, ni=b.ni, nj=b.nj, nk=b.nk, steps=1, dt=6.0, nsound=state["nsound"], dx=b.dx,
                                        dy=b.dy, dz=b.dz, scratch_outputs=False, check_status=False)
        return {n: a[n] for n in ("u3d", "v3d", "w3d", "th3d", "pp3d")}
    if kind == "gradient":
        out, stages = state["adj"].forward(state["state"])
        return {"state": out, "gradient": state["adj"].reverse(stages, state["lam"])}
    cfg, m, grid = state["cfg"], state["m"], state["grid"]
    flat = cfg.column is not None
    if kind == "acoustic":
        kw = dict(grid, nrk=state["nrk"], dt=cfg.dt, nsound=cfg.nsound, dx=cfg.dx, dy=cfg.dy,
                  compiled=state["compiled"])
        if flat:
            col = StretchedMomentumColumn(True, m["rho0_padded"], mh=m["mh_profile"], mf=m["mf_profile"],
                                          rdz=_rdz(cfg))
            launch_cuda_gm1_child_psolver3_open_stage(state["a"], m, vertical=col, **kw)
        else:
            launch_cuda_psolver3_terrain_open_stage(state["a"], m, dz=cfg.dz, **kw)
        return {n: state["a"][n] for n in ACOUSTIC_OUTPUTS}
    if kind == "scalar":
        kw = dict(grid, nrk=state["nrk"], dx=cfg.dx, dy=cfg.dy, weps=THETA_WEPS, lateral_sides=OPEN, write_fluxes=False)
        met = {n: m[n] for n in ("c1", "c2", "rr0", "gz")}
        if flat:
            col = StretchedColumn(True, mh=m["mh_profile"], rdz=_rdz(cfg))
            launch_cuda_gm1_child_stretched_scalar_advection5(state["scalar"], state["flux"], met, state["divx"],
                                                              state["out"], None, col, **kw)
        else:
            launch_cuda_scalar_advection5(state["scalar"], state["flux"], met, state["divx"], state["out"], None,
                                          dz=cfg.dz, **kw)
        return {"tendency": state["out"]}
    if kind == "momentum":
        a = state["a"]
        if flat:
            col = StretchedMomentumColumn(True, m["rho0_padded"], mh=m["mh_profile"], mf=m["mf_profile"], rr0=m["rr0"],
                                          rdz=_rdz(cfg))
            launch_cuda_gm1_child_stretched_momentum5(a, m, col, nrk=1, dx=cfg.dx, dy=cfg.dy, divx=state["divx"],
                                                      lateral_sides=OPEN, **grid)
        else:
            launch_cuda_terrain_open_momentum_advection5(a, m, nrk=1, dx=cfg.dx, dy=cfg.dy, dz=cfg.dz,
                                                         divx=state["divx"], lateral_sides=OPEN, **grid)
        return {n: a[n] for n in ("uten", "vten", "wten", "rru", "rrv", "rrw")} | {"divx": state["divx"]}
    assert kind == "tke", kind
    a = state["a"]
    kw = dict(grid, workspace=state["ws"], nrk=state["nrk"], dx=cfg.dx, dy=cfg.dy, dt=cfg.dt)
    if flat:
        launch_cuda_flat_tke_rk_stage(a, mf_profile=m["mf_profile"], rdz=_rdz(cfg), **kw)
    else:
        launch_cuda_tke_rk_stage(a, dz=cfg.dz, **kw)
    return {"tke3d": a["tke3d"]}


# ------------------------------------------------------- work and tolerance


def work(case):
    """Compulsory words per cell: every field once per pass between two grid-
    wide dependencies (an RK stage's tendencies, an acoustic small step, the
    closure, the microphysics), which no larger-than-cache domain avoids.
    The flops are counted from the formulas, to the nearest ten."""
    cells = case["ni"] * case["nj"] * case["nk"]
    kind = case["kind"]
    loops = lambda dt, stages: sum(sound3_stage_schedule_f32(dt, case["nsound"], r)[0] for r in stages)  # noqa: E731
    dt = 6.0 if kind == "dry" else 5.0 if case["column"] == "uniform" else 0.6
    if kind == "step":
        n = loops(dt, (1, 2, 3))
        words, flops = 149 + 20 * n, 3600 + 90 * n
        if case["closure"]:
            words, flops = words + 40, flops + 500
    elif kind == "dry":
        n = loops(dt, (1, 2, 3))
        words, flops = 3 * 14 + 20 * n + 2, 900 + 90 * n
    elif kind == "acoustic":
        n = loops(dt, (case["nrk"],))
        words, flops = 24 + 20 * n, 20 + 90 * n
    elif kind == "scalar":
        words, flops = 6, 250 if case["nrk"] == 3 else 60
    elif kind == "momentum":
        words, flops = 13, 200
    elif kind == "tke":
        words, flops = 8, 270 if case["nrk"] == 3 else 80
    else:
        words, flops = 2 * (8 + 12) + 3 * 4 * 2 * 6, 5000
    return {"bytes": 4.0 * words * cells, "flops": float(flops) * cells}


def tolerance(case):
    """About four times what a correct implementation in binary32 differs by:
    the operators measured against `exact`, the whole steps between two runs
    whose starting words differ in their last bit.  The radiation histories
    (a ratio of two small differences of winds, averaged) set the acoustic
    stage's bound; a limiter's branch taken the other way in a cell sets the
    gradient's."""
    return {"step": {"rel": 1e-4, "max": 5e-3}, "dry": {"rel": 2e-5, "max": 1e-4},
            "acoustic": {"rel": 2e-2, "max": 0.5}, "scalar": {"rel": 4e-4, "max": 1e-2},
            "momentum": {"rel": 5e-5, "max": 5e-3}, "tke": {"rel": 2e-7, "max": 1e-4},
            "gradient": {"rel": 2e-2, "max": 0.9}}[case["kind"]]


# ------------------------------------------------- the same in 64 bits (torch)

F5 = (2.0 / 60.0, -13.0 / 60.0, 47.0 / 60.0, 27.0 / 60.0, -3.0 / 60.0)
F3 = (-1.0 / 6.0, 5.0 / 6.0, 2.0 / 6.0)


def _flx5(s):
    return F5[0] * s[0] + F5[1] * s[1] + F5[2] * s[2] + F5[3] * s[3] + F5[4] * s[4]


def _flx3(s):
    return F3[0] * s[0] + F3[1] * s[1] + F3[2] * s[2]


def _weno5(s, eps):
    s1, s2, s3, s4, s5 = s
    b1 = 13.0 / 12.0 * (s1 - 2 * s2 + s3) ** 2 + 0.25 * (s1 - 4 * s2 + 3 * s3) ** 2
    b2 = 13.0 / 12.0 * (s2 - 2 * s3 + s4) ** 2 + 0.25 * (s2 - s4) ** 2
    b3 = 13.0 / 12.0 * (s3 - 2 * s4 + s5) ** 2 + 0.25 * (3 * s3 - 4 * s4 + s5) ** 2
    tau = (b1 - b3).abs()
    cap = torch.full_like(tau, 1.0e30)
    w1, w2, w3 = (g * (1.0 + torch.minimum(tau / (b + eps), cap) ** 2)
                  for g, b in ((0.1, b1), (0.6, b2), (0.3, b3)))
    p1 = s1 / 3.0 - 7.0 / 6.0 * s2 + 11.0 / 6.0 * s3
    p2 = -s2 / 6.0 + 5.0 / 6.0 * s3 + s4 / 3.0
    p3 = s3 / 3.0 + 5.0 / 6.0 * s4 - s5 / 6.0
    return (w1 * p1 + w2 * p2 + w3 * p3) / (w1 + w2 + w3)


def _upstrpd(s, eps):
    dd = s[1] - s[0]
    rr = (s[2] - s[1]) / (dd + torch.where(dd >= 0, torch.full_like(dd, eps), torch.full_like(dd, -eps)))
    phi = torch.clamp(torch.minimum(rr, torch.clamp(1.0 / 6.0 + rr / 3.0, max=1.0)), min=0.0)
    return s[1] + phi * dd


def _up5(m, s, weno, eps):
    """m times the upwind reconstruction from the six points around a face."""
    r = (lambda v: _weno5(v, eps)) if weno else _flx5
    return m * torch.where(m >= 0, r(s[:5]), r(s[:0:-1]))


def _near_ends(face, first, last, m, S, lin, weno, eps):
    """The vertical face flux: five-point inside, three-point or linear near
    the two ends of the column (S(k) is the value k points above the first
    point below the face: S(0), S(1) are its two neighbours)."""
    three = (lambda a, b, c: _upstrpd((a, b, c), eps)) if weno else (lambda a, b, c: _flx3((a, b, c)))
    five = (lambda v: _weno5(v, eps)) if weno else _flx5
    up = (lambda: five([S(q) for q in (-2, -1, 0, 1, 2)]))
    dn = (lambda: five([S(q) for q in (3, 2, 1, 0, -1)]))
    if face == first:
        return m * torch.where(m >= 0, lin, three(S(2), S(1), S(0)))
    if face == last:
        return m * torch.where((m > 0) if weno else (m >= 0), three(S(-1), S(0), S(1)), lin)
    if face == first + 1:
        return m * torch.where(m >= 0, three(S(-1), S(0), S(1)), dn())
    return m * torch.where(m >= 0, up(), dn()) if face != last - 1 else None


def _scalar_exact(s, f, rdsf, nrk, cfg, eps):
    """The tendency of the padded scalar s in 64 bits, open sides."""
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    rru, rrv, rrw, c1, c2 = f["rru"], f["rrv"], f["rrw"], f["c1"], f["c2"]
    weno = nrk == 3
    K, J, I = slice(1, nk + 1), slice(NG, NG + nj), slice(NG, NG + ni)
    fx = _up5(rru[K, J, NG:NG + ni + 1], [s[K, J, q:q + ni + 1] for q in range(6)], weno, eps)
    fy = _up5(rrv[K, NG:NG + nj + 1, I], [s[K, q:q + nj + 1, I] for q in range(6)], weno, eps)
    col = s[:, J, I]
    fz = [torch.zeros_like(col[0])]
    for k in range(2, nk + 1):
        m = rrw[k, J, I]
        S = lambda q, k=k: col[k - 1 + q]  # noqa: E731
        lin = c1[k - 1] * S(0) + c2[k - 1] * S(1)
        if k == nk - 1:
            dn = _upstrpd((S(2), S(1), S(0)), eps) if weno else _flx3((S(2), S(1), S(0)))
            up = [S(q) for q in (-2, -1, 0, 1, 2)]
            fz.append(m * torch.where(m >= 0, _weno5(up, eps) if weno else _flx5(up), dn))
        else:
            fz.append(_near_ends(k, 2, nk, m, S, lin, weno, eps))
    fz.append(torch.zeros_like(col[0]))
    fz = torch.stack(fz)
    sv = col[K]

    def direction(lo, hi, mlo, mhi, first, last, rd):
        a, b = first & (mlo >= 0), last & (mhi <= 0)
        lo2 = torch.where(a, hi, lo)
        hi2 = torch.where(b, lo2, hi)
        t = (lo2 - hi2) * rd
        return torch.where(a | b, t - sv * (mhi - mlo) * rd, t)

    ii = torch.arange(ni, device=s.device).view(1, 1, ni)
    jj = torch.arange(nj, device=s.device).view(1, nj, 1)
    ax = direction(fx[..., :-1], fx[..., 1:], rru[K, J, NG:NG + ni], rru[K, J, NG + 1:NG + ni + 1], ii == 0,
                   ii == ni - 1, 1.0 / cfg.dx)
    ay = direction(fy[:, :-1], fy[:, 1:], rrv[K, NG:NG + nj, I], rrv[K, NG + 1:NG + nj + 1, I], jj == 0, jj == nj - 1,
                   1.0 / cfg.dy)
    az = (fz[:-1] - fz[1:]) * rdsf.view(-1, 1, 1)
    return (ax + ay + az + sv * f["divx"]) * f["rr0"]


def _momentum_exact(cfg, m, a, rds, rdsf):
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    u, v, w = (a[n].double() for n in ("u3d", "v3d", "w3d"))
    rho, rf, rr0, rrf0, c1, c2 = (m[n][:, 0, 0].double() for n in ("rho0_3d", "rf0", "rr0", "rrf0", "c1", "c2"))
    K, J, I = slice(1, nk + 1), slice(NG, NG + nj), slice(NG, NG + ni)
    rru, rrv, rrw = (a[n].double().clone() for n in ("rru", "rrv", "rrw"))
    r3 = rho.view(-1, 1, 1)
    rru[K, J, NG:NG + ni + 1] = r3 * u[K, J, NG:NG + ni + 1]
    rrv[K, NG:NG + nj + 1, I] = r3 * v[K, NG:NG + nj + 1, I]
    rrw[2:nk + 1, J, I] = rf[1:nk].view(-1, 1, 1) * w[2:nk + 1, J, I]
    rrw[1, J, I] = 0.0
    rrw[nk + 1, J, I] = 0.0
    rdx, rdy = 1.0 / cfg.dx, 1.0 / cfg.dy
    div = (rru[K, J, NG + 1:NG + ni + 1] - rru[K, J, I]) * rdx + (rrv[K, NG + 1:NG + nj + 1, I] - rrv[K, J, I]) * rdy
    div = div + (rrw[2:nk + 2, J, I] - rrw[1:nk + 1, J, I]) * rdsf.view(-1, 1, 1)

    def along(q, ra, rb, na, nb, da, db, dv, rw):
        """The increment of the wind q on its own axis (last): faces 1..na-1,
        rows 0..nb-1; ra, rb the mass fluxes along and across, dv the
        divergence and rw the vertical mass flux with the same axes."""
        A, B = slice(NG, NG + na), slice(NG, NG + nb)
        fa = _up5(0.5 * (ra[K, B, NG:NG + na] + ra[K, B, NG + 1:NG + na + 1]),
                  [q[K, B, 1 + p:1 + p + na] for p in range(6)], False, 0.0)
        adva = -(fa[..., 1:] - fa[..., :-1]) * da
        mt = rb[K, NG:NG + nb + 1, NG + 1:NG + na] + rb[K, NG:NG + nb + 1, NG:NG + na - 1]
        fb = _up5(0.5 * mt, [q[K, p:p + nb + 1, NG + 1:NG + na] for p in range(6)], False, 0.0)
        f0 = torch.where(mt[:, :1] >= 0, fb[:, 1:2], fb[:, :1])
        fn = torch.where(mt[:, -1:] <= 0, fb[:, -2:-1], fb[:, -1:])
        fb = torch.cat((f0, fb[:, 1:-1], fn), 1)
        advb = -(fb[:, 1:] - fb[:, :-1]) * db
        qc = q[K, B, NG + 1:NG + na]
        d = rb[K, NG + 1:NG + nb + 1] - rb[K, NG:NG + nb]
        corr = 0.5 * qc * (d[..., NG:NG + na - 1] + d[..., NG + 1:NG + na]) * db
        advb[:, :1] -= torch.where(mt[:, :1] >= 0, corr[:, :1], torch.zeros_like(corr[:, :1]))
        advb[:, -1:] -= torch.where(mt[:, -1:] <= 0, corr[:, -1:], torch.zeros_like(corr[:, -1:]))
        fz = [torch.zeros_like(qc[0])]
        for kf in range(2, nk + 1):
            mm = 0.5 * (rw[kf, B, NG + 1:NG + na] + rw[kf, B, NG:NG + na - 1])
            S = lambda p, kf=kf: q[kf - 1 + p, B, NG + 1:NG + na]  # noqa: E731
            lin = c1[kf - 1] * S(0) + c2[kf - 1] * S(1)
            if kf == nk - 1:
                fz.append(mm * torch.where(mm >= 0, _flx5([S(p) for p in (-2, -1, 0, 1, 2)]), _flx3((S(2), S(1), S(0)))))
            else:
                fz.append(_near_ends(kf, 2, nk, mm, S, lin, False, 0.0))
        fz.append(torch.zeros_like(qc[0]))
        fz = torch.stack(fz)
        advz = -(fz[1:] - fz[:-1]) * rdsf.view(-1, 1, 1)
        return (adva + advb + advz + qc * 0.5 * (dv[..., 1:] + dv[..., :-1])) * rr0.view(-1, 1, 1)

    T = lambda t: t.transpose(1, 2)  # noqa: E731
    uten, vten, wten = (a[n].double().clone() for n in ("uten", "vten", "wten"))
    uten[K, J, NG + 1:NG + ni] += along(u, rru, rrv, ni, nj, rdx, rdy, div, rrw)
    vten[K, NG + 1:NG + nj, I] += T(along(T(v), T(rrv), T(rru), nj, ni, rdy, rdx, T(div), T(rrw)))
    F = slice(2, nk + 1)
    k2, k1 = c2[1:nk].view(-1, 1, 1), c1[1:nk].view(-1, 1, 1)

    def across(q, ra, n, rd):
        """w advected along the last axis (n cells)."""
        B = slice(NG, q.shape[1] - NG)
        mm = k2 * ra[2:nk + 1, B, NG:NG + n + 1] + k1 * ra[1:nk, B, NG:NG + n + 1]
        fa = _up5(mm, [q[F, B, p:p + n + 1] for p in range(6)], False, 0.0)
        first = torch.where(mm[..., :1] >= 0, fa[..., 1:2], fa[..., :1])
        last = torch.where(mm[..., -1:] <= 0, fa[..., -2:-1], fa[..., -1:])
        fa = torch.cat((first, fa[..., 1:-1], last), 2)
        adv = -(fa[..., 1:] - fa[..., :-1]) * rd
        corr = q[F, B, NG:NG + n] * (mm[..., 1:] - mm[..., :-1]) * rd
        adv[..., :1] -= torch.where(mm[..., :1] >= 0, corr[..., :1], torch.zeros_like(corr[..., :1]))
        adv[..., -1:] -= torch.where(mm[..., -1:] <= 0, corr[..., -1:], torch.zeros_like(corr[..., -1:]))
        return adv

    ra, rb = rru[:, :nj + 6], rrv[:, :, :ni + 6]
    advx, advy = across(w, ra, ni, rdx), T(across(T(w), T(rb), nj, rdy))
    fz = []
    for k in range(1, nk + 1):
        mm = 0.5 * (rrw[k, J, I] + rrw[k + 1, J, I])
        S = lambda p, k=k: w[k + p, J, I]  # noqa: E731
        if k == nk - 1:
            fz.append(mm * torch.where(mm >= 0, _flx5([S(p) for p in (-2, -1, 0, 1, 2)]), _flx3((S(2), S(1), S(0)))))
        else:
            fz.append(_near_ends(k, 1, nk, mm, S, 0.5 * (S(0) + S(1)), False, 0.0))
    fz = torch.stack(fz)
    advz = -(fz[1:] - fz[:-1]) * rds[1:nk].view(-1, 1, 1)
    total = advx + advy + advz + w[F, J, I] * (k2 * div[1:] + k1 * div[:-1])
    wten[F, J, I] += total * rrf0[1:nk].view(-1, 1, 1)
    return {"uten": uten, "vten": vten, "wten": wten, "rru": rru, "rrv": rrv, "rrw": rrw, "divx": div}


def _tke_exact(cfg, m, a, nrk, rds):
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    eps = float(np.float32(100.0) * np.float32(1.0e-18))
    weno = nrk == 3
    q = a["tke3d"].double()
    rru, rrv, rrw, div = (a[n].double() for n in ("rru", "rrv", "rrw", "divx"))
    c2, c1, rrf0 = (m[n][:, 0, 0].double()[1:nk].view(-1, 1, 1) for n in ("c2", "c1", "rrf0"))
    c1 = 1.0 - c2
    T = lambda t: t.transpose(1, 2)  # noqa: E731
    qi = q[1:nk]

    def across(qq, r, n, rd):
        p = torch.nn.functional.pad(qq[None], (3, 3, 0, 0), mode="replicate")[0]
        r = r[:, NG:NG + qq.shape[1], NG:NG + n + 1]
        mm = c2 * r[2:nk + 1] + c1 * r[1:nk]
        f = _up5(mm, [p[..., s:s + n + 1] for s in range(6)], weno, eps)
        first = torch.where(mm[..., :1] >= 0, f[..., 1:2], f[..., :1])
        last = torch.where(mm[..., -1:] <= 0, f[..., -2:-1], f[..., -1:])
        f = torch.cat((first, f[..., 1:-1], last), 2)
        adv = -(f[..., 1:] - f[..., :-1]) * rd
        corr = qq * (mm[..., 1:] - mm[..., :-1]) * rd
        adv[..., :1] -= torch.where(mm[..., :1] >= 0, corr[..., :1], torch.zeros_like(corr[..., :1]))
        adv[..., -1:] -= torch.where(mm[..., -1:] <= 0, corr[..., -1:], torch.zeros_like(corr[..., -1:]))
        return adv

    ax = across(qi, rru, ni, 1.0 / cfg.dx)
    ay = T(across(T(qi).contiguous(), T(rrv), nj, 1.0 / cfg.dy))
    J, I = slice(NG, NG + nj), slice(NG, NG + ni)
    fz = []
    for k in range(1, nk + 1):
        mm = 0.5 * (rrw[k, J, I] + rrw[k + 1, J, I])
        S = lambda p, k=k: q[k - 1 + p]  # noqa: E731
        if k == nk - 1:
            up = [S(p) for p in (-2, -1, 0, 1, 2)]
            dn = _upstrpd((S(2), S(1), S(0)), eps) if weno else _flx3((S(2), S(1), S(0)))
            fz.append(mm * torch.where((mm > 0) if weno else (mm >= 0), _weno5(up, eps) if weno else _flx5(up), dn))
        else:
            fz.append(_near_ends(k, 1, nk, mm, S, 0.5 * (S(0) + S(1)), weno, eps))
    fz = torch.stack(fz)
    az = -(fz[1:] - fz[:-1]) * rds[1:nk].view(-1, 1, 1)
    total = ax + ay + az + qi * (c2 * div[1:] + c1 * div[:-1])
    out = torch.zeros_like(q)
    value = a["tkea"].double()[1:nk] + cfg.dt / (4 - nrk) * (a["tketen"].double()[1:nk] + total * rrf0)
    out[1:nk] = torch.where(value < 1e-10, torch.zeros_like(value), value)
    return {"tke3d": out}


def _acoustic_exact(cfg, m, a, nrk, rds, rdsf):
    ni, nj, nk = cfg.ni, cfg.nj, cfg.nk
    nloop, dts = sound3_stage_schedule_f32(cfg.dt, cfg.nsound, nrk)
    alph, kdiv, cp = float(np.float32(0.6)), float(np.float32(0.1)), 1005.7
    beta, rdx, rdy = 1.0 - alph, 1.0 / cfg.dx, 1.0 / cfg.dy
    a = {n: a[n].double().clone() for n in a if a[n].numel() > 1}
    prof = {n: m[n][:, 0, 0].double().view(-1, 1, 1) for n in ("rr0", "rf0", "c1", "c2")}
    K, B = slice(1, nk + 1), (slice(1, nk + 1), slice(2, nj + 4), slice(2, ni + 4))
    a["ppd"][K] = a["ppx"][K]
    for n in ("rru", "rrv"):
        a[n][B] = 0.0
    a["rrw"][B] = a["wa"][B] * beta
    if nrk != 1:
        a["pp3d"][K] = a["ppi"][K]
        for n in ("u", "v", "w"):
            a[n + "3d"][B] = a[n + "a"][B]
    u, v, w, pp, ppd, th = (a[n] for n in ("u3d", "v3d", "w3d", "pp3d", "ppd", "thv"))
    C = (K, slice(1, nj + 1), slice(1, ni + 1))
    up = lambda t: t[2:nk + 2, 1:nj + 1, 1:ni + 1]  # noqa: E731
    lo = lambda t: t[0:nk, 1:nj + 1, 1:ni + 1]  # noqa: E731
    t0 = dts * rdsf.view(-1, 1, 1)
    r2, r1 = t0 * prof["rr0"] * prof["rf0"][1:], t0 * prof["rr0"] * prof["rf0"][:-1]
    pi = a["piadv"]
    qk = t0 * a["ppterm"][C]
    pk2 = r2 * (-prof["c2"][1:] * up(pi) + (1.0 - prof["c1"][1:]) * pi[C])
    pk1 = r1 * (prof["c1"][:-1] * lo(pi) + (prof["c2"][:-1] - 1.0) * pi[C])
    pk2[-1], pk1[0] = 0.0, 0.0
    mm = dts * cp * rds[:nk].view(-1, 1, 1) * (prof["c2"][:-1] * th[C] + prof["c1"][:-1] * lo(th))
    a1, a2 = pk1 + qk, pk2 - qk
    J, I = slice(NG, NG + nj), slice(NG, NG + ni)
    tx, ty = 0.5 * dts * rdx, 0.5 * dts * rdy
    n0, n1 = slice(NG, NG + nj + 1), slice(NG, NG + ni + 1)
    for n in range(1, nloop + 1):
        for f, x, xi, rad, sgn in ((u, NG, NG + 1, "radbcw", 1), (u, ni + NG, ni + NG - 1, "radbce", -1)):
            d = sgn * (f[K, J, xi] - f[K, J, x])
            f[K, J, x] += dts * (-a[rad][K, J] * d * rdx + a["uten"][K, J, x])
        for f, y, yi, rad, sgn in ((v, NG, NG + 1, "radbcs", 1), (v, nj + NG, nj + NG - 1, "radbcn", -1)):
            d = sgn * (f[K, yi, I] - f[K, y, I])
            f[K, y, I] += dts * (-a[rad][K, I] * d * rdy + a["vten"][K, y, I])
        P, Q = ppd[C], th[C]
        g = 0.5 * cp * rdx * (P[..., 1:] - P[..., :-1]) * (Q[..., 1:] + Q[..., :-1])
        u[K, J, NG + 1:NG + ni] += dts * (a["uten"][K, J, NG + 1:NG + ni] - g)
        g = 0.5 * cp * rdy * (P[:, 1:] - P[:, :-1]) * (Q[:, 1:] + Q[:, :-1])
        v[K, NG + 1:NG + nj, I] += dts * (a["vten"][K, NG + 1:NG + nj, I] - g)
        xw, xe, ys, yn = u[K, J, I], u[K, J, NG + 1:NG + ni + 1], v[K, J, I], v[K, NG + 1:NG + nj + 1, I]
        div = (xe - xw) * rdx + (yn - ys) * rdy
        c0 = pi[C]
        jj, ii = slice(1, nj + 1), slice(1, ni + 1)
        adv = -tx * (xw * (c0 - pi[K, jj, 0:ni]) + xe * (pi[K, jj, 2:ni + 2] - c0)) \
            - ty * (ys * (c0 - pi[K, 0:nj, ii]) + yn * (pi[K, 2:nj + 2, ii] - c0))
        wk, wk1 = w[1:nk + 1, J, I], w[2:nk + 2, J, I]
        fpk = dts * (a["ppten"][C] - a["ppterm"][C] * div) + adv + beta * (wk * a1 + wk1 * a2)
        old = pp[C].clone()
        fw = dts * a["wten"][2:nk + 1, J, I] - beta * mm[1:] * (old[1:] - old[:-1])
        dd = wk[1:] + fw - alph * mm[1:] * ((old + fpk)[1:] - (old + fpk)[:-1])
        aa, cc = -alph * alph * mm[1:] * a1[:-1], alph * alph * mm[1:] * a2[1:]
        bb = 1.0 - alph * alph * mm[1:] * (a2[:-1] - a1[1:])
        ec, ed = [], []
        for k in range(nk - 1):
            piv = bb[k] + aa[k] * ec[-1] if k else bb[k]
            ec.append(-cc[k] / piv)
            ed.append((dd[k] - aa[k] * ed[-1]) / piv if k else dd[k] / piv)
        x = ed[-1]
        w[nk, J, I] = x
        for k in range(nk - 3, -1, -1):
            x = ec[k] * x + ed[k]
            w[k + 2, J, I] = x
        new = old + fpk + alph * (w[1:nk + 1, J, I] * a1 + w[2:nk + 2, J, I] * a2)
        tend = kdiv * (new - old)
        pp[C] = new
        ppd[C] = new + tend
        last = n == nloop
        if last and nrk == 3:
            a["ppx"][C] = tend
        if not last:
            ppd[K] = torch.nn.functional.pad(ppd[C][None], (1, 1, 1, 1), mode="replicate")[0]
        for s, f, wt in (("rru", u, 1.0), ("rrv", v, 1.0), ("rrw", w, alph if last else 1.0)):
            a[s][K, n0, n1] = (a[s][K, n0, n1] + wt * f[K, n0, n1]) * (1.0 / nloop if last else 1.0)
    # the radiation histories: each boundary line's mean phase speed
    dttmp = cfg.dt / (4 - nrk)
    for n, q, q0, f2, f1, lo_, hi_, dim in (
            ("radbcw", "ua", u, 5, 4, -350.0, 0.0, 2), ("radbce", "ua", u, ni + 2, ni + 1, 0.0, 350.0, 2),
            ("radbcs", "va", v, 5, 4, -350.0, 0.0, 1), ("radbcn", "va", v, nj + 2, nj + 1, 0.0, 350.0, 1)):
        A, at = a[q][K], f1 if lo_ < 0.0 else f2
        foo = (A.select(dim, f2) - A.select(dim, f1))
        num = (cfg.dx if dim == 2 else cfg.dy) * (A.select(dim, at) - q0[K].select(dim, at))
        den = dttmp * (foo + torch.copysign(torch.full_like(foo, 1.0e-10), foo))
        line = J if dim == 2 else I
        a[n][K, line] = torch.clamp(num / den, lo_, hi_).mean(0)[line]
    Y = slice(2, nj + 4)
    u[K, Y, :3], u[K, Y, ni + 4:] = u[K, Y, 3:4], u[K, Y, ni + 3:ni + 4]
    v[K, :3, 2:ni + 4], v[K, nj + 4:, 2:ni + 4] = v[K, 3:4, 2:ni + 4], v[K, nj + 3:nj + 4, 2:ni + 4]
    F = slice(2, nk + 1)
    w[F, Y, :3], w[F, Y, ni + 3:] = w[F, Y, 3:4], w[F, Y, ni + 2:ni + 3]
    w[1, Y, 2:ni + 4] = 0.0
    w[nk + 1, Y, 2:ni + 4] = 0.0
    u[K, :3, 2:ni + 5], u[K, nj + 3:, 2:ni + 5] = u[K, 3:4, 2:ni + 5], u[K, nj + 2:nj + 3, 2:ni + 5]
    Y = slice(2, nj + 5)
    v[K, Y, :3], v[K, Y, ni + 3:] = v[K, Y, 3:4], v[K, Y, ni + 2:ni + 3]
    w[F, :3, 2:ni + 4], w[F, nj + 3:, 2:ni + 4] = w[F, 3:4, 2:ni + 4], w[F, nj + 2:nj + 3, 2:ni + 4]
    if nrk < 3:
        pp[K, :, 0], pp[K, :, ni + 1] = pp[K, :, 1], pp[K, :, ni]
        pp[K, 0], pp[K, nj + 1] = pp[K, 1], pp[K, nj]
    return {n: a[n] for n in ACOUSTIC_OUTPUTS}


def _f32(x):
    return float(np.float32(x))


def _gradient_exact(cfg, f, state, lam):
    """The warm-rain transport step and its gradient by autograd, 64 bits."""
    f = {n: t.double() for n, t in f.items()}
    leaves = [t.double().requires_grad_(True) for t in state]
    rdsf = torch.full((cfg.nk,), 1.0 / cfg.dz, device="cuda", dtype=torch.float64)
    new = []
    for q, eps in zip(leaves, (THETA_WEPS, Q_WEPS, Q_WEPS, Q_WEPS)):
        cur = q
        for nrk in (1, 2, 3):
            p = torch.nn.functional.pad(cur[None], (3, 3, 3, 3), mode="replicate")[0]
            p = torch.nn.functional.pad(p, (0, 0, 0, 0, 1, 1))
            cur = q + cfg.dt / (4 - nrk) * _scalar_exact(p, f, rdsf, nrk, cfg, eps)
        new.append(cur)
    th, qv, qc, qr = new[0], new[1], torch.clamp(new[2], min=0.0), torch.clamp(new[3], min=0.0)
    zero = torch.zeros_like(qc)
    ar = torch.where(qc > 0, torch.clamp(0.001 * (qc - 0.001), min=0.0) * cfg.dt, zero)
    rp = torch.where(qr > 0, torch.clamp(qr, min=1e-300) ** 0.875, zero)
    t = torch.minimum(ar + torch.where((qc > 0) & (qr > 0), 2.2 * qc * rp * cfg.dt, zero), qc)
    qc, qr = qc - t, qr + t
    rd, rv, lv2 = _f32(287.04), _f32(461.5), 4190.0 - 1870.0
    lv1, pi = 2501000.0 + lv2 * 273.15, f["pi0"] + f["pp3d"]
    temp = (f["th0"] + th) * pi
    es = torch.minimum(611.2 * torch.exp(17.67 * (temp - 273.15) / (temp - 29.65)), 0.5 * f["prs"])
    qvs = rd / rv * es / (f["prs"] - es)
    lhv = lv1 - lv2 * temp
    dq = (qvs - qv) / (1.0 + lhv * qvs * 17.67 * 243.5 / (1005.7 * (temp - 29.65) ** 2))
    dq = torch.where(qv + dq < 1.0e-20, 1.0e-20 - qv, dq)
    dq = torch.minimum(dq, torch.clamp(qc, min=0.0))
    out = (th - dq * lhv / (1005.7 * pi), qv + dq, qc - dq, qr)
    grads = torch.autograd.grad(sum((w.double() * x).sum() for w, x in zip(lam, out)), leaves)
    return {"state": tuple(x.detach() for x in out), "gradient": grads}


def exact(case, seed):
    """`run`'s outputs in 64 bits.  None for the whole steps: one is some
    thirty coupled operators, and a chain of torch operators for them would
    be a second framework."""
    if case["kind"] in ("step", "dry"):
        return None
    s = prepare(case, seed)
    cfg = s["cfg"]
    if case["kind"] == "gradient":
        return _gradient_exact(cfg, s["fields"], s["state"], s["lam"])
    m = s["m"]
    rds, rdsf = (t.double() for t in _levels(cfg, m))
    if case["kind"] == "acoustic":
        return _acoustic_exact(cfg, m, s["a"], case["nrk"], rds, rdsf)
    if case["kind"] == "momentum":
        return _momentum_exact(cfg, m, s["a"], rds, rdsf)
    if case["kind"] == "tke":
        return _tke_exact(cfg, m, s["a"], case["nrk"], rds)
    f = {n: t.double() for n, t in dict(s["flux"], divx=s["divx"], c1=m["c1"], c2=m["c2"], rr0=m["rr0"]).items()}
    return {"tendency": _scalar_exact(s["scalar"].double(), f, rdsf, case["nrk"], cfg, THETA_WEPS)}
