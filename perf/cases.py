"""Performance cases of the D3Q19 lattice-Boltzmann engine.

Each case is one piece of work a program gives the engine through its public
entry points: a lattice advanced some steps and read back, a capture run, a
drop-in call pair of the reference's pure functions, a gradient through taped
steps, an ensemble of lattices.  ``listed()`` names the cases, ``draw(rng)``
gives further ones of the same ranges, ``prepare`` builds what a program holds
before the call, ``run`` is one pass, ``work`` its bytes and operations, and
``exact`` the same result in 64-bit torch arithmetic without the engine.

Kinds of a case:
  run        Lattice.step(steps), then rho / u into device memory
  monitor    Lattice.step_monitor(steps) (FP64 sums per step), then rho / u
  capture    Lattice.run_capture(steps, every): frames in host arrays
  reference  `steps` times bgk_step + apply_bounce_back_y_walls on host arrays
  gradient   autograd.run through `steps` taped steps, gradient w.r.t. porosity
  ensemble   Batch.step(steps) of `count` lid-driven cavities, rho / u of each

Geometries: ``channel`` (inflow plane, outflow plane, random solid spheres),
``cavity`` (six walls, moving lid), ``couette`` / ``poiseuille`` (walls in y),
``forced`` (periodic, per-cell force field), ``porous`` (inflow, outflow, walls
in y, porosity drag).
"""

from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "bit-physics_b200"))

from lattice_boltzmann_d3q19_b200 import Batch, Lattice, autograd, reference  # noqa: E402

BYTES = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}
INFLOW = 0.04
FLOPS_PER_CELL = 250  # moments, equilibrium and relaxation of 19 directions


def _case(name, kind, geometry, storage, shape, steps, **more):
    nx, ny, nz = shape
    return {"name": name, "kind": kind, "geometry": geometry, "storage": storage, "nx": nx, "ny": ny, "nz": nz,
            "steps": steps, "tau": more.pop("tau", 0.7), **more}


def listed():
    return [
        # The canonical Couette lattice between two readbacks: launches and latency only.
        _case("couette_f64_32x16x3", "run", "couette", "f64", (32, 16, 3), 100),
        # The canonical Poiseuille capture: every step's rho / u to the host.
        _case("poiseuille_capture_64x32x3", "capture", "poiseuille", "f64", (64, 32, 3), 200, every=1),
        # A program written against the reference's pure functions, host arrays in and out.
        _case("reference_pair_64x32x3", "reference", "poiseuille", "f64", (64, 32, 3), 4),
        # Lid-driven cavity, six walls, small enough to stay in L2.
        _case("cavity_f32_64", "run", "cavity", "f32", (64, 64, 64), 100, tau=0.6),
        # Channel past spheres, the headline size, in each arithmetic that is used for it.
        _case("channel_f32_256x128x128", "run", "channel", "f32", (256, 128, 128), 50, tau=0.56),
        _case("channel_f16_256x128x128", "run", "channel", "f16", (256, 128, 128), 50, tau=0.56),
        _case("channel_f64_256x128x128", "run", "channel", "f64", (256, 128, 128), 20, tau=0.56),
        # The largest size of the precision sweep.
        _case("channel_bf16_512x256x256", "run", "channel", "bf16", (512, 256, 256), 20, tau=0.8),
        # Sizes of a user's own mesh: no axis a multiple of anything, odd rows.
        _case("channel_f16_150x101x75", "run", "channel", "f16", (150, 101, 75), 50, tau=0.56),
        # Production stepping with the mass / momentum drift watched in FP64 every step.
        _case("monitor_f32_192x96x98", "monitor", "channel", "f32", (192, 96, 98), 50, tau=0.56),
        # One iteration of a porosity optimisation: taped forward and adjoint.
        _case("gradient_f32_128", "gradient", "porous", "f32", (128, 128, 128), 100, tau=0.6, every=25),
        # Parameter study: independent cavities of mixed sizes advanced together.
        _case("ensemble_f16_16x96", "ensemble", "cavity", "f16", (96, 96, 96), 20, count=16, tau=0.7),
    ]


#: What a drawn case may cost: cell updates and population bytes of a run, at most the largest listed case's.
MOST_UPDATES = 512 * 256 * 256 * 20
MOST_BYTES = MOST_UPDATES * 38


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choices(["run", "monitor", "capture", "reference", "gradient", "ensemble"], [12, 2, 2, 1, 2, 1])[0]
    tau = rng.choice([0.51, 0.56, 0.6, 0.7, 0.8])
    if kind in ("capture", "reference"):
        shape = (_log_int(rng, 16, 64), _log_int(rng, 8, 48), rng.choice([3, 3, 4, 8, 17]))
        geometry = rng.choice(["poiseuille", "couette"])
        if kind == "reference":
            return _drawn(kind, geometry, "f64", shape, rng.randint(1, 6), tau=0.7)
        return _drawn(kind, geometry, rng.choice(["f64", "f64", "f32"]), shape, rng.randint(20, 300), tau=0.7,
                      every=rng.choice([1, 1, 10]))
    if kind == "ensemble":
        size, count = rng.randint(40, 96), rng.randint(4, 24)
        return _drawn(kind, "cavity", rng.choice(["f16", "f32"]), (size, size, size), rng.randint(8, 24),
                      tau=tau, count=count, schedule=rng.choice(["branches", "single"]))
    if kind == "gradient":
        shape = tuple(_log_int(rng, 24, 128) for _ in range(3))
        steps = rng.randint(20, 100)
        return _drawn(kind, "porous", rng.choice(["f32", "f32", "f16", "f64"]), shape, steps, tau=0.6,
                      every=rng.randint(5, 50))
    geometry = rng.choice(["channel", "channel", "channel", "cavity", "couette", "poiseuille", "forced"])
    storage = rng.choice(["f32", "f16", "bf16", "f64"])
    if geometry in ("couette", "poiseuille"):
        shape = (_log_int(rng, 16, 256), _log_int(rng, 8, 128), _log_int(rng, 3, 128))
    elif geometry == "cavity":
        shape = tuple(_log_int(rng, 24, 192) for _ in range(3))
    else:
        shape = (_log_int(rng, 32, 512), _log_int(rng, 24, 256), _log_int(rng, 24, 256))
    cells = shape[0] * shape[1] * shape[2]
    most = min(MOST_UPDATES // cells, MOST_BYTES // (cells * 19 * BYTES[storage]), 200)
    steps = rng.randint(max(1, min(8, most)), max(8, most)) if most > 8 else max(1, most)
    return _drawn(kind, geometry, storage, shape, steps, tau=tau)


def _drawn(*args, **kw):
    case = _case("", *args, **kw)
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# Inputs, from the seed alone
# ---------------------------------------------------------------------------

def _noise(gen, comps, shape):
    """Smooth random fields in [-1, 1] (trilinear from an 8^3 grid), f64 on the GPU."""
    coarse = (2.0 * torch.rand((1, comps, 8, 8, 8), generator=gen, dtype=torch.float64) - 1.0).cuda()
    return torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0].contiguous()


def _spheres(rng, shape):
    """uint8 cell types: inflow plane, outflow plane, solid spheres in the middle of the channel."""
    nx, ny, nz = shape
    scale = min(nx / 256.0, ny / 128.0, nz / 128.0)
    flags = np.zeros(shape, np.uint8)
    ys, zs = np.arange(ny, dtype=np.float64), np.arange(nz, dtype=np.float64)
    for _ in range(40):
        c = rng.uniform(0.2 * nx, 0.8 * nx), rng.uniform(0.0, ny), rng.uniform(0.0, nz)
        r = rng.uniform(4.0, 10.0) * scale
        dy, dz = np.abs(ys - c[1]), np.abs(zs - c[2])
        d2 = np.minimum(dy, ny - dy)[:, None] ** 2 + np.minimum(dz, nz - dz)[None, :] ** 2
        for x in range(max(0, math.ceil(c[0] - r)), min(nx, math.floor(c[0] + r) + 1)):
            flags[x][(x - c[0]) ** 2 + d2 <= r * r] = 1
    flags[0], flags[-1] = 2, 3
    return flags


def _inputs(case, seed):
    """Initial rho / u (f64 GPU tensors) and the lattice's configuration."""
    shape = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator().manual_seed(seed)
    rng = np.random.default_rng(seed)
    noise = _noise(gen, 4, shape)
    g = case["geometry"]
    cfg = {"shape": shape, "tau": case["tau"], "periodic": (True, True, True), "walls": {}, "force_mode": "none",
           "body": (0.0, 0.0, 0.0), "inflow_u": (0.0, 0.0, 0.0), "flags": None, "field": None, "alpha": None,
           "drag_k": 0.0}
    rho = 1.0 + 0.002 * noise[0]
    u = 0.01 * noise[1:]
    if g == "channel":
        cfg |= {"flags": _spheres(rng, shape), "inflow_u": (INFLOW, 0.0, 0.0)}
        u[0] += INFLOW
    elif g == "cavity":
        cfg |= {"periodic": (False, False, False), "walls": {"y+": (0.05, 0.0, 0.0)}}
    elif g == "couette":
        cfg |= {"periodic": (True, False, True), "walls": {"y+": (0.05, 0.0, 0.0)}}
    elif g == "poiseuille":
        # the canonical force at 32 rows and tau 0.7; at other heights the same mean velocity
        force = 1e-5 * (32.0 / shape[1]) ** 2 * (case["tau"] - 0.5) / 0.2
        cfg |= {"periodic": (True, False, True), "force_mode": "uniform", "body": (force, 0.0, 0.0)}
    elif g == "forced":
        cfg |= {"force_mode": "field", "field": 1e-6 * _noise(gen, 3, shape)}
    elif g == "porous":
        flags = np.zeros(shape, np.uint8)
        flags[0], flags[-1] = 2, 3
        cfg |= {"flags": flags, "inflow_u": (INFLOW, 0.0, 0.0), "periodic": (True, False, True),
                "force_mode": "drag", "drag_k": 0.05, "alpha": (0.5 + 0.5 * _noise(gen, 1, shape)[0]).float()}
        rho = torch.ones_like(rho)
        u = torch.zeros_like(u)
    return rho, u, cfg


def _lattice(case, cfg, stream):
    lat = Lattice(cfg["shape"], cfg["tau"], storage=case["storage"], periodic=cfg["periodic"],
                  wall_velocity=cfg["walls"], force_mode=cfg["force_mode"], body_force=cfg["body"],
                  drag_k=cfg["drag_k"], inflow_u=cfg["inflow_u"])
    lat.set_stream(stream.cuda_stream)
    if cfg["flags"] is not None:
        lat.set_flags(cfg["flags"])
    if cfg["field"] is not None:
        lat.set_force_field(cfg["field"].cpu().numpy())
    return lat


def _fields(case, shape):
    """rho / u buffers on the device, and their f32 copies, which programs on reduced storages keep."""
    rho = torch.empty(shape, dtype=torch.float64, device="cuda")
    u = torch.empty((3, *shape), dtype=torch.float64, device="cuda")
    if case["storage"] == "f64":
        return rho, u, rho, u
    return rho, u, torch.empty_like(rho, dtype=torch.float32), torch.empty_like(u, dtype=torch.float32)


def _cavities(case, seed):
    rng = np.random.default_rng(seed)
    n = case["nx"]
    # Sizes are the case's, not the seed's: the work of a pass does not depend on the inputs.
    sizes = np.random.default_rng(7 * n + case["count"]).integers(max(16, n // 3), n + 1, size=(case["count"], 3))
    return [dict(shape=tuple(int(v) for v in s), tau=case["tau"], storage=case["storage"],
                 periodic=(False, False, False), wall_velocity={"y+": (float(rng.uniform(0.02, 0.08)), 0.0, 0.0)})
            for s in sizes]


def _cavity_start(k, seed, shape):
    noise = _noise(torch.Generator().manual_seed(1000 * seed + k), 4, shape)
    return 1.0 + 0.002 * noise[0], 0.01 * noise[1:]


def prepare(case, seed):
    if case["kind"] == "ensemble":
        specs = _cavities(case, seed)
        batch = Batch(specs)
        if case.get("schedule", "branches") == "branches":
            batch.set_schedule("branches", 128, 8)
        fields = []
        for k, spec in enumerate(specs):
            rho, u = _cavity_start(k, seed, spec["shape"])
            batch[k].set_equilibrium(rho.cpu().numpy(), u.cpu().numpy())
            fields.append(_fields(case, spec["shape"]))
        return {"case": case, "batch": batch, "fields": fields}
    rho, u, cfg = _inputs(case, seed)
    if case["kind"] == "reference":
        f = reference.feq_field(rho.cpu().numpy(), u.cpu().numpy())
        force = np.zeros((3, *cfg["shape"]))
        force[0] = cfg["body"][0]
        return {"case": case, "f": f, "force": force if cfg["force_mode"] != "none" else None,
                "top": cfg["walls"].get("y+", (0.0, 0.0, 0.0))}
    stream = torch.cuda.Stream()
    lat = _lattice(case, cfg, stream)
    state = {"case": case, "lat": lat, "stream": stream}
    if case["kind"] == "gradient":
        state["alpha"] = cfg["alpha"].requires_grad_(True)
        return state
    lat.set_equilibrium(rho.cpu().numpy(), u.cpu().numpy())
    if case["kind"] != "capture":
        state["fields"] = _fields(case, cfg["shape"])
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _read(lat, fields):
    rho, u, rho_out, u_out = fields
    lat.rho_u_device(rho.data_ptr(), u.data_ptr())
    if rho_out is not rho:
        rho_out.copy_(rho)
        u_out.copy_(u)
    return {"rho": rho_out, "u": u_out}


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        batch = state["batch"]
        batch.step(steps)
        for k, (rho, u, _, _) in enumerate(state["fields"]):
            batch[k].rho_u_device(rho.data_ptr(), u.data_ptr())
        batch.synchronize()  # the batch has a stream of its own
        rhos, us, rho_outs, u_outs = zip(*state["fields"])
        if rho_outs[0] is not rhos[0]:
            torch._foreach_copy_(list(rho_outs + u_outs), list(rhos + us))
        return {"rho": list(rho_outs), "u": list(u_outs)}
    if kind == "reference":
        f, force, top = state["f"], state["force"], state["top"]
        for _ in range(steps):
            f = reference.bgk_step(f, case["tau"], force)
            f = reference.apply_bounce_back_y_walls(f, wall_velocity_top=top)
        return {"f": f, "rho": reference.density_field(f), "u": reference.macroscopic_velocity(f, force)}
    lat = state["lat"]
    if kind == "capture":
        _, rho, u = lat.run_capture(steps, case["every"])
        return {"rho": rho, "u": u}
    with torch.cuda.stream(state["stream"]):
        if kind == "gradient":
            alpha = state["alpha"]
            rho, u = autograd.run(lat, alpha, steps, checkpoint_every=case["every"])
            loss = autograd.box_kinetic_energy(rho, u, (1, case["nx"] // 2))  # what the inflow has reached
            (grad,) = torch.autograd.grad(loss, alpha)
            return {"rho": rho.detach().float() if case["storage"] != "f64" else rho.detach(),
                    "u": u.detach().float() if case["storage"] != "f64" else u.detach(), "grad": grad}
        if kind == "monitor":
            sums = lat.step_monitor(steps)
            return {"sums": sums, **_read(lat, state["fields"])}
        lat.step(steps)
        return _read(lat, state["fields"])


def work(case):
    """Populations in and out once, rho / u (f64) out, fields in once; the collision's operations of every step."""
    size, steps = BYTES[case["storage"]], case["steps"]
    if case["kind"] == "ensemble":
        cells = sum(int(np.prod(s["shape"])) for s in _cavities(case, 0))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    per_cell = 2 * 19 * size + 32
    flops = FLOPS_PER_CELL * cells * steps
    if case["geometry"] in ("channel", "porous"):
        per_cell += 1
    if case["geometry"] == "forced":
        per_cell += 3 * (8 if size == 8 else 4)
    if case["kind"] == "capture":
        frames = steps // case["every"] + 1 + (1 if steps % case["every"] else 0)
        per_cell = 2 * 19 * size + 32 * frames
    if case["kind"] == "gradient":
        per_cell += 4 + 4 + 32  # alpha, its gradient, the seeds
        flops *= 3  # forward, and the adjoint of moments, equilibrium and relaxation
    return {"bytes": cells * per_cell, "flops": flops}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------

_C = ([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
      + [(a, b, 0) for a, b in ((1, 1), (-1, -1), (1, -1), (-1, 1))]
      + [(a, 0, b) for a, b in ((1, 1), (-1, -1), (1, -1), (-1, 1))]
      + [(0, a, b) for a, b in ((1, 1), (-1, -1), (1, -1), (-1, 1))])
_W = [1.0 / 3.0] + [1.0 / 18.0] * 6 + [1.0 / 36.0] * 12
_OPP = [_C.index((-a, -b, -c)) for a, b, c in _C]


def _dot(c, v):
    out = None
    for a, x in zip(c, v):
        if a:
            t = x if a > 0 else -x
            out = t if out is None else out + t
    return torch.zeros_like(v[0]) if out is None else out


def _feq(rho, u):
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    out = []
    for c, w in zip(_C, _W):
        cu = _dot(c, u)
        out.append(w * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq))
    return out


class _Exact:
    def __init__(self, cfg):
        self.cfg, self.tau, shape = cfg, cfg["tau"], cfg["shape"]
        grid = [torch.arange(n, device="cuda").view([-1 if k == a else 1 for k in range(3)]).expand(shape)
                for a, n in enumerate(shape)]
        types = torch.zeros(shape, dtype=torch.uint8, device="cuda")
        if cfg["flags"] is not None:
            types = torch.from_numpy(cfg["flags"]).cuda()
        self.solid, self.inflow, self.outflow = types == 1, types == 2, types == 3
        one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
        self.inflow_f = [float(v) for v in _feq(one, [one * v for v in cfg["inflow_u"]])]
        # per direction: the walled face its pull crosses (the first of y+, y-, x-, x+, z-, z+)
        self.face, self.gain, self.behind = [], [], []
        for c, w in zip(_C, _W):
            hit, gain = torch.zeros(shape, dtype=torch.bool, device="cuda"), torch.zeros(shape, dtype=torch.float64, device="cuda")
            for axis, sign, name in ((1, -1, "y+"), (1, 1, "y-"), (0, 1, "x-"), (0, -1, "x+"), (2, 1, "z-"), (2, -1, "z+")):
                if cfg["periodic"][axis] or c[axis] != sign:
                    continue
                new = (grid[axis] == (shape[axis] - 1 if sign < 0 else 0)) & ~hit
                uw = cfg["walls"].get(name, (0.0, 0.0, 0.0))
                gain = torch.where(new, -6.0 * w * sum(a * b for a, b in zip(c, uw)), gain)
                hit = hit | new
            self.face.append(hit if bool(hit.any()) else None)
            self.gain.append(gain if bool(hit.any()) else None)
            behind = torch.roll(self.solid, c, (0, 1, 2)) & ~hit & ~self.solid
            self.behind.append(behind if bool(behind.any()) else None)
        self.special = {k: bool(getattr(self, k).any()) for k in ("solid", "inflow", "outflow")}

    def force(self, m, alpha):
        cfg, mode = self.cfg, self.cfg["force_mode"]
        if mode == "uniform":
            return [torch.full_like(m[0], v) for v in cfg["body"]]
        if mode == "field":
            return list(cfg["field"])
        if mode == "drag":
            ka = cfg["drag_k"] * alpha
            beta = ka / (1.0 + 0.5 * ka)
            return [-beta * v for v in m]
        return None

    def moments(self, f, alpha):
        rho = sum(f[1:], f[0])
        m = [sum(c[a] * v for c, v in zip(_C, f) if c[a]) for a in range(3)]
        F = self.force(m, alpha)
        u = [(v if F is None else v + 0.5 * F[a]) / rho for a, v in enumerate(m)]
        return rho, u, F

    def collide(self, f, alpha):
        rho, u, F = self.moments(f, alpha)
        usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        out = []
        for c, w, v in zip(_C, _W, f):
            cu = _dot(c, u)
            p = v - (v - w * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq)) / self.tau
            if F is not None:
                cF = _dot(c, F)
                uF = u[0] * F[0] + u[1] * F[1] + u[2] * F[2]
                p = p + (1.0 - 0.5 / self.tau) * w * (3.0 * (cF - uF) + 9.0 * cu * cF)
            out.append(torch.where(self.solid, w, p) if self.special["solid"] else p)
        return out

    def resolve(self, P):
        g = [torch.roll(v, c, (0, 1, 2)) if any(c) else v for c, v in zip(_C, P)]
        walled = any(h is not None for h in self.face)
        rho_w = sum(g[1:], g[0]) if walled else None
        out = []
        for d in range(19):
            v = g[d]
            if self.behind[d] is not None:
                v = torch.where(self.behind[d], P[_OPP[d]], v)
            if self.face[d] is not None:
                v = torch.where(self.face[d], g[_OPP[d]] + self.gain[d] * rho_w, v)
            if self.special["inflow"]:
                v = torch.where(self.inflow, self.inflow_f[d], v)
            if self.special["solid"]:
                v = torch.where(self.solid, _W[d], v)
            if self.special["outflow"]:
                v = torch.where(self.outflow, torch.roll(v, 1, 0), v)
            out.append(v)
        return out

    def read(self, f, alpha):
        rho, u, _ = self.moments(f, alpha)
        if self.special["solid"]:
            rho, u = torch.where(self.solid, 0.0, rho), [torch.where(self.solid, 0.0, v) for v in u]
        return rho, torch.stack(u)

    def sums(self, f):
        live = [torch.where(self.solid, 0.0, v) for v in f] if self.special["solid"] else f
        m = [sum(c[a] * v for c, v in zip(_C, live) if c[a]) for a in range(3)]
        return [float(v.sum()) for v in (sum(live[1:], live[0]), *m)]

    def start(self, rho, u):
        return _feq(rho, list(u))

    def steps(self, f, n, alpha=None, seen=None):
        for _ in range(n):
            if seen is not None:
                seen(f)
            f = self.resolve(self.collide(f, alpha))
        return f


def _exact_gradient(case, ex, rho, u, alpha):
    from torch.utils.checkpoint import checkpoint

    a = alpha.detach().double().requires_grad_(True)
    f = ex.start(rho, u)
    for _ in range(case["steps"]):
        f = list(checkpoint(lambda a, *f: tuple(ex.steps(list(f), 1, a)), a, *f, use_reentrant=False))
    r, v = ex.read(f, a)
    x1 = case["nx"] // 2
    (grad,) = torch.autograd.grad(0.5 * (r[1:x1] * (v[:, 1:x1] ** 2).sum(0)).sum(), a)
    return {"rho": r.detach(), "u": v.detach(), "grad": grad}


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        out = {"rho": [], "u": []}
        for k, spec in enumerate(_cavities(case, seed)):
            ex = _Exact({"shape": spec["shape"], "tau": spec["tau"], "periodic": spec["periodic"],
                         "walls": spec["wall_velocity"], "force_mode": "none", "flags": None,
                         "inflow_u": (0.0, 0.0, 0.0)})
            rho, u = ex.read(ex.steps(ex.start(*_cavity_start(k, seed, spec["shape"])), steps), None)
            out["rho"].append(rho)
            out["u"].append(u)
        return out
    rho, u, cfg = _inputs(case, seed)
    ex = _Exact(cfg)
    if kind == "gradient":
        # about 250 f64 fields of the lattice live through one step's backward
        if case["nx"] * case["ny"] * case["nz"] * (19 * steps + 400) * 8 > 120e9:
            return None
        return _exact_gradient(case, ex, rho, u, cfg["alpha"])
    f = ex.start(rho, u)
    if kind == "capture":
        frames = []
        for s in range(steps + 1):
            if s % case["every"] == 0 or s == steps:
                frames.append(ex.read(f, None))
            if s < steps:
                f = ex.steps(f, 1)
        return {"rho": torch.stack([r for r, _ in frames]), "u": torch.stack([v for _, v in frames])}
    if kind == "monitor":
        sums = []
        f = ex.steps(f, steps, seen=lambda f: sums.append(ex.sums(f)))
        r, v = ex.read(f, None)
        return {"sums": torch.tensor(sums, dtype=torch.float64), "rho": r, "u": v}
    f = ex.steps(f, steps)
    r, v = ex.read(f, None)
    if kind == "reference":
        return {"f": torch.stack(f), "rho": r, "u": v}
    return {"rho": r, "u": v}
