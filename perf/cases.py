"""The workloads the library's speed is measured on, and what each computes in 64 bits.

A case is a plain dict.  Its `kind` says which public entry points a pass goes through:

  step    a host-owned state goes in (`write_state_ptr`, pinned buffers), `steps` calls of
          `step(dt)`, and the state comes back (`read_state_ptr`): a simulation loop that draws
          or logs its particles
  grad    the same under a tape, then `step_backward` with the loss's cotangents: one optimiser
          iteration over a short rollout
  bodies  a game tick with one coupled rigid box (`step_with_bodies`)
  sort    `sort_by_cell_noalloc` on device arrays the caller owns

Scenes are dam breaks: a block of nx x ny x nz lattice particles, jittered, in the corner of a box
container of tx x ty x tz spacings (tx = 0: no container), with normal initial velocities, as in
the seeded scenes and the precision and adjoint studies of this repository.  Particles are given
in the sort's own order, so no pass pays for a first shuffle that a running simulation never sees.
"""
from __future__ import annotations

import copy
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from solunar_b200 import fluid
from solunar_b200.abi import Arithmetic, BodyPose, FluidSettings, FluidSolver, Positions, Shape, body_handle

CASE = {
    "kind": "step", "solver": "wcsph", "arithmetic": "exact", "relative": False, "warm": False, "tolerance": 0.0,
    "spacing": 0.02, "support": 2.0, "viscosity": 0.15, "gravity": -9.81, "nx": 0, "ny": 0, "nz": 0, "tx": 0, "ty": 0,
    "tz": 0, "origin": 0.0, "jitter": 0.02, "sigma": 0.05, "dt": 2e-4, "steps": 1, "every": 0,
}


def listed():
    def case(name, **fields):
        return dict(CASE, name=name, **fields)

    dam1m = dict(solver="dfsph", spacing=0.01, nx=100, ny=100, nz=100, tx=200, ty=100, tz=100, dt=1e-3)
    return [
        # one frame of a small pool in a game: 21 substeps of 720 particles, launches and latency
        case("wcsph_pool_tick", nx=10, ny=12, nz=6, tx=30, ty=20, tz=10, dt=1.0 / 60.0),
        # the CPU-sized WCSPH dam at support 4, four steps between read-outs
        case("wcsph_dam_8k", support=4.0, viscosity=0.01, nx=20, ny=20, nz=20, tx=50, ty=50, tz=50, steps=4),
        # the forward half of the differentiable WCSPH scene: ~250 neighbours a particle
        case("wcsph_64k_support4", support=4.0, viscosity=0.01, nx=40, ny=40, nz=40, tx=50, ty=50, tz=50, sigma=0.1,
             steps=2),
        # a larger WCSPH scene at the default support, ragged sizes
        case("wcsph_dam_315k", spacing=0.01, nx=61, ny=97, nz=53, tx=122, ty=100, tz=53, dt=3e-4, steps=2),
        # the warm-started DFSPH dam at 0.1 % tolerances, two steps (the second starts warm)
        case("dfsph_dam_250k_warm", **dict(dam1m, nx=50, nz=50), warm=True, tolerance=1e-3, steps=2),
        # the headline scene: one DFSPH step of a million particles with the reference's tolerances
        case("dfsph_dam_1m", **dam1m),
        # the same scene in FAST arithmetic
        case("dfsph_dam_1m_fast", **dam1m, arithmetic="fast"),
        # a free block far from the origin on cell-relative positions, odd sizes
        case("dfsph_far_relative", solver="dfsph", arithmetic="fast", relative=True, spacing=0.01, gravity=0.0, nx=61,
             ny=67, nz=59, origin=1024.0, dt=1e-3, steps=2),
        # the differentiable WCSPH scene: four taped steps, checkpoints, gradients of the initial state
        case("wcsph_grad_64k", kind="grad", support=4.0, viscosity=0.01, nx=40, ny=40, nz=40, tx=50, ty=50, tz=50,
             sigma=0.1, steps=4, every=2),
        # the differentiable DFSPH scene: two taped steps in one checkpoint segment
        case("dfsph_grad_500k", kind="grad", **dict(dam1m, ny=50), steps=2, every=2),
        # a tick of the coupling pool: a box meets the water, which pushes back
        case("wcsph_bodies_75k", kind="bodies", nx=50, ny=30, nz=50, tx=50, ty=60, tz=50, sigma=0.0, dt=1.0 / 60.0),
        # the cell sort for hosts that own the device memory
        case("sort_noalloc_200k", kind="sort", nx=59, ny=61, nz=56, spacing=0.01, jitter=0.45),
    ]


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, odd ones among them."""
    def counts(low, high):
        n = math.exp(rng.uniform(math.log(low), math.log(high)))
        a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
        s = n ** (1.0 / 3.0)
        return {"nx": max(3, round(s * a)), "ny": max(3, round(s * b)), "nz": max(3, round(s / (a * b)))}

    def tank(c):
        return {"tx": 2 * c["nx"], "ty": c["ny"] + rng.randrange(0, 12), "tz": c["nz"]}

    kind = rng.choice(["step", "step", "step", "step", "grad", "bodies", "sort"])
    arithmetic = rng.choice(["exact", "exact", "fast"])
    relative = arithmetic == "fast" and rng.random() < 0.5
    if kind == "sort":
        return dict(CASE, kind="sort", spacing=rng.choice([0.01, 0.02]), jitter=0.45, **counts(500, 230000))
    if kind == "bodies":
        s = rng.randrange(18, 56)
        return dict(CASE, kind="bodies", spacing=1.0 / s, nx=s, ny=s * 6 // 10, nz=s, tx=s, ty=s * 6 // 5, tz=s,
                    sigma=0.0, dt=1.0 / 60.0)
    if rng.random() < 0.5:
        support = rng.choice([2.0, 2.0, 3.0, 4.0])
        c = counts(500, 500000 * (2.0 / support) ** 3)
        return dict(CASE, kind=kind, arithmetic=arithmetic, relative=relative, support=support, viscosity=0.01,
                    steps=rng.randrange(1, 4), every=rng.randrange(0, 3) if kind == "grad" else 0, **c, **tank(c))
    c = counts(500, 600000 if kind == "step" else 250000)
    warm = rng.random() < 0.4
    return dict(CASE, kind=kind, solver="dfsph", arithmetic=arithmetic, relative=relative, spacing=0.01, dt=1e-3,
                warm=warm, tolerance=1e-3 if warm else 0.0, steps=rng.randrange(1, 3),
                every=rng.randrange(0, 3) if kind == "grad" else 0, **c, **tank(c))


# ---- a case's inputs ----------------------------------------------------------------------------

def settings_of(c):
    s = FluidSettings(solver=FluidSolver.DFSPH if c["solver"] == "dfsph" else FluidSolver.WCSPH, spacing=c["spacing"],
                      support=c["support"], viscosity=c["viscosity"], gravity=(0.0, c["gravity"], 0.0),
                      arithmetic=Arithmetic.FAST if c["arithmetic"] == "fast" else Arithmetic.EXACT,
                      positions=Positions.CELL_RELATIVE if c["relative"] else Positions.ABSOLUTE,
                      warm_start=c["warm"])
    if c["tolerance"]:
        s.divergence_tolerance = s.density_tolerance = c["tolerance"]
    return s


def inputs_of(c, seed):
    """Positions and velocities in (cell, id) order, float32."""
    rng = np.random.default_rng(seed)
    h = np.float32(c["spacing"])
    x, y, z = np.meshgrid(*(np.arange(c[k], dtype=np.float32) for k in ("nx", "ny", "nz")), indexing="ij")
    p = (np.stack([x.ravel(), y.ravel(), z.ravel()], 1) + np.float32(0.5)) * h
    p += rng.uniform(-1.0, 1.0, p.shape).astype(np.float32) * np.float32(c["jitter"] * c["spacing"])
    p += np.float32(c["origin"])
    v = rng.standard_normal(p.shape, dtype=np.float32) * np.float32(c["sigma"])
    cell = np.floor(p / np.float32(h * np.float32(c["support"]))).astype(np.int64)
    order = np.lexsort((cell[:, 2], cell[:, 1], cell[:, 0]))
    if c["kind"] == "sort":
        order = rng.permutation(len(p))
    return np.ascontiguousarray(p[order]), np.ascontiguousarray(v[order])


def cotangents_of(c, seed, n):
    g = np.random.default_rng(seed + 1).standard_normal((2, n, 3), dtype=np.float32)
    return g[0], g[1] * np.float32(0.01)


def box_pose(c):
    """The 0.3 m box of the coupling pool, half a spacing above the water and falling."""
    top = c["ny"] * c["spacing"]
    return BodyPose(body_handle(1), (0.5, top + 0.15 + 0.5 * c["spacing"], 0.5), linear_velocity=(0.0, -0.5, 0.0))


def prepare(case, seed):
    p, v = inputs_of(case, seed)
    n = len(p)
    if case["kind"] == "sort":
        ids = np.random.default_rng(seed + 2).permutation(n).astype(np.int32)
        return {"case": case, "n": n, "positions": torch.from_numpy(p).cuda(), "ids": torch.from_numpy(ids).cuda(),
                "order": torch.zeros(n, dtype=torch.int32, device="cuda")}
    w = fluid.FluidWorld(settings_of(case))
    if case["tx"]:
        w.add_box_container((0.0, 0.0, 0.0), tuple(case[k] * case["spacing"] for k in ("tx", "ty", "tz")))
    w.add_particles(p, v)
    state = {"case": case, "n": n, "world": w, "in": [torch.from_numpy(a).pin_memory() for a in (p, v)],
             "out": [torch.empty(n, 3, pin_memory=True) for _ in range(2)]}
    if case["kind"] == "grad":
        state["cotangents"] = cotangents_of(case, seed, n)
    if case["kind"] == "bodies":
        w.couple(body_handle(1), Shape.CUBOID, (0.15, 0.15, 0.15))
        state["pose"] = box_pose(case)
    return state


def run(state):
    case, n = state["case"], state["n"]
    if case["kind"] == "sort":
        radius = float(np.float32(case["spacing"]) * np.float32(case["support"]))
        fluid.sort_by_cell_noalloc(state["positions"].data_ptr(), state["ids"].data_ptr(), n, radius,
                                   state["order"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["order"]
    w, (p, v), (po, vo) = state["world"], state["in"], state["out"]
    w.write_state_ptr(p.data_ptr(), v.data_ptr(), n)
    if case["kind"] == "bodies":
        _, pushes = w.step_with_bodies(case["dt"], [state["pose"]])
        w.read_state_ptr(po.data_ptr(), vo.data_ptr(), n)
        return {"positions": po, "velocities": vo, "lift": torch.tensor([q.lift for q in pushes]),
                "damping": torch.tensor([q.damping for q in pushes])}
    if case["kind"] == "grad":
        w.tape_begin(case["every"])
        for _ in range(case["steps"]):
            w.step(case["dt"])
        dp, dv, g = w.step_backward(*state["cotangents"])
        w.tape_end()
        return {"positions": dp, "velocities": dv, "gravity": torch.tensor(g["gravity"]),
                "viscosity": torch.tensor([g["viscosity"]]), "sound_speed": torch.tensor([g["sound_speed"]])}
    for _ in range(case["steps"]):
        w.step(case["dt"])
    w.read_state_ptr(po.data_ptr(), vo.data_ptr(), n)
    return {"positions": po, "velocities": vo}


def work(case):
    """Each host input and output once, and the pair arithmetic of the passes no substep can leave
    out: for WCSPH a density and a force per pair (20 and 40 operations), for DFSPH the density
    with its factor (35), the viscosity (30) and two solves of the two iterations each takes at
    the least (a check and a push, 10 and 10).  A gradient runs them once and twice as much back."""
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "sort":
        return {"bytes": n * 20, "flops": 0}
    pairs = n * min(4.0 / 3.0 * math.pi * case["support"] ** 3, n)
    radius = case["spacing"] * case["support"]
    per = 60 if case["solver"] == "wcsph" else 35 + 30 + 2 * (3 * 10 + 2 * 10)
    substeps = 1 if case["solver"] == "dfsph" else max(1, math.ceil(case["dt"] * 20.0 / (0.4 * radius)))
    grad = case["kind"] == "grad"
    return {"bytes": n * (96 if grad else 48), "flops": case["steps"] * substeps * pairs * per * (3 if grad else 1)}


# ---- the same in 64 bits ------------------------------------------------------------------------

class Sph64:
    """The WCSPH and DFSPH substeps over pair arrays in float64, from the f32 settings a world holds."""

    def __init__(self, c, device):
        f = np.float32
        self.c, self.device = c, device
        self.h, self.rest = float(f(c["spacing"])), 1000.0
        self.r = float(f(c["spacing"]) * f(c["support"]))
        self.scale = 21.0 / (2.0 * math.pi * self.r ** 3)
        k = np.arange(-math.ceil(c["support"]), math.ceil(c["support"]) + 1)
        d = np.sqrt(sum(a.astype(np.float64) ** 2 for a in np.meshgrid(k, k, k))) * self.h
        q = np.minimum(d / self.r, 1.0)
        self.mass = self.rest / float((self.scale * (1 - q) ** 4 * (1 + 4 * q)).sum())
        t = lambda x: torch.tensor(x, dtype=torch.float64, device=device)  # noqa: E731
        self.g, self.nu, self.sound = t([0.0, float(f(c["gravity"])), 0.0]), t(float(f(c["viscosity"]))), t(20.0)
        self.walls = None
        if c["tx"]:
            layers, n = math.ceil(c["support"]), [c[k] for k in ("tx", "ty", "tz")]
            ax = [np.arange(-layers, m + layers) for m in n]
            ix = np.stack([a.ravel() for a in np.meshgrid(*ax, indexing="ij")], 1)
            ix = ix[~np.all((ix >= 0) & (ix < n), axis=1)]
            self.walls = t(((ix.astype(f) + f(0.5)) * f(c["spacing"])).astype(np.float64))
            self.low, self.high = t([self.h / 2] * 3), t([float(f(m * c["spacing"])) - self.h / 2 for m in n])

    def near(self, a, b):
        """(i, j) with |a_i - b_j| < r, through cells of side r."""
        if b is None:
            z = torch.zeros(0, dtype=torch.long, device=self.device)
            return z, z
        ca, cb = torch.floor(a / self.r).long(), torch.floor(b / self.r).long()
        low = torch.minimum(ca.amin(0), cb.amin(0)) - 1
        span = torch.maximum(ca.amax(0), cb.amax(0)) + 2 - low
        key = lambda q: ((q[:, 0] - low[0]) * span[1] + (q[:, 1] - low[1])) * span[2] + (q[:, 2] - low[2])  # noqa: E731
        kb, order = torch.sort(key(cb))
        ka, found = key(ca), []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                mid = ka + (dx * span[1] + dy) * span[2]
                first, last = torch.searchsorted(kb, mid - 1), torch.searchsorted(kb, mid + 1, right=True)
                count = last - first
                i = torch.repeat_interleave(torch.arange(len(a), device=self.device), count)
                k = torch.arange(len(i), device=self.device) - torch.repeat_interleave(count.cumsum(0) - count, count)
                j = order[first[i] + k]
                keep = (a[i] - b[j]).square().sum(1) < self.r * self.r
                found.append((i[keep], j[keep]))
        return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])

    def geometry(self, x):
        """Pair lists, offsets, kernel gradients and densities at positions x."""
        n = len(x)
        with torch.no_grad():
            i, j = self.near(x, x)
            self.crowd = torch.bincount(i, minlength=n)
            keep = i != j
            self.i, self.j = i[keep], j[keep]
            self.wi, self.wj = self.near(x, self.walls)
            self.crowd += torch.bincount(self.wi, minlength=n)
        self.o = x[self.i] - x[self.j]
        self.wo = x[self.wi] - self.walls[self.wj] if self.walls is not None else x[self.wi]

        def kernel(o):
            d = o.square().sum(1).sqrt()
            q = d / self.r
            grad = self.scale * -20.0 * q * (1 - q) ** 3 / self.r / d
            return self.scale * (1 - q) ** 4 * (1 + 4 * q), o * grad[:, None]

        value, self.G = kernel(self.o)
        wvalue, self.wG = kernel(self.wo)
        total = torch.full((n,), self.scale, dtype=torch.float64, device=self.device)  # the particle itself
        return self.mass * total.index_add(0, self.i, value).index_add(0, self.wi, wvalue)

    def sum3(self, n, fluid_terms, wall_terms):
        zero = torch.zeros(n, 3, dtype=torch.float64, device=self.device)
        return zero.index_add(0, self.i, fluid_terms).index_add(0, self.wi, wall_terms)

    def wall_damping(self, v, rho, dt):
        """The water's motion into a wall, damped pair by pair along the wall's normal."""
        n = len(v)
        nuw = torch.minimum(self.sound * self.r, torch.tensor(0.25 * self.r ** 2 / dt, dtype=torch.float64,
                                                              device=self.device))
        zero = torch.zeros(n, 3, dtype=torch.float64, device=self.device)
        away = zero.index_add(0, self.wi, -self.wG)
        length = away.square().sum(1, keepdim=True)
        normal = torch.where(length > 0, away / torch.where(length > 0, length, 1.0).sqrt(), 0.0)
        into = normal * torch.clamp((v * normal).sum(1, keepdim=True), max=0.0)
        toward = torch.clamp((into[self.wi] * self.wo).sum(1), max=0.0)
        damp = -nuw * toward / (self.wo.square().sum(1) + 0.01 * self.r ** 2) / rho[self.wi]
        return zero.index_add(0, self.wi, -self.wG * (self.mass * damp)[:, None])

    def pair_damping(self, v, rho, dt):
        nu = torch.minimum(self.nu * self.sound * self.r, torch.tensor(0.05 * self.r ** 2 / dt, dtype=torch.float64,
                                                                       device=self.device))
        toward = torch.clamp(((v[self.i] - v[self.j]) * self.o).sum(1), max=0.0)
        return -nu * toward / (self.o.square().sum(1) + 0.01 * self.r ** 2) * 2.0 / (rho[self.i] + rho[self.j])

    def advance(self, x, v, dt):
        y = x + v * dt
        if self.walls is not None:
            inside = torch.minimum(torch.maximum(y, self.low), self.high)
            v = torch.where(inside != y, 0.0, v)
            y = inside
        return y, v

    def wcsph(self, x, v, dt):
        rho = self.geometry(x)
        stiffness = self.rest * self.sound ** 2 / 7.0
        ratio = torch.clamp(rho / self.rest, max=float(np.float32(1.1)))
        press = torch.clamp(stiffness * (ratio ** 7 - 1.0), min=0.0)
        s = press / rho ** 2
        term = self.mass * (s[self.i] + s[self.j] + self.pair_damping(v, rho, dt))
        wall = self.mass * (s + press / self.rest ** 2)[self.wi]
        a = self.sum3(len(x), -self.G * term[:, None], -self.wG * wall[:, None])
        a = a + self.wall_damping(v, rho, dt) + self.g
        return self.advance(x, v + a * dt, dt)

    def rate(self, v):
        zero = torch.zeros(len(v), dtype=torch.float64, device=self.device)
        rate = zero.index_add(0, self.i, ((v[self.i] - v[self.j]) * self.G).sum(1))
        return self.mass * rate.index_add(0, self.wi, (v[self.wi] * self.wG).sum(1))

    def push(self, v, kappa, dt):
        own = self.mass * kappa
        return v - dt * self.sum3(len(v), self.G * (own[self.i] + own[self.j])[:, None],
                                  self.wG * own[self.wi][:, None])

    def check(self, which, v, rho, dt):
        """Each particle's stiffness over its factor, and its error."""
        rate = self.rate(v)
        if which:
            over = torch.clamp(rho + dt * rate - self.rest, min=0.0)
            return over / dt ** 2, over / self.rest
        positive = torch.where(self.crowd < 20, 0.0, torch.clamp(rate, min=0.0))
        return positive / dt, dt * positive / self.rest

    def solve(self, which, v, rho, alpha, dt, grad):
        c = self.c
        tolerance = float(np.float32(c["tolerance"] or (5e-4 if which else 1e-3)))
        if c["warm"]:
            kappa = 0.5 * self.impulse[which] / dt
            self.impulse[which] = kappa * dt
            v = self.push(v, kappa, dt)
        here = copy.copy(self)  # this substep's pairs, for the backward's second run of an iteration
        for iteration in range(101):
            with torch.no_grad():
                _, error = self.check(which, v, rho, dt)
                loaded = max(1, int((error > 0).sum()))
                if iteration >= 2 and float(error.sum()) / loaded <= tolerance or iteration == 100:
                    return v

            def iterate(v):
                kappa = here.check(which, v, rho, dt)[0] * alpha
                return here.push(v, kappa, dt), kappa

            v, kappa = checkpoint(iterate, v, use_reentrant=False) if grad else iterate(v)
            if c["warm"]:
                self.impulse[which] = self.impulse[which] + kappa * dt

    def dfsph(self, x, v, dt, grad):
        rho = self.geometry(x)
        total = self.sum3(len(x), self.mass * self.G, self.mass * self.wG).square().sum(1)
        total = total.index_add(0, self.i, self.mass ** 2 * self.G.square().sum(1))
        alpha = torch.where(total > 0, 1.0 / torch.where(total > 0, total, 1.0), 0.0)
        v = self.solve(0, v, rho, alpha, dt, grad)
        damp = self.mass * self.pair_damping(v, rho, dt)
        zero = torch.zeros_like(v)
        v = v + dt * (zero.index_add(0, self.i, -self.G * damp[:, None]) + self.wall_damping(v, rho, dt) + self.g)
        v = self.solve(1, v, rho, alpha, dt, grad)
        return self.advance(x, v, dt)

    def step(self, x, v, dt, grad=False):
        if self.c["solver"] == "dfsph":
            return self.dfsph(x, v, dt, grad)
        fastest = float(v.detach().square().sum(1).amax().sqrt())
        substeps = max(1, math.ceil(dt / (float(np.float32(0.4)) * self.r / (20.0 + fastest))))
        for _ in range(substeps):
            x, v = self.wcsph(x, v, dt / substeps)
        return x, v


def exact(case, seed):
    """The case in float64 from the same float32 inputs.  None for `bodies`, whose body points and
    lift are sampled in float32 by their definition, and for `sort`, which gives whole numbers."""
    if case["kind"] in ("bodies", "sort"):
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    p, v = inputs_of(case, seed)
    x, u = (torch.from_numpy(a).to(device, torch.float64) for a in (p, v))
    m, dt, grad = Sph64(case, device), float(np.float32(case["dt"])), case["kind"] == "grad"
    m.impulse = [torch.zeros(len(p), dtype=torch.float64, device=device) for _ in range(2)]
    wanted = [x, u, m.g, m.nu, m.sound]
    if grad:
        for t in wanted:
            t.requires_grad_(True)
    y, w = x, u
    with torch.set_grad_enabled(grad):
        for _ in range(case["steps"]):
            y, w = m.step(y, w, dt, grad)
        if not grad:
            return {"positions": y, "velocities": w}
        dp, dv = (torch.from_numpy(a).to(device, torch.float64) for a in cotangents_of(case, seed, len(p)))
        loss = (y * dp).sum() + (w * dv).sum()
    got = torch.autograd.grad(loss, wanted, allow_unused=True)
    gx, gv, gg, gn, gs = (torch.zeros_like(t) if g is None else g for t, g in zip(wanted, got))
    return {"positions": gx, "velocities": gv, "gravity": gg, "viscosity": gn.reshape(1), "sound_speed": gs.reshape(1)}
