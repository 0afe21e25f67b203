"""Workloads of the LBM framework, as its users run them.

Every case goes through the public Python API (b200lbm.Sim, RigidSphere,
CompositeSolid, Batch).  A pass is one stretch of simulation work:

  tick    the host-driven worker tick, Sim.step / absorbDeadCells /
          RigidSphere.step, `steps` times, then the packed frame
          (src/worker.js:94-111 of the reference) and, where asked for, a read
          of the fields
  stream  the same tick with the frame of every second step delivered into two
          alternating page-locked buffers while the next steps run
  run     `steps` ticks on the device (Sim.run_coupled), with or without frames
          on the way, then a read of phi, rho and u
  phases  the seven phases of a step called one by one, as a program with its
          own solid or its own instrumentation between them does
  batch   many independent scenes of uneven sizes advanced together with the
          frame every server tick delivers

A case is a dict of plain values: `api`, the grid (`nx`, `ny`, `nz`), the
population storage, the number of steps, `frame_every`, the number of spheres,
the physics (`pool`: liquid below, gravity -1e-5, the benchmark's scene family;
`tank`: the interactive demo's parameters) and, for batches, the number of
scenes and the range of their edges.  Levels, sphere positions, radii,
densities and velocities come from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "claude-vibe-code-raytracing_b200"))

import b200lbm  # noqa: E402

PHYSICS = {
    "pool": dict(tau=0.6, tauPhi=0.8, sigma=1e-3, gravity=-1e-5, rhoL=1.0, rhoG=0.1, W=4.0),
    "tank": dict(tau=0.85, tauPhi=0.7, sigma=0.008, gravity=0.0015, rhoL=1.0, rhoG=0.1, W=4.0),
}
FIELDS = ("phi", "rho", "ux", "uy", "uz")
# algorithmic bytes per interior cell and step: 34 populations and 5 macros
# read and written once, one tag read
STEP_BYTES = {"f32": 313, "f16": 177, "bf16": 177, "f64": 626}
STEP_FLOPS = 600


def _case(name, api, nx, ny, nz, storage="f32", steps=1, frame_every=0, spheres=1, physics="pool", scenes=0):
    c = dict(api=api, nx=nx, ny=ny, nz=nz, storage=storage, steps=steps, frame_every=frame_every,
             spheres=spheres, physics=physics, scenes=scenes)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's smoke scene: one tick and a look at the fields
        _case("tick-12", "tick", 12, 12, 12, physics="tank"),
        # the demo's worker frame at its own grid: two ticks and a packed frame
        _case("worker-frame-40x28x40", "tick", 40, 28, 40, steps=2, frame_every=2, physics="tank"),
        # the demo grid run on the device, 80 ticks (the reference's own bench length)
        _case("run-40x28x40", "run", 40, 28, 40, steps=80, physics="tank"),
        # no edge a multiple of anything
        _case("run-61x47x83", "run", 61, 47, 83, steps=60),
        # a middling scene with three spheres in FP16, frames on the way
        _case("run-128x97x110-f16", "run", 128, 97, 110, "f16", steps=80, frame_every=20, spheres=3),
        # a finer demo tank, host-driven, every second frame streamed out
        _case("stream-160x112x160", "stream", 160, 112, 160, steps=40, frame_every=2),
        # the FP64 form, which precision studies compare with
        _case("run-96x80x72-f64", "run", 96, 80, 72, "f64", steps=30),
        # the phase-by-phase path (programs with their own solids)
        _case("phases-112x96x120", "phases", 112, 96, 120, steps=10),
        # one server tick pair of mixed scenes in FP16
        _case("batch-16", "batch", 32, 32, 32, "f16", steps=40, frame_every=20, scenes=16),
        # the benchmark grid, plain FP32 and FP16
        _case("run-256", "run", 256, 256, 256, steps=80),
        _case("run-256-f16", "run", 256, 256, 256, "f16", steps=80),
        # a grid past 2^31 population elements, BF16, with its last frame
        _case("run-448x400x440-bf16", "run", 448, 400, 440, "bf16", steps=16, frame_every=16, spheres=2),
    ]


def draw(rng):
    """Single scenes from 10 to about 280 cells an edge (their logarithms spread
    evenly), every API and storage form; batches of 2 to 16 scenes."""
    api = rng.choice(("run", "run", "run", "tick", "stream", "phases", "batch"))
    if api == "batch":
        return _case(None, api, 32, 32, 32, rng.choice(("f16", "f16", "f32", "bf16")), 2 * rng.randint(5, 20),
                     rng.choice((0, 10)), scenes=rng.randint(2, 16))
    top = 150 if api == "phases" else 280
    base = math.exp(rng.uniform(math.log(12), math.log(top)))
    nx, ny, nz = (max(10, min(288, int(round(base * rng.uniform(0.75, 1.3))))) for _ in range(3))
    if rng.random() < 0.35:
        nx = max(16, nx // 16 * 16)
    storage = "f32" if api == "phases" else rng.choice(("f32", "f32", "f32", "f16", "f16", "bf16", "f64"))
    cells = nx * ny * nz
    if storage == "f64" and cells > 4_000_000:
        storage = "f32"
    physics = "tank" if max(nx, ny, nz) <= 48 and rng.random() < 0.5 else "pool"
    if api == "run":
        steps = max(4, min(100, int(1.2e9 / cells) // 2 * 2))
    elif api == "stream":
        steps = max(4, min(40, int(5.0e8 / cells) // 2 * 2))
    elif api == "phases":
        steps = max(2, min(20, int(2.0e7 / cells)))
    else:
        steps = rng.choice((1, 2, 2, 10)) if cells < 1_000_000 else 2
    frame = {"run": rng.choice((0, 0, steps // 2)), "stream": 2, "tick": rng.choice((0, steps)), "phases": 0}[api]
    return _case(None, api, nx, ny, nz, storage, steps, frame, rng.choice((1, 1, 1, 2, 3)), physics)


# ------------------------------------------------------------------ scenes
def _scene(rs, nx, ny, nz, nsph, physics):
    """Waterline and spheres of one scene: a pool (or a tank filled from its
    high y side) with spheres around the interface, inside the walls'
    clamp margin r + 1.5 and apart from each other, moving at up to 0.02."""
    level = rs.uniform(0.3, 0.6) * ny
    edge = min(nx, ny, nz)
    placed = []
    for _ in range(200):
        if len(placed) == nsph:
            break
        r = min(rs.uniform(0.10, 0.17) * edge, 24.0)
        m = r + 1.5
        if edge - 1 - 2 * m <= 0.5:
            r = 0.12 * edge
            m = r + 1.5
        c = [rs.uniform(m, n - 1 - m) for n in (nx, ny, nz)]
        # near the interface, so that the sphere meets both fluids
        c[1] = float(np.clip(level + rs.uniform(-1.5, 1.5) * r, m, ny - 1 - m))
        if any(math.dist(c, p["c"]) <= r + p["r"] + 1 for p in placed):
            continue
        d = rs.normal(size=3)
        v = rs.uniform(0.005, 0.02) * d / (np.linalg.norm(d) or 1.0)
        placed.append(dict(c=c, r=r, density=rs.uniform(1.2, 3.0), v=[float(x) for x in v]))
    sign = 1.0 if physics == "tank" else -1.0
    W = PHYSICS[physics]["W"]
    column = 0.5 * (1 + np.tanh(sign * 2 * (np.arange(ny, dtype=np.float64) - level) / W))
    return dict(dims=(nx, ny, nz), column=column, spheres=placed, physics=PHYSICS[physics])


def _scenes(case, seed):
    rs = np.random.RandomState((seed * 2654435761 + 12345) % (1 << 32))
    if case["api"] != "batch":
        return [_scene(rs, case["nx"], case["ny"], case["nz"], case["spheres"], case["physics"])]
    # the edges are the case's, not the seed's: the same sizes for every seed
    sizes = np.random.RandomState(case["scenes"])
    out = []
    for _ in range(case["scenes"]):
        nx, ny, nz = (int(v) for v in sizes.randint(case["nx"], 161, size=3))
        out.append(_scene(rs, nx, ny, nz, int(sizes.randint(1, 4)), case["physics"]))
    return out


def _build(scene, storage):
    nx, ny, nz = scene["dims"]
    sim = b200lbm.Sim(nx, ny, nz, storage=storage)
    for k, v in scene["physics"].items():
        setattr(sim, k, v)
    sim.initProfile(scene["column"])
    balls = []
    for p in scene["spheres"]:
        b = b200lbm.RigidSphere(nx, ny, nz, cx=p["c"][0], cy=p["c"][1], cz=p["c"][2], r=p["r"], density=p["density"])
        b.vx, b.vy, b.vz = p["v"]
        balls.append(b)
    solid = balls[0] if len(balls) == 1 else b200lbm.CompositeSolid(balls)
    return sim, solid, balls


def prepare(case, seed):
    built = [_build(s, case["storage"]) for s in _scenes(case, seed)]
    state = dict(case=case, sims=[b[0] for b in built], solids=[b[1] for b in built], balls=[b[2] for b in built])
    if case["api"] == "batch":
        state["batch"] = b200lbm.Batch(list(zip(state["sims"], state["solids"])))
    if case["api"] == "stream":
        state["frames"] = [state["sims"][0].frameBuffer() for _ in range(2)]
    if case["api"] == "tick" and case["frame_every"]:
        state["frames"] = [np.empty(2 * state["sims"][0].n, dtype=np.uint8)]
    return state


def _bodies(balls):
    return np.array([[b.cx, b.cy, b.cz, b.vx, b.vy, b.vz] for b in balls], dtype=np.float64)


def _fields(sim):
    return {k: getattr(sim, k) for k in FIELDS}


# ------------------------------------------------------------------ the pass
def _tick(sim, solid):
    sim.step(solid)
    solid.absorbDeadCells(sim)
    solid.step(1.0, sim.gravity)


def run(state):
    case, sim, solid = state["case"], state["sims"][0], state["solids"][0]
    api, steps, every = case["api"], case["steps"], case["frame_every"]
    out = {}
    if api == "batch":
        frames = state["batch"].run(steps, frame_every=every)
        out["phi"] = [s.phi for s in state["sims"]]
        if frames is not None:
            out["frames"] = frames
        out["bodies"] = [_bodies(b) for b in state["balls"]]
        return out
    if api == "tick":
        for t in range(steps):
            _tick(sim, solid)
        if every:
            out["frames"] = sim.packVolume(state["frames"][0])
        else:
            out.update(_fields(sim))
    elif api == "stream":
        for t in range(steps):
            if (t + 1) % every == 0:
                sim.waitFrameSlot()
                sim.stepFrame(solid, state["frames"][(t + 1) // every % 2])
            else:
                sim.step(solid)
            solid.absorbDeadCells(sim)
            solid.step(1.0, sim.gravity)
        sim.waitFrames()
        out["frames"] = state["frames"]
        out.update(_fields(sim))
    elif api == "phases":
        for t in range(steps):
            sim.retagCells(solid)
            sim.handleFreshCells(solid)
            sim.computePhiGradients()
            sim.collidePhase()
            sim.streamPhase()
            sim.collideHydro()
            sim.streamHydroAndMacro(solid)
            solid.absorbDeadCells(sim)
            solid.step(1.0, sim.gravity)
        out.update(_fields(sim))
    else:
        frames = sim.run_coupled(solid, steps, frame_every=every)
        if frames is not None:
            out["frames"] = frames
        else:
            out.update(_fields(sim))
    out["bodies"] = _bodies(state["balls"][0])
    return out


def work(case):
    nbytes = flops = 0
    for s in _scenes(case, 0):
        nx, ny, nz = s["dims"]
        inner, n = (nx - 2) * (ny - 2) * (nz - 2), nx * ny * nz
        nbytes += case["steps"] * inner * STEP_BYTES[case["storage"]]
        flops += case["steps"] * inner * STEP_FLOPS
        if case["frame_every"]:
            nbytes += case["steps"] // case["frame_every"] * n * 2
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ 64-bit values
# The same model in plain torch float64: D3Q27 BGK with Guo forcing for the
# flow, D3Q7 with interface sharpening for the phase field, halfway bounce-back,
# moving-wall links, rigid spheres with momentum exchange.
_DIRS = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
         (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1),
         (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1), (1, 1, 1), (-1, -1, -1),
         (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]
_OPP = [0] + [k + 1 if k % 2 else k - 1 for k in range(1, 27)]
_W27 = [float(np.float32((8 / 27, 2 / 27, 1 / 54, 1 / 216)[sum(map(abs, e))])) for e in _DIRS]
_W7 = [0.25] + [0.125] * 6


def _at(a, e, n):
    """a's interior shifted to the sources i - e of the interior cells."""
    return a[1 - e[2]:n[0] - 1 - e[2], 1 - e[1]:n[1] - 1 - e[1], 1 - e[0]:n[2] - 1 - e[0]]


def _along(e, x, y, z):
    """e . (x, y, z) of a lattice direction, None for the rest direction."""
    s = None
    for c, v in zip(e, (x, y, z)):
        if c:
            s = (v if c > 0 else -v) if s is None else (s + v if c > 0 else s - v)
    return s


class _Exact:
    def __init__(self, scene, dev):
        nx, ny, nz = scene["dims"]
        self.nx, self.ny, self.nz, self.n = nx, ny, nz, (nz, ny, nx)
        self.P, self.dev = dict(scene["physics"]), dev
        P, g = self.P, scene["physics"]["gravity"]
        rho = np.empty(ny)
        col = scene["column"]
        ph = P["rhoG"] + col * (P["rhoL"] - P["rhoG"])
        rho[0] = 1.0
        for y in range(1, ny):
            rho[y] = rho[y - 1] + ph[y - 1] * g * 3.0

        def full(c):
            return torch.as_tensor(c, dtype=torch.float64, device=dev)[None, :, None].expand(self.n).contiguous()

        self.phi, self.rho = full(col), full(rho)
        self.u = [torch.zeros(self.n, dtype=torch.float64, device=dev) for _ in range(3)]
        uy = -0.5 * g
        self.f, self.h = [], []
        for k, e in enumerate(_DIRS):
            eu = e[1] * uy
            self.f.append(full(_W27[k] * (rho + ph * (eu * (3 + 4.5 * eu) - 1.5 * uy * uy))))
        for k in range(7):
            self.h.append(full(_W7[k] * col))
        self.tag = torch.full(self.n, 2, dtype=torch.uint8, device=dev)
        self.tag[1:-1, 1:-1, 1:-1] = 0
        self.tag = self.retagged([])
        V = [4 / 3 * math.pi * p["r"] ** 3 for p in scene["spheres"]]
        self.balls = [dict(c=list(p["c"]), v=list(p["v"]), w=[0.0] * 3, r=p["r"], m=p["density"] * vol,
                           I=0.4 * p["density"] * vol * p["r"] ** 2, F=[0.0] * 3, T=[0.0] * 3)
                      for p, vol in zip(scene["spheres"], V)]

    def owners(self, x, y, z):
        """First sphere holding each cell (-1: none), for index tensors."""
        own = torch.full(torch.broadcast_shapes(x.shape, y.shape, z.shape), -1, dtype=torch.int64, device=self.dev)
        for b in reversed(range(len(self.balls))):
            s = self.balls[b]
            d2 = (x + 0.5 - s["c"][0]) ** 2 + (y + 0.5 - s["c"][1]) ** 2 + (z + 0.5 - s["c"][2]) ** 2
            own = torch.where(d2 <= s["r"] ** 2, torch.full_like(own, b), own)
        return own

    def box(self, s):
        lo = [max(1, int(math.floor(s["c"][a] - s["r"])) - 2) for a in range(3)]
        hi = [min(n - 1, int(math.ceil(s["c"][a] + s["r"])) + 3) for a, n in enumerate((self.nx, self.ny, self.nz))]
        return tuple(slice(lo[a], hi[a]) for a in (2, 1, 0))

    def axes(self, b):
        return [torch.arange(s.start, s.stop, device=self.dev, dtype=torch.float64) for s in b]

    def retagged(self, balls):
        t = torch.where(self.tag == 2, self.tag, torch.zeros_like(self.tag))
        for s in balls:
            b = self.box(s)
            z, y, x = self.axes(b)
            own = self.owners(x[None, None, :], y[None, :, None], z[:, None, None])
            t[b] = torch.where(own >= 0, torch.ones_like(t[b]), t[b])
        return t

    def impulse(self, own, x, y, z, p):
        """Momentum p (three tensors) given to the owners at cells (x, y, z)."""
        for b, s in enumerate(self.balls):
            m = own == b
            if not bool(m.any()):
                continue
            r = [c[m] + 0.5 - s["c"][a] for a, c in enumerate((x, y, z))]
            q = [c[m] for c in p]
            for a in range(3):
                i, j = (a + 1) % 3, (a + 2) % 3
                s["F"][a] += float(q[a].sum())
                s["T"][a] += float((r[i] * q[j] - r[j] * q[i]).sum())

    def fill_fresh(self, fresh):
        """Cells uncovered by a sphere take the mean of their fluid neighbours, in scan order."""
        P = self.P
        for z, y, x in fresh.nonzero().tolist():
            b = (slice(z - 1, z + 2), slice(y - 1, y + 2), slice(x - 1, x + 2))
            fluid = self.tag[b] == 0
            fluid[1, 1, 1] = False
            if bool(fluid.any()):
                p, r = float(self.phi[b][fluid].mean()), float(self.rho[b][fluid].mean())
                v = [float(c[b][fluid].mean()) for c in self.u]
            else:
                p, r, v = float(self.phi[z, y, x]), 1.0, [0.0] * 3
            self.phi[z, y, x], self.rho[z, y, x] = p, r
            for c, val in zip(self.u, v):
                c[z, y, x] = val
            u2 = sum(c * c for c in v)
            for k, e in enumerate(_DIRS):
                eu = sum(a * c for a, c in zip(e, v))
                self.f[k][z, y, x] = _W27[k] * (
                    r + (P["rhoG"] + p * (P["rhoL"] - P["rhoG"])) * (eu * (3 + 4.5 * eu) - 1.5 * u2))
                if k < 7:
                    self.h[k][z, y, x] = _W7[k] * p * (1 + 4 * eu)

    def chemical(self, p, lap):
        P = self.P
        return 48 * P["sigma"] / P["W"] * p * (p - 1) * (2 * p - 1) - 1.5 * P["sigma"] * P["W"] * lap

    def step(self):
        P, n, g = self.P, self.n, self.P["gravity"]
        inner = (slice(1, -1),) * 3
        before = self.tag
        self.tag = self.retagged(self.balls)
        self.fill_fresh((self.tag == 0) & (before == 1))
        fluid = self.tag == 0
        here = fluid[inner]
        p = self.phi[inner]
        s = [(_at(self.phi, tuple(-v for v in e), n)) for e in _DIRS[1:7]]
        grad = [0.5 * (s[2 * a] - s[2 * a + 1]) for a in range(3)]
        lap = sum(s) - 6 * p
        del s
        iw, iwp, dRho = 1 / P["tau"], 1 / P["tauPhi"], P["rhoL"] - P["rhoG"]
        u = [c[inner] for c in self.u]
        ph = P["rhoG"] + p * dRho
        # phase field: collide, then pull
        sharp = 4 * (0.25 * (P["tauPhi"] - 0.5)) * (1 - 0.5 * iwp) / P["W"] * 4 * p * (1 - p)
        sharp = sharp / (torch.sqrt(grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2) + 1e-12)
        S = [4 * iwp * p * c + sharp * d for c, d in zip(u, grad)]
        del sharp
        h2 = [t.clone() for t in self.h]
        for k in range(7):
            along = _along(_DIRS[k], *S)
            eq = iwp * p if along is None else iwp * p + along
            h2[k][inner] = torch.where(here, (1 - iwp) * self.h[k][inner] + _W7[k] * eq, h2[k][inner])
        del S
        for k in range(7):
            got = torch.where(_at(fluid, _DIRS[k], n), _at(h2[k], _DIRS[k], n), h2[_OPP[k]][inner])
            self.h[k][inner] = torch.where(here, got, self.h[k][inner])
        del h2
        # flow: collide
        mu = self.chemical(p, lap)
        F = [mu * grad[0], mu * grad[1] + ph * g, mu * grad[2]]
        u2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        uF = u[0] * F[0] + u[1] * F[1] + u[2] * F[2]
        A, rho = 3 * (1 - 0.5 * iw), self.rho[inner]
        f2 = []
        for k, e in enumerate(_DIRS):
            eu, eF = _along(e, *u), _along(e, *F)
            if eu is None:
                q = iw * (rho - 1.5 * ph * u2) - A * uF
            else:
                q = iw * (rho + ph * (eu * (3 + 4.5 * eu) - 1.5 * u2)) + A * (eF * (1 + 3 * eu) - uF)
            t = self.f[k].clone()
            t[inner] = torch.where(here, (1 - iw) * self.f[k][inner] + _W27[k] * q, t[inner])
            f2.append(t)
        del mu, F, u2, uF, rho
        # pull, bounce-back, moving walls and their momentum exchange
        total, mom = torch.zeros_like(p), [torch.zeros_like(p) for _ in range(3)]
        for k, e in enumerate(_DIRS):
            opp = f2[_OPP[k]][inner]
            got = torch.where(_at(fluid, e, n), _at(f2[k], e, n), opp)
            for s in self.balls if k else ():
                b = self.box(s)
                link = (fluid[b] & (self.tag[tuple(slice(r.start - d, r.stop - d) for r, d in zip(b, e[::-1]))] == 1))
                if not bool(link.any()):
                    continue
                z, y, x = (c + r.start for c, r in zip(link.nonzero(as_tuple=True), b))
                sx, sy, sz = x - e[0], y - e[1], z - e[2]
                own = self.owners(sx.double(), sy.double(), sz.double())
                mine = own == self.balls.index(s)
                z, y, x, sx, sy, sz, own = (c[mine] for c in (z, y, x, sx, sy, sz, own))
                r = [c.double() + 0.5 - o for c, o in zip((sx, sy, sz), s["c"])]
                wall = [s["v"][a] + (s["w"][(a + 1) % 3] * r[(a + 2) % 3] - s["w"][(a + 2) % 3] * r[(a + 1) % 3])
                        for a in range(3)]
                back = f2[_OPP[k]][z, y, x]
                old = P["rhoG"] + self.phi[z, y, x] * dRho
                val = back + 6 * _W27[k] * old * sum(c * v for c, v in zip(e, wall) if c)
                got[z - 1, y - 1, x - 1] = val
                self.impulse(own, sx.double(), sy.double(), sz.double(), [-(back + val) * c for c in e])
            self.f[k][inner] = torch.where(here, got, self.f[k][inner])
            total += got
            for a in range(3):
                if e[a]:
                    mom[a] += e[a] * got
        del f2
        self.rho[inner] = torch.where(here, total.clamp(min=0.01), self.rho[inner])
        pn = sum(t[inner] for t in self.h).clamp(0, 1)
        phn, mu = P["rhoG"] + pn * dRho, self.chemical(pn, lap)
        F = [mu * grad[0], mu * grad[1] + phn * g, mu * grad[2]]
        new = [(m + 0.5 * c) / phn for m, c in zip(mom, F)]
        size = torch.sqrt(new[0] ** 2 + new[1] ** 2 + new[2] ** 2)
        cap = torch.where(size > 0.2, 0.2 / size, torch.ones_like(size))
        for c, v in zip(self.u, new):
            c[inner] = torch.where(here, v * cap, c[inner])
        self.phi[inner] = torch.where(here, pn, p)
        # cells a sphere has just covered give it their momentum
        dead = (self.tag == 1) & (before == 0)
        if bool(dead.any()):
            z, y, x = dead.nonzero(as_tuple=True)
            own = self.owners(x.double(), y.double(), z.double())
            ph = P["rhoG"] + self.phi[z, y, x] * dRho
            self.impulse(own, x.double(), y.double(), z.double(), [ph * c[z, y, x] for c in self.u])
        for s in self.balls:
            self.move(s)

    def move(self, s):
        """The rigid sphere's capped, damped and clamped explicit step."""
        g = self.P["gravity"]
        s["F"][1] += s["m"] * g
        acc = [c / s["m"] for c in s["F"]]
        a, cap = math.sqrt(sum(c * c for c in acc)), 3.5 * abs(g or 0.001)
        scale = cap / a if a > cap else 1.0
        s["v"] = [v + c * scale for v, c in zip(s["v"], acc)]
        s["w"] = [w + t / s["I"] for w, t in zip(s["w"], s["T"])]
        speed = math.sqrt(sum(v * v for v in s["v"]))
        if speed > 0.08:
            s["v"] = [v * 0.08 / speed for v in s["v"]]
        s["v"] = [0.0 if abs(0.98 * v) < 1e-4 else 0.98 * v for v in s["v"]]
        s["w"] = [0.0 if abs(0.95 * w) < 1e-4 else 0.95 * w for w in s["w"]]
        m = s["r"] + 1.5
        for a, n in enumerate((self.nx, self.ny, self.nz)):
            s["c"][a] += s["v"][a]
            if s["c"][a] < m:
                s["c"][a], s["v"][a] = m, max(0.0, s["v"][a])
            if s["c"][a] > n - 1 - m:
                s["c"][a], s["v"][a] = n - 1 - m, min(0.0, s["v"][a])
        s["F"], s["T"] = [0.0] * 3, [0.0] * 3


def exact(case, seed):
    scenes = _scenes(case, seed)
    cells = sum(int(np.prod(s["dims"])) for s in scenes)
    on_gpu = torch.cuda.is_available()
    if cells * case["steps"] > (1.5e9 if on_gpu else 2e7):
        return None
    dev = "cuda" if on_gpu else "cpu"
    # of a batch, as many scenes as fit in a few seconds
    count = max(1, min(len(scenes), 160 // case["steps"]))
    done = []
    for s in scenes[:count]:
        e = _Exact(s, dev)
        for _ in range(case["steps"]):
            e.step()
        e.f = e.h = None
        done.append(e)
    bodies = [np.array([b["c"] + b["v"] for b in e.balls], dtype=np.float64) for e in done]
    out = {}
    if case["api"] == "batch":
        rest = [None] * (len(scenes) - count)
        out["bodies"] = bodies + rest
        out["phi"] = [e.phi.reshape(-1) for e in done] + rest
        if case["frame_every"]:
            out["frames"] = [None] * len(scenes)
        return out
    e = done[0]
    out["bodies"] = bodies[0]
    if case["frame_every"]:
        out["frames"] = [None] * 2 if case["api"] == "stream" else None
    if not case["frame_every"] or case["api"] == "stream":
        for k, v in zip(FIELDS, (e.phi, e.rho, *e.u)):
            out[k] = v.reshape(-1)
    return out
