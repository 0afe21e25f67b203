"""Tags written between step_begin and step_end.  The fused step then meets
SOLID cells that no sphere contains (walls at rest), SOLID cells on the domain's
faces and FLUID cells deep inside a sphere; it gives what the phase-by-phase
kernels give from the same state in FP64.

Tolerances.  FP64: the association of the collision differs, 1e-10 of the
largest value.  FP32 arithmetic (FP16 storage rounds the populations only, after
the macros): a population is about ten operations on values of at most 1.6, rho
and phi sums of 27 and 7 of them, 64 units in the last place of 2; u divides
such a sum by a density of at least 0.1, ten times that.  A force is a sum of
links, each within that bar: at most 18 on each cell of the shell, 120 more on
the written cells."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

DIMS = (35, 22, 27)
STATE = ("f", "h", "phi", "rho", "ux", "uy", "uz")
IMPULSE = ("Fx", "Fy", "Fz", "Tx", "Ty", "Tz")


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _random_state(n, seed):
    rs = np.random.RandomState(seed)
    w27 = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8)
    w7 = np.array([0.25] + [0.125] * 6)
    st = {"phi": rs.uniform(0, 1, n), "rho": rs.uniform(0.9, 1.1, n)}
    st["f"] = (w27 * rs.uniform(0.9, 1.1, (n, 27))).ravel()
    st["h"] = (w7 * st["phi"][:, None] * rs.uniform(0.9, 1.1, (n, 7))).ravel()
    for k in ("ux", "uy", "uz"):
        st[k] = rs.uniform(-0.05, 0.05, n)
    return {k: v.astype(np.float32) for k, v in st.items()}


def _sphere(gpu, where):
    c = {"free": (17.3, 11.1, 13.6), "none": None, "wall": (2.1, 11.1, 13.6)}[where]
    if c is None:
        return None
    sol = gpu.RigidSphere(*DIMS, cx=c[0], cy=c[1], cz=c[2], r=4.3, density=2.0)
    if where == "free":
        sol.vx, sol.vy, sol.vz, sol.wy = 0.03, -0.02, 0.015, 0.004
    return sol


def _write(tag, where):
    """tag (z, y, x): SOLID cells of no sphere near and far from one, FLUID cells
    inside it; where the sphere meets a face, that face SOLID."""
    if where == "wall":
        tag[8:20, 5:18, 0] = 1
        return
    if where == "free":
        tag[13, 10:13, 16:19] = 0           # a pocket around the centre
        tag[14, 11, 11] = tag[13, 12, 10] = 1  # one and two cells off the surface
    for z, y, x in ((3, 4, 5), (3, 4, 6), (3, 5, 5), (22, 17, 30), (24, 20, 32), (1, 1, 1)):
        tag[z, y, x] = 1


@pytest.mark.parametrize("where", ["free", "none", "wall"])
@pytest.mark.parametrize("storage,rows", [("f32", 0), ("f32", 2), ("f16", 0), ("f64", 0)])
def test_step_end_after_a_tag_write(gpu, where, storage, rows):
    sim, twin = gpu.Sim(*DIMS, storage=storage), gpu.Sim(*DIMS, storage="f64")
    for s in (sim, twin):
        scenes._params(s, 0.8, 0.7, 0.008, 0.0015)
        s.initFlat(10)
    if rows:
        sim.set_fused_config(rows, 5)
    a, b = _sphere(gpu, where), _sphere(gpu, where)
    for _ in range(3):
        sim.step(a)
    for k, v in _random_state(sim.n, 4).items():
        getattr(sim, k)[:] = v
    sim.step_begin(a)
    tag = np.array(sim.tag).reshape(DIMS[::-1])
    _write(tag, where)
    sim.tag[:] = tag.ravel()
    twin.retagCells(b)
    for k in STATE:
        getattr(twin, k)[:] = np.array(getattr(sim, k))
    twin.tag[:] = tag.ravel()
    twin.computePhiGradients()
    twin.collidePhase()
    twin.streamPhase()
    twin.collideHydro()
    twin.streamHydroAndMacro(b)
    if a is not None:
        for k in IMPULSE:
            setattr(a, k, 0.0)
    sim.step_end(a)
    fluid = tag.ravel() == 0
    for k in ("phi", "rho", "ux", "uy", "uz"):
        ref = twin.field64(k)
        got = sim.field64(k) if storage == "f64" else np.asarray(getattr(sim, k), np.float64)
        tol = 1e-10 if storage == "f64" else 128 * 2.0 ** -24 * (10 if k[0] == "u" else 1)
        err = np.abs(got - ref)[fluid].max()
        assert err <= tol, (k, err)
    if a is not None:
        per = (1e-10 if storage == "f64" else 64 * 2.0 ** -24) * (18 * 4 * 3.2 * (a.r + 1) ** 2 + 120)
        for j, k in enumerate(IMPULSE):
            assert abs(getattr(a, k) - getattr(b, k)) <= per * (1 if j < 3 else a.r + 1), k
    for k in STATE[:2] if storage in ("f32", "f64") else ():
        ref = twin.field64(k)
        got = sim.field64(k) if storage == "f64" else np.asarray(getattr(sim, k), np.float64)
        tol = 1e-10 if storage == "f64" else 128 * 2.0 ** -24
        assert np.abs(got - ref).max() <= tol, k
    sim.close()
    twin.close()


@pytest.mark.parametrize("storage", ["f32", "f64"])
def test_absorb_after_a_tag_write(gpu, storage):
    """Dead cells are those of the tags as they stand (src/solid.js:87-101)."""
    sim = gpu.Sim(*DIMS, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(10)
    sol = _sphere(gpu, "free")
    for _ in range(4):
        scenes.substep(sim, sol)
    for k in ("ux", "uy", "uz"):
        getattr(sim, k)[:] = _random_state(sim.n, 5)[k]
    sol.cx += 0.7
    sim.step_begin(sol)
    tag, prev = np.array(sim.tag), np.array(sim.tagPrev)
    dead = np.nonzero((tag == 1) & (prev == 0))[0]
    assert len(dead) > 12
    tag[dead[::2]] = 0
    sim.tag[:] = tag
    sim.step_end(sol)
    for k in IMPULSE:
        setattr(sol, k, 0.0)
    sol.absorbDeadCells(sim)
    left = dead[1::2]
    rho = sim.rhoG + sim.field64("phi")[left] * (sim.rhoL - sim.rhoG)
    for k, u in (("Fx", "ux"), ("Fy", "uy"), ("Fz", "uz")):
        want = (rho * sim.field64(u)[left]).sum()
        assert abs(getattr(sol, k) - want) <= 1e-13 * len(left), (k, getattr(sol, k), want)
    sim.close()
