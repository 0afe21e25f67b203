"""Written tags on the domain's faces: handleFreshCells and absorbDeadCells run
over the interior (1 .. n-2), like the reference's loops, also when the last
step's retag covered the whole grid."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

DIMS = (13, 11, 12)
FIELDS = ("phi", "rho", "ux", "uy", "uz", "f", "h")


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _faces():
    z, y, x = np.indices(DIMS[::-1])
    return np.logical_or.reduce([x == 0, x == DIMS[0] - 1, y == 0, y == DIMS[1] - 1, z == 0, z == DIMS[2] - 1])


@pytest.mark.parametrize("storage", ["f32", "f64"])
def test_fresh_cells_are_inside(gpu, storage):
    sim = gpu.Sim(*DIMS, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(5)
    sim.tag[:] = np.array(sim.tag)  # the next step retags the whole grid
    sim.step(gpu.RigidSphere(*DIMS, cx=6.2, cy=5.1, cz=6.3, r=2.2, density=2.0))
    face = _faces()
    tag, prev = np.zeros(face.shape, np.uint8), np.zeros(face.shape, np.uint8)
    prev[face] = 1
    prev[4:7, 4:7, 4:8] = 1
    prev[1, 1, 1] = 1
    was = {k: sim.field64(k).reshape(sim.n, -1) for k in FIELDS}
    sim.tag[:] = tag.ravel()
    sim.tagPrev[:] = prev.ravel()
    sim.handleFreshCells()
    fresh, dead = sim.last_sets()
    inside = ((prev == 1) & ~face).ravel()
    assert np.array_equal(fresh, np.nonzero(inside)[0]) and len(dead) == 0
    for k in FIELDS:
        assert np.array_equal(sim.field64(k).reshape(sim.n, -1)[~inside], was[k][~inside]), k
    sim.close()


@pytest.mark.parametrize("storage", ["f32", "f64"])
def test_dead_cells_are_inside(gpu, storage):
    sim = gpu.Sim(*DIMS, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(5)
    sol = gpu.RigidSphere(*DIMS, cx=1.6, cy=5.1, cz=6.3, r=2.6, density=2.0)  # it contains cells of the face x = 0
    sim.tag[:] = np.array(sim.tag)
    sim.step(sol)
    rs = np.random.RandomState(3)
    for k in ("ux", "uy", "uz"):
        getattr(sim, k)[:] = rs.uniform(-0.05, 0.05, sim.n).astype(np.float32)
    sim.tag[:] = np.ones(sim.n, np.uint8)
    sim.tagPrev[:] = np.zeros(sim.n, np.uint8)
    for k in ("Fx", "Fy", "Fz"):
        setattr(sol, k, 0.0)
    sol.absorbDeadCells(sim)
    z, y, x = np.indices(DIMS[::-1])
    own = (x + 0.5 - sol.cx) ** 2 + (y + 0.5 - sol.cy) ** 2 + (z + 0.5 - sol.cz) ** 2 <= sol.r ** 2
    assert (own & _faces()).sum() > 8
    at = (own & ~_faces()).ravel()
    rho = sim.rhoG + sim.field64("phi")[at] * (sim.rhoL - sim.rhoG)
    for k, u in (("Fx", "ux"), ("Fy", "uy"), ("Fz", "uz")):
        want = (rho * sim.field64(u)[at]).sum()
        assert abs(getattr(sol, k) - want) <= 1e-13 * at.sum(), k
    sim.close()
