"""The two launches around the fused step: the retag, the fresh / dead lists
and the fresh fill (k_sets, 2,048-cell chunks of the retag box), and the shells
(k_shell, 1,024-cell chunks of each sphere's box: moving-wall links, momentum
exchange, dead-cell impulses).  In the FP64 storage form, against the FP64
oracle for one sphere and against the phase-by-phase kernels for two touching
spheres.

Bars.  The lists are integers: exact.  The fields differ by the association of
the collision algebra only: 1e-10 relative, as for the FP64 form elsewhere.  A
force is a sum of at most ~60 r^2 link terms below 0.3, each within that bar:
1e-10 * 20 r^2; a torque has the arm r on top."""
import functools

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

BAR = 1e-10
FIELDS = ("phi", "rho", "ux", "uy", "uz", "f", "h")
IMPULSE = ("Fx", "Fy", "Fz", "Tx", "Ty", "Tz")


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _tank(SimC, dims):
    sim = SimC(*dims)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(dims[1] * 0.45)
    return sim


# boxes of one chunk, a little over one, many; a sphere against a wall
@pytest.mark.parametrize("r,c,v", [
    (1.2, (9.3, 12.6, 8.1), (0.07, -0.05, 0.04)),
    (2.9, (16.5, 15.2, 14.8), (0.06, 0.05, -0.06)),
    (4.4, (6.0, 14.1, 19.7), (-0.08, 0.03, 0.05)),
    (9.3, (20.2, 14.4, 19.1), (0.05, -0.06, 0.07)),
])
def test_one_sphere_against_the_oracle(gpu, oracle_mod, r, c, v):
    dims = (40, 29, 38)
    o = _tank(functools.partial(oracle_mod.OracleSim, store="f64"), dims)
    g = _tank(functools.partial(gpu.Sim, storage="f64"), dims)
    so, sg = (S(*dims, cx=c[0], cy=c[1], cz=c[2], r=r, density=1.7)
              for S in (oracle_mod.OracleSphere, gpu.RigidSphere))
    seen = 0
    for t in range(8):
        for s in (so, sg):  # the same motion on both sides, faster than the integrator allows
            s.cx, s.cy, s.cz = (a + 4 * t * b for a, b in zip(c, v))
            s.vx, s.vy, s.vz = v
            s.wx, s.wy, s.wz = 0.01, -0.02, 0.015
            for k in IMPULSE:
                setattr(s, k, 0.0)
        o.step(so)
        g.step(sg)
        tag, prev = np.asarray(o.tag), np.asarray(o.tagPrev)
        fresh, dead = g.last_sets()
        assert np.array_equal(np.asarray(g.tag), tag), t
        assert np.array_equal(fresh, np.nonzero((tag == 0) & (prev == 1))[0]), t
        assert np.array_equal(dead, np.nonzero((tag == 1) & (prev == 0))[0]), t
        seen += len(fresh) + len(dead)
        so.absorbDeadCells(o)
        sg.absorbDeadCells(g)
        for j, k in enumerate(IMPULSE):
            bar = BAR * 20 * r * r * (1 if j < 3 else r + 1)
            assert abs(getattr(sg, k) - getattr(so, k)) <= bar, (t, k, getattr(sg, k), getattr(so, k))
    assert seen > 20
    for k in FIELDS:
        ref = np.asarray(getattr(o, k), np.float64)
        assert np.abs(g.field64(k) - ref).max() <= BAR * np.abs(ref).max(), k
    g.close()


def test_touching_spheres_against_the_phases(gpu):
    """Cells with links to both spheres of a composite solid."""
    dims = (38, 30, 33)
    r = (5.2, 4.1)
    sims = [_tank(functools.partial(gpu.Sim, storage="f64"), dims) for _ in range(2)]
    solids = []
    for _ in sims:
        a = gpu.RigidSphere(*dims, cx=14.2, cy=14.5, cz=16.3, r=r[0], density=2.0)
        b = gpu.RigidSphere(*dims, cx=23.4, cy=15.1, cz=15.9, r=r[1], density=1.4)
        solids.append(gpu.CompositeSolid([a, b]))
    fused, phased = sims
    for t in range(6):
        for solid in solids:
            for q, s in enumerate(solid.spheres):
                s.cy += 0.11 if q else -0.13
                s.vx, s.vy, s.vz = 0.02, 0.11 if q else -0.13, -0.03
                for k in IMPULSE:
                    setattr(s, k, 0.0)
        fused.step(solids[0])
        phased.retagCells(solids[1])
        phased.handleFreshCells(solids[1])
        phased.computePhiGradients()
        phased.collidePhase()
        phased.streamPhase()
        phased.collideHydro()
        phased.streamHydroAndMacro(solids[1])
        for q in range(2):
            for j, k in enumerate(IMPULSE):
                bar = BAR * 20 * r[q] ** 2 * (1 if j < 3 else r[q] + 1)
                a, b = (getattr(s.spheres[q], k) for s in solids)
                assert abs(a - b) <= bar, (t, q, k, a, b)
    for k in FIELDS:
        ref = phased.field64(k)
        assert np.abs(fused.field64(k) - ref).max() <= BAR * np.abs(ref).max(), k
    for sim in sims:
        sim.close()
