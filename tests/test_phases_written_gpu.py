"""The phases called one by one on tags and values that the caller wrote,
against the oracle."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _phases(sim, sol, write):
    sim.retagCells(sol)
    sim.handleFreshCells(sol)
    write(sim)
    sim.computePhiGradients()
    sim.collidePhase()
    sim.streamPhase()
    sim.collideHydro()
    sim.streamHydroAndMacro(sol)


@pytest.mark.parametrize("r", [4.3, 7.2])
def test_links_inside_the_sphere_count(gpu, oracle_mod, r):
    """FLUID cells written at the sphere's centre have links to the cells around
    them, which the sphere contains: their momentum exchange is the sphere's.
    About 26 links a cell, each within 1e-12 (FP64)."""
    dims = (31, 22, 27)

    def pocket(sim):
        tag = np.array(sim.tag).reshape(dims[::-1])
        tag[13, 10:13, 14:18] = 0
        sim.tag[:] = tag.ravel()

    got = []
    for SimC, SphC, kw in ((oracle_mod.OracleSim, oracle_mod.OracleSphere, {"store": "f64"}),
                           (gpu.Sim, gpu.RigidSphere, {"storage": "f64"})):
        sim = SimC(*dims, **kw)
        scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
        sim.initFlat(10)
        rs = np.random.RandomState(7)
        for k in ("ux", "uy", "uz"):
            getattr(sim, k)[:] = rs.uniform(-0.05, 0.05, sim.n).astype(np.float32)
        sol = SphC(*dims, cx=15.3, cy=11.1, cz=13.6, r=r, density=2.0)
        sol.vx, sol.vy, sol.wz = 0.03, -0.02, 0.004
        _phases(sim, sol, pocket)
        got.append([sol.Fx, sol.Fy, sol.Fz, sol.Tx, sol.Ty, sol.Tz])
    links = 12 * 26 + 18 * 4 * 3.2 * (r + 1) ** 2
    err = np.abs(np.subtract(*got))
    assert err[:3].max() <= 1e-12 * links and err[3:].max() <= 1e-12 * links * (r + 1), err


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("field,k", [("f", 0), ("f", 1), ("f", 20), ("h", 0), ("h", 3), ("phi", 0), ("rho", 0),
                                     ("ux", 0), ("uy", 0), ("uz", 0)])
def test_a_non_finite_value_spreads_as_in_the_reference(gpu, oracle_mod, storage, value, field, k):
    """0 times a non-finite value is NaN: it reaches every direction, not only
    those that have the component.  One step from one such cell away from the
    sphere and one beside it: the same cells are finite."""
    dims = (26, 17, 19)
    sims = []
    for SimC, SphC, kw in ((oracle_mod.OracleSim, oracle_mod.OracleSphere, {"store": storage}),
                           (gpu.Sim, gpu.RigidSphere, {"storage": storage})):
        sim = SimC(*dims, **kw)
        scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
        sim.initFlat(8)
        sol = SphC(*dims, cx=17.3, cy=9.1, cz=9.6, r=3.2, density=2.0)
        sol.vx, sol.wy = 0.02, 0.003
        sim.retagCells(sol)

        def put(s):
            per = {"f": 27, "h": 7}.get(field, 1)
            a = np.array(getattr(s, field))
            for at in ((6, 8, 9), (13, 9, 9)):
                a[s.idx(*at) * per + k] = value
            getattr(s, field)[:] = a

        _phases(sim, sol, put)
        sims.append(sim)
    o, g = sims
    for f in ("f", "h", "phi", "rho", "ux", "uy", "uz"):
        a, b = (np.isfinite(np.asarray(getattr(s, f))) for s in (o, g))
        assert np.array_equal(a, b), (f, int((~a).sum()), int((~b).sum()))
    assert not all(np.isfinite(np.asarray(getattr(g, f))).all() for f in ("f", "h", "phi", "ux"))
    g.close()
