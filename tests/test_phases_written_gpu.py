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
