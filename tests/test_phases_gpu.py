"""The seven phases of a step, called one by one, against the oracle: one step
from a random state, so that every population group, wall, corner and link of
the grid counts.  Edges below, at and above a block of 8 cells and a warp; a
sphere inside, and one that reaches the walls.

Tolerances.  FP64: the same double arithmetic but for the order of a few sums,
1e-12 of the largest value.  FP32: a population is about ten operations on
values of at most 1.6 and rho and phi are sums of 27 and 7 of them, 64 units in
the last place of the largest value (7.7e-6 absolute at 2); u divides such a
sum by a density of at least 0.1, ten times that."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

TOL = {"f32": 64 * 2.0 ** -24, "f64": 1e-12}


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _random_state(dims, seed):
    rs = np.random.RandomState(seed)
    n = dims[0] * dims[1] * dims[2]
    w27 = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8)
    w7 = np.array([0.25] + [0.125] * 6)
    st = {
        "f": (w27 * rs.uniform(0.9, 1.1, (n, 27))).ravel(),
        "h": (w7 * rs.uniform(0.0, 1.1, (n, 7))).ravel(),
        "phi": rs.uniform(0, 1, n),
        "rho": rs.uniform(0.9, 1.1, n),
    }
    for k in ("ux", "uy", "uz"):
        st[k] = rs.uniform(-0.05, 0.05, n)
    return {k: v.astype(np.float32) for k, v in st.items()}


@pytest.mark.parametrize("dims,r", [
    ((3, 3, 3), 0.0), ((4, 5, 3), 0.0), ((10, 11, 12), 2.2), ((8, 8, 8), 5.0), ((16, 9, 7), 2.0),
    ((33, 6, 5), 1.2), ((41, 18, 21), 6.3), ((64, 17, 9), 3.4),
])
@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("force", [False, True])
def test_one_step_from_a_random_state(gpu, oracle_mod, dims, r, storage, force):
    st = _random_state(dims, sum(dims))
    o = oracle_mod.OracleSim(*dims, store=storage)
    g = gpu.Sim(*dims, storage=storage)
    c = [0.5 * d + 0.13 * a for a, d in enumerate(dims)]
    got = {}
    for sim, Sphere in ((o, oracle_mod.OracleSphere), (g, gpu.RigidSphere)):
        scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
        sim.initFlat(dims[1] * 0.4)
        sol = Sphere(*dims, cx=c[0], cy=c[1], cz=c[2], r=r or 0.1, density=2.0)
        sol.vx, sol.vy, sol.vz, sol.wz = 0.01, -0.02, 0.015, 0.003
        sim.retagCells(sol)  # (SOLID before the step too: no fresh or dead cells)
        for k, v in st.items():
            getattr(sim, k)[:] = v
        if force:
            for a, k in enumerate(("bodyFx", "bodyFy", "bodyFz")):
                getattr(sim, k)[:] = np.float32(1e-4 * (a + 1))
        sim.retagCells(sol)
        sim.handleFreshCells(sol)
        sim.computePhiGradients()
        sim.collidePhase()
        sim.streamPhase()
        sim.collideHydro()
        sim.streamHydroAndMacro(sol)
        got[sim] = [sol.Fx, sol.Fy, sol.Fz]
    assert np.array_equal(np.asarray(g.tag), np.asarray(o.tag))
    for k in ("gx", "gy", "gz", "lap", "f", "h", "phi", "rho", "ux", "uy", "uz"):
        ref = np.asarray(getattr(o, k), np.float64)
        val = g.field64(k) if storage == "f64" else np.asarray(getattr(g, k), np.float64)
        tol = TOL[storage] * (10 if k[0] == "u" else 1) * 2
        err = np.abs(val.ravel() - ref.ravel()).max()
        assert err <= tol, (k, err)
    links = 18 * 4 * 3.2 * (r + 1) ** 2  # at most 18 links on each cell of the shell
    assert np.abs(np.subtract(got[g], got[o])).max() <= TOL[storage] * links
    g.close()
