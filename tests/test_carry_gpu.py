"""SOLID cells keep their values in both population halves: copied once when
they turn SOLID (k_sets), or over the whole grid after calls that work on one
half alone (k_carry_solid).  Nothing is computed for a SOLID cell, so the bits
stay the same through even and odd numbers of fused steps, after writes to the
other half (f2, h2), and after phase-by-phase steps."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("f", "h", "phi", "rho", "ux", "uy", "uz")


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _solid_values(sim):
    solid = np.asarray(sim.tag) == 1
    n = solid.size
    return {k: np.array(getattr(sim, k)).reshape(n, -1)[solid] for k in FIELDS}


@pytest.mark.parametrize("r,storage", [(1.3, "f32"), (6.4, "f32"), (6.4, "f16"), (5.1, "bf16"), (5.1, "f64")])
@pytest.mark.parametrize("between", ["nothing", "f2", "phases"])
def test_solid_cells_keep_their_values(gpu, r, storage, between):
    if between == "phases" and storage not in ("f32", "f64"):
        pytest.skip("the phases need FP32 or FP64 storage")
    dims = (34, 27, 30)
    sim = gpu.Sim(*dims, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(12)
    sol = gpu.RigidSphere(*dims, cx=16.3, cy=13.1, cz=14.6, r=r, density=2.0)
    for t in range(3):  # the sphere arrives: cells turn SOLID at several steps
        sol.cx += 0.4
        sim.step(sol)
    want = _solid_values(sim)
    assert len(want["phi"]) > 5
    if between == "f2":
        sim.f2[:] = np.float32(0.25)
        sim.h2[:] = np.float32(0.125)
    elif between == "phases":
        for _ in range(2):
            sim.retagCells(sol)
            sim.handleFreshCells(sol)
            sim.computePhiGradients()
            sim.collidePhase()
            sim.streamPhase()
            sim.collideHydro()
            sim.streamHydroAndMacro(sol)
    for t in range(3):  # the sphere rests: its cells keep what they had, in either half
        sim.step(sol)
        got = _solid_values(sim)
        for k in FIELDS:
            assert np.array_equal(got[k], want[k]), (t, k)
    sim.close()
