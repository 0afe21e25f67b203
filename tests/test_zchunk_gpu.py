"""The default z-chunk lengths (short chunks on grids whose tiles would leave
SMs idle, evened-out chunks per scene of a batch) against explicit ones: every
field bit for bit, on grids whose chunk is one plane, a few, and uneven."""
import functools

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


def _scene(SimC, SphC, dims):
    sim = SimC(*dims)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(dims[1] * 0.4)
    sol = SphC(*dims, cx=dims[0] * 0.5, cy=dims[1] * 0.5, cz=dims[2] * 0.5, r=0.15 * min(dims), density=2.0)
    sol.vx, sol.vy = 0.04, -0.03
    return sim, sol


def _state(sim):
    return {k: np.array(getattr(sim, k)) for k in ("phi", "rho", "ux", "uy", "uz", "f", "h", "tag")}


DIMS = ((12, 13, 3), (11, 12, 14), (40, 28, 41), (64, 37, 70), (96, 70, 50))


@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
def test_default_chunks_give_the_same_bits(gpu, storage):
    SimS = functools.partial(gpu.Sim, storage=storage)
    want = []
    for dims in DIMS:
        sim, sol = _scene(SimS, gpu.RigidSphere, dims)
        rows, z = sim.fused_config()
        assert 1 <= z <= max(1, dims[2] - 2)
        sim.set_fused_config(4, 7)  # the plain form, chunks of 7 planes
        sim.run_coupled(sol, 6)
        want.append((_state(sim), sol.state()))
        sim.close()
    made = [_scene(SimS, gpu.RigidSphere, dims) for dims in DIMS]
    for (sim, sol), (w, s) in zip(made, want):
        sim.run_coupled(sol, 6)
        assert all(np.array_equal(a, w[k]) for k, a in _state(sim).items()), (sim.nx, sim.nz)
        assert sol.state() == s
        sim.close()
    made = [_scene(SimS, gpu.RigidSphere, dims) for dims in DIMS]
    with gpu.Batch(made) as batch:
        batch.run(6)
    for (sim, sol), (w, s) in zip(made, want):
        assert all(np.array_equal(a, w[k]) for k, a in _state(sim).items()), (sim.nx, sim.nz)
        assert sol.state() == s
        sim.close()
