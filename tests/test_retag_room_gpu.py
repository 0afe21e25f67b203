"""A device-resident run whose sphere was moved too far for its retag box
reports LBM_ERR_CAPACITY.  The steps that could not retag leave the SOLID cells
where they were, as walls at rest, with every field finished; the next step
retags the whole grid.  Against the phase-by-phase kernels on the same tags, in
FP64: the collision differs by its association only, 1e-10 of the largest value."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

DIMS = (64, 50, 56)
STATE = ("f", "h", "phi", "rho", "ux", "uy", "uz")


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _moved(gpu, storage="f64"):
    """A few steps with the sphere in one corner, then the sphere in another."""
    sim = gpu.Sim(*DIMS, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(25)
    sol = gpu.RigidSphere(*DIMS, cx=10.2, cy=9.8, cz=11.1, r=5.3, density=2.0)
    rs = np.random.RandomState(2)
    for k in ("ux", "uy", "uz"):
        getattr(sim, k)[:] = rs.uniform(-0.05, 0.05, sim.n).astype(np.float32)
    for _ in range(4):
        sim.step(sol)
    # float32 values, which another handle can be given exactly
    for k in STATE:
        getattr(sim, k)[:] = np.array(getattr(sim, k))
    sol.cx, sol.cy, sol.cz = 52.3, 39.8, 44.1
    return sim, sol


def _run(gpu, sim, sol, steps):
    from b200lbm import _capi
    from b200lbm.solid import to_c_array
    sim._sync()
    arr = to_c_array([sol])
    rc = _capi.lib().lbm_run_coupled(sim.handle, arr, 1, steps, 0, None)
    sim._moved()
    sol.from_c(arr[0])
    return rc


def _phases(sim, sol):
    sim.computePhiGradients()
    sim.collidePhase()
    sim.streamPhase()
    sim.collideHydro()
    sim.streamHydroAndMacro(sol)


def _same(a, b):
    for k in STATE:
        ref = b.field64(k)
        err = np.abs(a.field64(k) - ref).max()
        assert err <= 1e-10 * np.abs(ref).max(), (k, err)


@pytest.mark.parametrize("steps", [1, 2, 3])
def test_fields_of_a_run_without_room(gpu, steps):
    from b200lbm import _capi
    sim, sol = _moved(gpu)
    tag = np.array(sim.tag)
    twin, rest = gpu.Sim(*DIMS, storage="f64"), None
    scenes._params(twin, 0.8, 0.7, 0.008, 0.0015)
    twin.initFlat(25)
    for k in STATE:
        getattr(twin, k)[:] = np.array(getattr(sim, k))
    # in the first two steps the box reaches from corner to corner, and the tags
    # stay; in the third it is the moved sphere's again
    two = gpu.RigidSphere(*DIMS, cx=10, cy=10, cz=10, r=5.3, density=2.0)
    ref, at = _moved(gpu)
    assert _run(gpu, ref, at, 2) == _capi.ERR_CAPACITY
    two.cx, two.cy, two.cz, two.vx, two.vy, two.vz = at.cx, at.cy, at.cz, at.vx, at.vy, at.vz
    two.wx, two.wy, two.wz = at.wx, at.wy, at.wz
    assert np.array_equal(np.asarray(ref.tag), tag)
    for t in range(steps):
        if t == 2:
            twin.retagCells(two)
            new = np.array(twin.tag)
            twin.tag[:] = np.where(tag == 1, tag, new)
        else:
            twin.tag[:] = tag
        _phases(twin, two if t == 2 else rest)
    assert _run(gpu, sim, sol, steps) == _capi.ERR_CAPACITY
    assert np.array_equal(np.asarray(sim.tag), np.asarray(twin.tag))
    _same(sim, twin)
    for s in (sim, twin, ref):
        s.close()


@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_the_next_step_retags_the_whole_grid(gpu, storage):
    sim, sol = _moved(gpu, storage)
    assert _run(gpu, sim, sol, 2) != 0
    for _ in range(2):
        sim.step(sol)
        z, y, x = np.nonzero(np.asarray(sim.tag).reshape(DIMS[::-1]) == 1)
        assert len(z) > 500
        assert np.all((x + 0.5 - sol.cx) ** 2 + (y + 0.5 - sol.cy) ** 2 + (z + 0.5 - sol.cz) ** 2 <= sol.r ** 2)
        for k in STATE:
            assert np.isfinite(np.asarray(getattr(sim, k))).all(), k
    sim.close()


@pytest.mark.parametrize("storage", ["f32", "f64"])
def test_nothing_of_a_run_without_room_is_left_in_later_steps(gpu, storage):
    """A split step with written tags gives the same bits on a handle with such a
    run behind it as on a new one."""
    got = []
    for failed in (True, False):
        if failed:
            sim, sol = _moved(gpu, storage)
            assert _run(gpu, sim, sol, 2) != 0
        else:
            sim = gpu.Sim(*DIMS, storage=storage)
            scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
        sim.initFlat(25)
        sol = gpu.RigidSphere(*DIMS, cx=30.2, cy=29.8, cz=27.1, r=5.3, density=2.0)
        rs = np.random.RandomState(5)
        for k in ("ux", "uy", "uz"):
            getattr(sim, k)[:] = rs.uniform(-0.05, 0.05, sim.n).astype(np.float32)
        for _ in range(2):
            sim.step_begin(sol)
            tag = np.array(sim.tag).reshape(DIMS[::-1])
            tag[11, 10, 8:12] = 1  # where the first sphere was
            sim.tag[:] = tag.ravel()
            sim.step_end(sol)
        got.append({k: sim.field64(k) for k in STATE})
        sim.close()
    for k in STATE:
        assert np.array_equal(got[0][k], got[1][k]), k
