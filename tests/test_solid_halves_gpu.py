"""Cells that a step does not update (SOLID, written WALL, the domain's faces)
through the calls that touch one half, or tags, between steps: nothing is
computed for them, so they hold one value in both halves whatever number of
steps follows."""
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


DIMS = (32, 17, 26)  # (nx * ny divisible by 8: plane copies)


def _tank(gpu, storage="f32", level=8, dims=DIMS):
    sim = gpu.Sim(*dims, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(level)
    sol = gpu.RigidSphere(*dims, cx=dims[0] / 2 + 0.3, cy=dims[1] / 2 + 0.1, cz=dims[2] / 2 - 0.4, r=4.2, density=2.0)
    return sim, sol


def _cells(sim, k):
    return np.array(getattr(sim, k)).reshape(sim.n, -1)


@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
def test_copied_planes_hold_their_solid_cells_in_both_halves(gpu, storage):
    """lbm_slab_copy_planes copies the current half; the SOLID and face cells of
    those planes, and no others, are the same in the other half when it returns."""
    (src, sol), (dst, _) = _tank(gpu, storage, 8), _tank(gpu, storage, 12)
    for _ in range(2):
        src.step(sol)
        dst.step(sol)
    was = {k: _cells(dst, k) for k in ("f", "f2", "h2")}
    plane, nxny = 12, DIMS[0] * DIMS[1]
    gpu._capi.check(dst.handle, gpu._capi.lib().lbm_slab_copy_planes(dst.handle, plane, src.handle, plane, 2))
    dst._moved()
    z = np.arange(dst.n) // nxny
    assert (np.asarray(dst.tag) == 1).sum() > 60
    copied = (np.asarray(dst.tag) != 0) & (z >= plane) & (z < plane + 2)
    assert copied.sum() > 60
    assert not np.array_equal(_cells(src, "f")[copied], was["f"][copied])
    for k, k2 in (("f", "f2"), ("h", "h2")):
        assert np.array_equal(_cells(dst, k)[copied], _cells(src, k)[copied]), k
        assert np.array_equal(_cells(dst, k2)[copied], _cells(src, k)[copied]), k2
    for k in ("f2", "h2"):
        assert np.array_equal(_cells(dst, k)[~copied], was[k][~copied]), k
    src.close()
    dst.close()


FIELDS = ("f", "h", "phi", "rho", "ux", "uy", "uz")


@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
@pytest.mark.parametrize("how", ["step", "run_coupled", "batch"])
def test_walls_that_turn_solid(gpu, storage, how):
    """Interior cells written WALL that the sphere then covers."""
    sim, sol = _tank(gpu, storage)
    away = gpu.RigidSphere(*DIMS, cx=5.2, cy=5.1, cz=5.3, r=1.4, density=2.0)
    for _ in range(3):
        sim.step(away)
    tag = np.array(sim.tag).reshape(DIMS[::-1])
    tag[8:17, 6:13, 12:21] = 2
    sim.tag[:] = tag.ravel()
    before = {k: _cells(sim, k) for k in FIELDS}
    sol.vx = sol.vy = sol.vz = 0.0
    for t in range(3):
        if how == "step":
            sim.step(sol)
        elif how == "run_coupled":
            sim.run_coupled(sol, 1)
        else:
            with gpu.Batch([(sim, sol)]) as batch:
                batch.run(1)
        now = np.asarray(sim.tag) == 1
        solid = now & (tag.ravel() == 2)  # (the sphere moves less than a cell)
        assert solid.sum() > 100
        for k in FIELDS:
            assert np.array_equal(_cells(sim, k)[solid], before[k][solid]), (t, k)
    sim.close()


@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
@pytest.mark.parametrize("write", ["tag", "f2"])
def test_a_write_inside_a_split_step(gpu, storage, write):
    """Cells written SOLID or WALL, and cells at rest whose other half was
    written, between step_begin and step_end keep their values through the step."""
    sim, sol = _tank(gpu, storage)
    for _ in range(4):
        sim.step(sol)
    sim.step_begin(sol)
    if write == "tag":
        for at in ((4, 12, 5), (5, 12, 5), (9, 13, 20), (16, 13, 12)):
            sim.tag[sim.idx(*at)] = 1
        for at in ((7, 4, 9), (7, 14, 9), (20, 3, 21)):
            sim.tag[sim.idx(*at)] = 2
    else:
        sim.f2[:] = np.float32(0.25)
        sim.h2[:] = np.float32(0.125)
    rest = np.asarray(sim.tag) != 0
    want = {k: _cells(sim, k)[rest] for k in FIELDS}
    sim.step_end(sol)
    for k in FIELDS:
        assert np.array_equal(_cells(sim, k)[rest], want[k]), k
    sim.close()


@pytest.mark.parametrize("how", ["run_coupled", "batch"])
def test_a_run_of_no_steps_changes_nothing(gpu, how):
    sim, sol = _tank(gpu)
    for _ in range(3):
        sim.step(sol)
    sim.f2[:] = np.float32(0.25)
    sim.h2[:] = np.float32(0.125)
    names = FIELDS + ("f2", "h2", "tag", "tagPrev")
    was = {k: _cells(sim, k) for k in names}
    state = sol.state()
    if how == "batch":
        with gpu.Batch([(sim, sol)]) as batch:
            batch.run(0)
    else:
        sim.run_coupled(sol, 0)
    for k in names:
        assert np.array_equal(_cells(sim, k), was[k]), k
    assert sol.state() == state
    sim.close()
