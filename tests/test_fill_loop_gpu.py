"""The fresh fill of a fused step (step_begin) against the reference's loop over
the scan-ordered list, written out in numpy, and the test hook's fill as a
kernel of its own.

The filled phi, rho and u are means of FP64 sums in a stated order: the loop's
bit for bit.  The equilibria are FP64 values rounded once to FP32 (half a unit in
the last place), in FP16 storage then as offsets rounded to FP16 (2^-11 of the
offset, or 2^-25 below FP16's normal range)."""
import numpy as np
import pytest

import scenes
from test_sets_gpu import W7, W27, _loop

pytestmark = pytest.mark.gpu

DIMS = (44, 29, 31)
MACROS = ("phi", "rho", "ux", "uy", "uz")


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


def _scene(gpu, storage):
    sim = gpu.Sim(*DIMS, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(12)
    sol = gpu.RigidSphere(*DIMS, cx=16.2, cy=14.1, cz=15.3, r=6.3, density=2.0)
    return sim, sol


def _hook(gpu, sim, on):
    gpu._capi.check(sim.handle, gpu._capi.lib().lbm_test_sequential_fill(sim.handle, int(on)))


@pytest.mark.parametrize("hook", [False, True])
@pytest.mark.parametrize("shift", [0.5, 2.2, 15.0])
@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
def test_step_begin_fills_as_the_loop(gpu, storage, shift, hook):
    sim, sol = _scene(gpu, storage)
    _hook(gpu, sim, hook)
    for _ in range(3):
        sim.step(sol)
    rs = np.random.RandomState(6)
    start = [rs.uniform(0, 1, sim.n), rs.uniform(0.9, 1.1, sim.n)] + [rs.uniform(-0.05, 0.05, sim.n) for _ in range(3)]
    for k, a in zip(MACROS, start):
        getattr(sim, k)[:] = a.astype(np.float32)
    sol.cx += shift
    sim.step_begin(sol)
    dtype = np.float64 if storage == "f64" else np.float32
    shape = DIMS[::-1]
    v = [a.astype(np.float32).astype(dtype).reshape(shape) for a in start]
    f, h = _loop(np.array(sim.tag).reshape(shape), np.array(sim.tagPrev).reshape(shape), v, 1.0, 0.1, dtype)
    assert len(f) > (40 if shift < 1 else 200)

    def field(k):
        return sim.field64(k) if storage == "f64" else np.array(getattr(sim, k))

    for k, a in zip(MACROS, v):
        assert np.array_equal(field(k).reshape(shape), a), k
    F, H = field("f").reshape(shape + (27,)), field("h").reshape(shape + (7,))
    eps = 2.0 ** -50 if storage == "f64" else 2.0 ** -23
    for at in f:
        for got, want, ref in ((F[at], np.array(f[at]), np.array(W27)), (H[at], np.array(h[at]), np.array(W7) * v[0][at])):
            bar = eps * (np.abs(want) + 1e-30)
            if storage == "f16":
                bar = bar + eps * np.abs(ref) + np.maximum(2.0 ** -11 * np.abs(want - ref), 2.0 ** -25)
            assert np.all(np.abs(got - want) <= bar), at
    sim.step_end(sol)
    sim.close()


def test_the_hook_has_a_kernel_of_its_own(gpu):
    """What the hook is compared with must not be the code it checks."""
    sim, sol = _scene(gpu, "f32")
    sim.step(sol)
    per = []
    for on in (False, True):
        _hook(gpu, sim, on)
        before = sim.launch_count()
        sim.step(sol)
        per.append(sim.launch_count() - before)
    assert per[1] == per[0] + 1, per
    sim.close()
