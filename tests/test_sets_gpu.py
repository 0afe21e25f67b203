"""The fresh and dead lists and the fresh fill (k_sets) where its groups, its
rounds and its tiles of the box have edges: one fresh cell, lists around a group
of 32, lists of a thousand cells whose values hang on one another from the first
to the last, a box of more than 256 chunks of 2,048 cells, and a cell without a
FLUID neighbour.  The filled phi, rho and u are means of FP64 sums in a stated
order, so they are the loop's bit for bit; the equilibria are rounded once from
FP64, so they are within one unit in the last place of the loop's."""
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


DIRS = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
        (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1),
        (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1), (1, 1, 1), (-1, -1, -1),
        (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]
W27 = [float(np.float32((8 / 27, 2 / 27, 1 / 54, 1 / 216)[sum(map(abs, e))])) for e in DIRS]
W7 = [0.25] + [0.125] * 6


def _loop(tag, prev, v, rhoL, rhoG, dtype):
    """handleFreshCells in scan order over v = [phi, rho, ux, uy, uz] (z, y, x);
    returns the filled cells' f and h."""
    f, h = {}, {}
    for z, y, x in np.argwhere((tag == 0) & (prev == 1)):
        sums, cnt = [0.0] * 5, 0
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if (dz, dy, dx) != (0, 0, 0) and tag[z + dz, y + dy, x + dx] == 0:
                        sums = [s + float(a[z + dz, y + dy, x + dx]) for s, a in zip(sums, v)]
                        cnt += 1
        p, r, ux, uy, uz = [s / cnt for s in sums] if cnt else [float(v[0][z, y, x]), 1.0, 0.0, 0.0, 0.0]
        for a, val in zip(v, (p, r, ux, uy, uz)):
            a[z, y, x] = dtype(val)
        ph, u2 = rhoG + p * (rhoL - rhoG), ux * ux + uy * uy + uz * uz
        eu = [e[0] * ux + e[1] * uy + e[2] * uz for e in DIRS]
        f[z, y, x] = [w * (r + ph * (c * (3 + 4.5 * c) - 1.5 * u2)) for w, c in zip(W27, eu)]
        h[z, y, x] = [w * p * (1 + 4 * c) for w, c in zip(W7, eu)]
    return f, h


def _field(sim, dtype, k):
    return np.array(getattr(sim, k)) if dtype == np.float32 else sim.field64(k)


def _check(sim, dtype, retag):
    nx, ny, nz = sim.nx, sim.ny, sim.nz
    rs = np.random.RandomState(5)
    start = [rs.uniform(0, 1, sim.n), rs.uniform(0.9, 1.1, sim.n)] + [rs.uniform(-0.05, 0.05, sim.n) for _ in range(3)]
    for k, a in zip(("phi", "rho", "ux", "uy", "uz"), start):
        getattr(sim, k)[:] = a.astype(np.float32)
    retag()
    tag, prev = (np.array(t).reshape(nz, ny, nx) for t in (sim.tag, sim.tagPrev))
    v = [a.astype(np.float32).astype(dtype).reshape(nz, ny, nx) for a in start]
    f, h = _loop(tag, prev, v, 1.0, 0.1, dtype)
    for k, a in zip(("phi", "rho", "ux", "uy", "uz"), v):
        assert np.array_equal(_field(sim, dtype, k).reshape(nz, ny, nx), a), k
    F, H = _field(sim, dtype, "f").reshape(nz, ny, nx, 27), _field(sim, dtype, "h").reshape(nz, ny, nx, 7)
    # FP32: the FP64 value rounded once; FP64: a few operations, contracted or not
    eps = 2.0 ** -23 if dtype == np.float32 else 2.0 ** -50
    for at in f:
        assert np.all(np.abs(F[at] - f[at]) <= eps * np.abs(f[at])), at
        assert np.all(np.abs(H[at] - h[at]) <= eps * (np.abs(h[at]) + 1e-30)), at
    return len(f)


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("dims,r,shift,least", [
    ((30, 26, 28), 0.8, 0.9, 1),        # a cell or two
    ((30, 26, 28), 4.2, 0.6, 20),       # less than or about a group
    ((44, 26, 28), 5.3, 3.0, 100),      # some groups, chains across them
    ((60, 26, 28), 7.4, 20.0, 1000),    # the whole sphere, from its rim inwards
    ((90, 86, 88), 40.2, 0.4, 300),     # more than 256 chunks in the box
])
def test_fill_equals_the_loop(gpu, storage, dims, r, shift, least):
    sim = gpu.Sim(*dims, storage=storage)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(12)
    m = r + 1.6
    sol = gpu.RigidSphere(*dims, cx=m, cy=dims[1] / 2 + 0.1, cz=dims[2] / 2 + 0.2, r=r, density=2.0)
    sim.retagCells(sol)

    def retag():
        sol.cx += shift
        sim.retagCells(sol)
        sim.handleFreshCells(sol)

    n = _check(sim, np.float32 if storage == "f32" else np.float64, retag)
    assert n >= least, n
    sim.close()


class _AllBut:
    """Everything but the given cells is inside, at rest."""
    def __init__(self, cells):
        self.cells = cells

    def contains(self, x, y, z):
        return (int(x), int(y), int(z)) not in self.cells

    def surfaceVelocity(self, x, y, z, out):
        out[:] = [0.0, 0.0, 0.0]
        return out


def test_fill_without_fluid_neighbours(gpu):
    sim = gpu.Sim(12, 11, 10)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(6)
    sim.retagCells(_AllBut(set()))

    def retag():
        sol = _AllBut({(4, 5, 6), (8, 2, 3), (8, 3, 3)})
        sim.retagCells(sol)
        sim.handleFreshCells(sol)

    assert _check(sim, np.float32, retag) == 3
    sim.close()
