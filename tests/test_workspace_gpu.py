"""Device memory a scene allocates beside its fields: the retag's workspace is no
larger than the whole grid can need (2,048-cell chunks of 8 + 512 bytes)."""
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import b200lbm
    return b200lbm


@pytest.mark.parametrize("dims", [(12, 12, 12), (64, 48, 56), (61, 47, 83)])
def test_the_retag_workspace(gpu, dims):
    sim = gpu.Sim(*dims)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(dims[1] / 2)
    sim.tag[:] = sim.tag[:]  # the next step retags the whole grid
    before = sim.device_bytes()
    sim.step(None)
    chunks = (sim.n + 2047) // 2048
    grown = sim.device_bytes() - before
    assert 0 < grown <= 520 * chunks + 256, grown
    sim.run_coupled(None, 3)
    assert sim.device_bytes() - before == grown
    sim.close()
