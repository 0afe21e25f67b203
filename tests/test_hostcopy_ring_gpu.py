"""Which copies go through the page-locked ring (lbm_test_ring_copies): results
of 16 MB and more into pageable memory, where the machine has four cores."""
import ctypes as C
import os

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


def _count(gpu):
    v = C.c_int64()
    gpu._capi.check(None, gpu._capi.lib().lbm_test_ring_copies(C.byref(v)))
    return v.value


def _copies(gpu, call):
    before = _count(gpu)
    call()
    return _count(gpu) - before


@pytest.mark.skipif(len(os.sched_getaffinity(0)) < 4, reason="the ring needs four cores")
@pytest.mark.parametrize("dims", [(128, 256, 127), (128, 256, 128), (251, 173, 199)])
def test_large_results_go_through_the_ring(gpu, dims):
    sim = gpu.Sim(*dims)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(dims[1] / 2)
    sim.synchronize()
    big = 4 * sim.n >= 16 << 20
    got = np.empty(sim.n, np.float32)

    def read():
        gpu._capi.check(sim.handle, gpu._capi.lib().lbm_download_field(
            sim.handle, gpu._capi.FIELDS["phi"], got.ctypes.data, got.size))

    assert _copies(gpu, read) == int(big)
    assert _copies(gpu, lambda: sim.packVolume(np.empty(2 * sim.n, np.uint8))) == int(2 * sim.n >= 16 << 20)
    locked = sim.frameBuffer()
    assert _copies(gpu, lambda: sim.packVolume(locked)) == 0
    sim.close()
