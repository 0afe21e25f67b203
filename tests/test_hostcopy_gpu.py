"""Large results arrive whole through the threaded copy: fields and frames at
sizes around its pieces (512 KB) and its least size (16 MB), read by one thread
and by several at once (one has the ring, the others the runtime's copy)."""
import threading

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


def _sim(gpu, dims, seed):
    sim = gpu.Sim(*dims)
    scenes._params(sim, 0.8, 0.7, 0.008, 0.0015)
    sim.initFlat(dims[1] * 0.5)
    want = np.random.RandomState(seed).uniform(0, 1, sim.n).astype(np.float32)
    sim.phi[:] = want
    sim._sync()
    return sim, want


def _read(gpu, sim):
    got = np.full(sim.n, -1, np.float32)
    gpu._capi.check(sim.handle, gpu._capi.lib().lbm_download_field(
        sim.handle, gpu._capi.FIELDS["phi"], got.ctypes.data, got.size))
    return got


@pytest.mark.parametrize("dims", [(12, 12, 12), (107, 89, 101), (160, 160, 163), (128, 256, 128), (128, 256, 129),
                                  (251, 173, 199)])
def test_fields_and_frames_arrive_whole(gpu, dims):
    sim, want = _sim(gpu, dims, 3)
    assert np.array_equal(_read(gpu, sim), want)
    pageable = sim.packVolume(np.zeros(2 * sim.n, np.uint8))
    locked = sim.frameBuffer()
    sim.packVolume(locked)
    assert np.array_equal(pageable, np.asarray(locked)[:2 * sim.n])
    assert np.array_equal(pageable[::2], np.floor(want.astype(np.float64) * 255).astype(np.uint8))
    sim.close()


def test_several_threads_read_at_once(gpu):
    made = [_sim(gpu, (200, 160, 140 + 7 * k), k) for k in range(4)]
    bad = []

    def loop(sim, want):
        for _ in range(8):
            if not np.array_equal(_read(gpu, sim), want):
                bad.append(sim.n)

    ts = [threading.Thread(target=loop, args=m) for m in made]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for sim, _ in made:
        sim.close()
    sim, want = _sim(gpu, (200, 160, 140), 9)  # the ring was given back and is made again
    assert np.array_equal(_read(gpu, sim), want)
    sim.close()
