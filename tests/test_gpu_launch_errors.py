"""A CUDA error that a caller has left pending on its thread (here an invalid
device ordinal, refused by the runtime) neither fails an evaluation, a
training step or the statistics, nor is it taken from the caller."""
import ctypes

import numpy as np
import pytest

from n2p2_b200 import _lib, water
from n2p2_b200.mode import Trainer
from n2p2_b200.training import ENERGY, FORCE, Training
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture
def runtime():
    _lib.load()
    rt = ctypes.CDLL("libcudart.so.12")
    rt.cudaGetLastError()
    yield rt
    rt.cudaGetLastError()


def _calls():
    """Every kind of call that checks its launches, one at a time."""
    boxes = water.water_batch(3, seed=1, n_min=32, n_max=40)
    m = H.gpu_mode(H.WATER40)
    b = m.batch(boxes)
    b.setPositions(np.concatenate([s.positions for s in boxes]))
    yield b.evaluate(forces=True, graph=False)
    yield b.autotune(useCache=False)
    for _ in range(2):   # captured, replayed
        b.evaluate(forces=True)
        yield b.synchronize()
    E, F = b.energies(), b.forces()
    yield b.symmetryFunctionStatistics()
    yield Trainer(m).step(b, E, F, update=True)
    t = Training(m, boxes, E, F)
    yield t.setupUpdaterKalman(0)
    yield t.update(ENERGY, [0])
    yield t.update(FORCE, [0], [1], [2])
    yield t.errors()
    t.close()
    m.close()


def test_pending_error_stays_the_callers(runtime):
    for _ in _calls():   # the CUDA runtime itself clears it where it loads a kernel for the first time
        pass
    assert runtime.cudaSetDevice(999) == 101   # cudaErrorInvalidDevice
    for _ in _calls():
        assert runtime.cudaPeekAtLastError() == 101
