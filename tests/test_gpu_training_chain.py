"""Training updates whose kernels start while their predecessors run: one call
with many updates (each update's first kernel runs beside the last update's
end) against one call per update (the stream is empty between them).  Every
kernel reads complete inputs either way, so errors and weights are the same
bits.  The last case has more weights per updater than the gain kernel reads
ahead (4096)."""
import os
import shutil

import numpy as np
import pytest

from n2p2_b200 import Mode, water
from n2p2_b200.training import ENERGY, FORCE, Training
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _wide(path):
    """The water40 model with 32-32 networks (4800 weights)."""
    src = os.path.join(H.GOLDEN, "models", "water40")
    os.makedirs(path)
    shutil.copy(os.path.join(src, "scaling.data"), path)
    with open(os.path.join(src, "input.nn")) as f, open(os.path.join(path, "input.nn"), "w") as g:
        g.write(f.read().replace("global_nodes_short 25 25", "global_nodes_short 32 32"))
    rng = np.random.default_rng(1)
    for z in (1, 8):
        np.savetxt(os.path.join(path, "weights.%03d.data" % z), rng.normal(0.0, 0.2, 40 * 32 + 32 + 32 * 32 + 32 + 33))
    return path


def _run(model, setup, split):
    mode = Mode(0).setupFromDirectory(model)
    structs = [water.water_box(n, 40 + n, sigma=0.1) for n in (8, 17, 40)]
    b = mode.batch(structs)
    b.setPositions(np.concatenate([s.positions for s in structs]))
    b.evaluate()
    energies, forces = b.energies(), b.forces()
    b.close()
    t = Training(mode, structs, energies, forces)
    rng = np.random.default_rng(3)
    t.setWeights(t.weights() + rng.normal(0.0, 0.02, t.weights().size))
    group = setup(t)
    t.setForceWeight(10.0)
    out = []
    for prop, count in ((ENERGY, 12), (FORCE, 12), (ENERGY, 6), (FORCE, 6)):
        # no structure twice in a group of three (a full Jacobian needs independent columns)
        s = np.concatenate([rng.permutation(len(structs)) for _ in range(count // 3)]).astype(np.int32)
        a = np.array([rng.integers(0, structs[k].numAtoms) for k in s], dtype=np.int32)
        c = rng.integers(0, 3, count).astype(np.int32)
        step = group if split else count
        for k in range(0, count, step):
            q = slice(k, k + step)
            out.append(t.update(prop, s[q]) if prop == ENERGY else t.update(prop, s[q], a[q], c[q]))
    w = t.weights()
    t.close()
    mode.close()
    return np.concatenate(out), w


def _kalman(kind, strategy=0, batch=1, jacobian=1):
    def setup(t):
        t.setUpdateStrategy(strategy)
        t.setJacobianMode(jacobian)
        t.setTaskBatchSize(batch, batch)
        t.setupUpdaterKalman(kind)
        return batch
    return setup


def _adam(t):
    t.setupUpdaterGradient(1)
    return 1


@pytest.mark.parametrize("wide,setup", [
    (False, _kalman(0)), (False, _kalman(1)), (False, _kalman(0, strategy=1)), (False, _kalman(0, batch=3)),
    (False, _kalman(0, batch=3, jacobian=2)), (False, _adam), (True, _kalman(0)),
], ids=["standard", "fading", "element", "batch", "jacobian", "adam", "wide"])
def test_updates_of_one_call_equal_single_calls(tmp_path, wide, setup):
    model = _wide(str(tmp_path / "model")) if wide else os.path.join(H.GOLDEN, "models", "water40")
    e0, w0 = _run(model, setup, False)
    e1, w1 = _run(model, setup, True)
    assert np.isfinite(w0).all() and np.any(e0 != 0.0)
    np.testing.assert_array_equal(e0, e1)
    np.testing.assert_array_equal(w0, w1)
