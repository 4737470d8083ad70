"""launchCount() of an evaluation launched kernel by kernel equals the kernels
of the captured graph, for models of the pair kernels, of the general kernels,
of the compact functions, with stored derivatives and symmetry functions
alone."""
import os

import numpy as np
import pytest

from n2p2_b200 import Mode, read_structures, water
from tests import helpers as H

pytestmark = pytest.mark.gpu

GENERAL = [f"symfunction_short {ec} 3 {a} {b} 0.01 1 2.5 12.0" for ec in "HO" for a, b in ("HH", "HO", "OO")]


def _general(d):
    (d / "input.nn").write_text(water.input_nn_text(GENERAL, nodes=(8, 8), scaling=False))
    rng = np.random.default_rng(5)
    for z in (1, 8):
        water.write_weights(str(d / f"weights.{z:03d}.data"), water.random_weights([3, 8, 8, 1], rng))
    m = Mode(0)
    m.initialize()
    m.loadSettingsFile(str(d / "input.nn"))
    m.setupGeneric()
    m.setupSymmetryFunctionScalingNone()
    m.setupNeuralNetworkWeights(str(d / "weights.%03zu.data"))
    return m


@pytest.mark.parametrize("model", ["water40", "mixed", "general", "anisole", "narrow", "weighted"])
def test_count_is_the_graphs(model, tmp_path):
    if model in ("water40", "mixed"):
        m, s = H.gpu_mode(H.WATER40, "fp64" if model == "water40" else "mixed"), [water.water_box(32, seed=1)]
    elif model == "general":
        m, s = _general(tmp_path), [water.water_box(32, seed=1)]
    else:
        d = {"anisole": ("examples", "Anisole_SCAN"), "narrow": ("models", "scan_narrow"),
             "weighted": ("models", "qm9_weighted")}[model]
        d = os.path.join(H.GOLDEN, *d)
        m, s = H.gpu_mode(d), read_structures(os.path.join(d, "input.data"))[:1]
    m.setAutotune(False)
    b = m.batch(s)
    b.setPositions(np.concatenate([x.positions for x in s]))
    kinds = [{}, {"forces": False}, {"symmetryFunctionsOnly": True}]
    if model == "water40":
        kinds.append({"storeDGdr": True})
    b.evaluate()
    for kind in kinds:
        b.evaluate(graph=False, **kind)
        direct = b.launchCount()
        b.evaluate(**kind)
        b.synchronize()
        assert b.launchCount() == direct, kind
