"""Which networks an evaluation of the mixed form runs depends on the model
alone: a structure's atomic energies, dE/dG and forces are the same bits alone
and in a batch of 5,000 and more atoms.  Elements with up to 2,048 parameters
run the FP64 networks, larger ones the tensor cores (split bfloat16), in every
batch: shown by the distance from the same networks in numpy over the batch's
own symmetry functions, which is rounding for the first and above 1e-9 Ha for
the second.

Tolerances.  FP64: a sum of n products is off by (n + 1) eps times the sum of
their sizes and softplus has slope <= 1: 2 * 200 eps times the network over absolute
values (at most 15 + 65 + 65 products and biases on a path).  Tensor cores: the
mixed form's budget, 1 meV per atom, half of it for an atom as in the direct
test of that kernel; dE/dG to 1e-3 of its largest value."""
import os

import numpy as np
import pytest

from n2p2_b200 import water
from n2p2_b200.mode import Mode
from n2p2_b200.scaling import collect_statistics, write_scaling
from tests import helpers as H

pytestmark = pytest.mark.gpu

# 14 inputs: 14-40-33-1 has 1,987 parameters, 14-40-35-1 2,071; the larger ones around the
# tensor-core kernel's padding of widths to 16 and up to its limit of 64
NODES = [(16, 16), (33, 37), (40, 33), (40, 35), (33, 64), (47, 48), (49, 49), (64, 33), (64, 64)]


def parameters(sizes):
    return sum(a * b + b for a, b in zip(sizes[:-1], sizes[1:]))


@pytest.fixture(scope="module")
def boxes():
    return water.water_batch(4, seed=17, n_min=32, n_max=64)


@pytest.fixture(scope="module")
def crowd():
    return water.water_batch(16, seed=18, n_min=100, n_max=140)


def _model(d, nodes, boxes):
    lines = []
    for ec in ("H", "O"):
        for e1 in ("H", "O"):
            lines += [f"symfunction_short {ec} 2 {e1} {eta} 0.0 12.0" for eta in (0.001, 0.01, 0.05, 0.2)]
        for e1, e2 in (("H", "H"), ("H", "O"), ("O", "O")):
            lines += [f"symfunction_short {ec} 3 {e1} {e2} 0.01 {lam} 1 12.0" for lam in (-1, 1)]
    text = water.input_nn_text(lines, nodes=nodes)
    (d / "input.nn").write_text(text)
    m = Mode(0)
    m.initialize()
    m.loadSettingsFile(str(d / "input.nn"))
    m.setupGeneric()
    m.setupSymmetryFunctionScalingNone()
    write_scaling(str(d / "scaling.data"), collect_statistics(m, boxes))
    m.close()
    rng = np.random.default_rng(5)
    for z in (1, 8):
        water.write_weights(str(d / f"weights.{z:03d}.data"), water.random_weights([14, *nodes, 1], rng))
    return str(d)


def _network(d, z, sizes, x):
    """Energies, dE/dG and the network over absolute values (softplus, softplus, linear)."""
    w, pos, layers = np.loadtxt(os.path.join(d, "weights.%03d.data" % z), usecols=0), 0, []
    for a, b in zip(sizes[:-1], sizes[1:]):
        layers.append((w[pos:pos + a * b].reshape(a, b), w[pos + a * b:pos + a * b + b]))
        pos += a * b + b
    assert pos == w.size
    (w1, b1), (w2, b2), (w3, b3) = layers
    z1 = x @ w1 + b1
    z2 = np.logaddexp(0.0, z1) @ w2 + b2
    e = (np.logaddexp(0.0, z2) @ w3 + b3)[:, 0]
    slope = ((w3[:, 0] / (1.0 + np.exp(-z2))) @ w2.T / (1.0 + np.exp(-z1))) @ w1.T
    t = np.logaddexp(0.0, np.logaddexp(0.0, np.abs(x) @ np.abs(w1) + np.abs(b1)) @ np.abs(w2) + np.abs(b2))
    return e, slope, (t @ np.abs(w3) + np.abs(b3))[:, 0]


def _run(m, structs):
    b = m.batch(structs)
    b.setPositions(np.concatenate([s.positions for s in structs]))
    b.evaluate(forces=True)
    return b


@pytest.mark.parametrize("nodes", NODES, ids=lambda n: "x".join(map(str, n)))
def test_networks_of_a_model(nodes, boxes, crowd, tmp_path):
    d = _model(tmp_path, nodes, boxes)
    m = H.gpu_mode(d, precision="mixed")
    few, many = _run(m, boxes), _run(m, boxes + crowd)
    n = few.numAtoms
    assert many.numAtoms >= 5000
    E, D, F = few.atomicEnergies(), few.dEdG().reshape(n, -1), few.forces()
    assert np.array_equal(E, many.atomicEnergies()[:n])
    assert np.array_equal(D, many.dEdG().reshape(many.numAtoms, -1)[:n])
    assert np.array_equal(F, many.forces()[:n])
    G = few.symmetryFunctions().reshape(n, -1)
    fp64 = parameters((14, *nodes, 1)) <= 2048
    for e, z in ((0, 1), (1, 8)):
        rows = few.elements == e
        want, slope, mag = _network(d, z, (14, *nodes, 1), G[rows])
        off = np.abs(E[rows] - want)
        if fp64:
            assert np.all(off <= 400 * np.finfo(float).eps * mag)
        else:
            assert off.max() > 1e-9
            assert off.max() * H.HA_TO_MEV <= 0.5
            assert np.abs(D[rows] - slope).max() <= 1e-3 * np.abs(slope).max()


@pytest.mark.parametrize("model", ["water40", "water56", "student_water56"])
def test_shipped_models_do_not_depend_on_the_batch(model, boxes, crowd):
    m = H.gpu_mode(os.path.join(H.GOLDEN, "models", model), precision="mixed")
    few, many = _run(m, boxes), _run(m, boxes + crowd)
    n = few.numAtoms
    assert np.array_equal(few.atomicEnergies(), many.atomicEnergies()[:n])
    assert np.array_equal(few.forces(), many.forces()[:n])
