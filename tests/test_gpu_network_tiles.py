"""Tiled FP64 networks of wide inputs (the Anisole SCAN model: 331-354 inputs,
30-20-1) against the same networks in numpy over the batch's own symmetry
functions: clusters around one tile of 8 atoms, one frame, and enough frames
for the tiles of 16.

Tolerance: a sum of n products is off by (n + 1) eps times the sum of their
sizes, softplus has slope <= 1 and curvature <= 1/4; so an atomic energy is off
by less than 2 * 420 eps T with T the same network over absolute values, and
dE/dG by less than that times (1 + T) over the product of absolute weights."""
import os

import numpy as np
import pytest

from n2p2_b200 import Structure, read_structures
from tests import helpers as H

pytestmark = pytest.mark.gpu

MODEL = os.path.join(H.GOLDEN, "examples", "Anisole_SCAN")
Z = {"H": 1, "C": 6, "O": 8}


def _layers(element, inputs):
    w = np.loadtxt(os.path.join(MODEL, "weights.%03d.data" % Z[element]), usecols=0)
    out, pos = [], 0
    for a, b in ((inputs, 30), (30, 20), (20, 1)):
        out.append((w[pos:pos + a * b].reshape(a, b), w[pos + a * b:pos + a * b + b]))
        pos += a * b + b
    assert pos == w.size
    return out


def _network(x, layers):
    (w1, b1), (w2, b2), (w3, b3) = layers
    z1 = x @ w1 + b1
    z2 = np.logaddexp(0.0, z1) @ w2 + b2
    e = (np.logaddexp(0.0, z2) @ w3 + b3)[:, 0]
    d = ((w3[:, 0] / (1.0 + np.exp(-z2))) @ w2.T / (1.0 + np.exp(-z1))) @ w1.T
    t = np.logaddexp(0.0, np.logaddexp(0.0, np.abs(x) @ np.abs(w1) + np.abs(b1)) @ np.abs(w2) + np.abs(b2))
    t = (t @ np.abs(w3) + np.abs(b3))[:, 0]
    p = (np.abs(w1) @ np.abs(w2) @ np.abs(w3))[:, 0]
    unit = 2 * 420 * np.finfo(float).eps
    return e, d, unit * t, unit * (1.0 + t)[:, None] * p


@pytest.mark.parametrize("atoms,copies", [(1, 1), (17, 1), (33, 1), (None, 1), (None, 20)])
def test_energies_and_derivatives(atoms, copies):
    f = read_structures(os.path.join(MODEL, "input.data"))[0]
    s = f
    if atoms:
        near = np.argsort(np.linalg.norm(f.positions - f.positions.mean(0), axis=1))[:atoms]
        s = Structure(f.positions[near], [f.elements[k] for k in near])
    b = H.gpu_mode(MODEL).batch([s] * copies)
    b.setPositions(np.concatenate([s.positions] * copies))
    b.evaluate()
    element = np.array(list(s.elements) * copies)
    G, D, E = b.symmetryFunctions(), b.dEdG(), b.atomicEnergies()
    width = {}
    for e in Z:   # inputs x 30 + 30, 30 x 20 + 20, 20 + 1 parameters
        size = np.loadtxt(os.path.join(MODEL, "weights.%03d.data" % Z[e]), usecols=0).size
        width[e] = (size - 671) // 30
    begin = np.concatenate([[0], np.cumsum([width[e] for e in element])])
    assert begin[-1] == G.size
    for e in Z:
        rows = np.flatnonzero(element == e)
        if rows.size == 0:
            continue
        take = begin[rows][:, None] + np.arange(width[e])
        want, slope, tolE, tolD = _network(G.ravel()[take], _layers(e, width[e]))
        assert np.all(np.abs(E[rows] - want) <= tolE)
        assert np.all(np.abs(D.ravel()[take] - slope) <= tolD)
