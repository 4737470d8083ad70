"""The staged compact kernels' two block shapes (atoms with up to 64
neighbours, and up to 256) on open clusters cut from the Anisole SCAN frame:
symmetry functions (types 20 and 22, p2 and p2a) against a numpy evaluation of
their definition within 1e-12 of each function's largest unscaled value, and
forces against central differences of the energies.

The difference quotient of step h = 1e-4 is off by h^2 E'''/6 and by rounding
2 eps |E| / h: |E| <= 600 Ha per cluster gives 3e-9 at most, and a third
derivative of 10 Ha/bohr^3 gives 2e-8; the bound is 1e-6."""
import os

import numpy as np
import pytest

from n2p2_b200 import Structure, read_structures
from tests import helpers as H

pytestmark = pytest.mark.gpu

MODEL = os.path.join(H.GOLDEN, "examples", "Anisole_SCAN")


def _part(x, lo, hi, asym):
    y = np.abs(x - 0.5 * (lo + hi)) / (0.5 * (hi - lo))
    inside = y < 1.0
    y = np.where(inside, y, 1.0)
    if asym:
        y = (2.0 - y) * y
    return np.where(inside, ((15.0 - 6.0 * y) * y - 10.0) * y ** 3 + 1.0, 0.0)


def _functions():
    """Per element, the functions in the networks' order (type, subtype, elements, rc, rl, angles)."""
    z = {"H": 1, "C": 6, "O": 8}
    key, rows = {}, {"H": [], "C": [], "O": []}
    for line in open(os.path.join(MODEL, "input.nn")):
        w = line.split("#")[0].split()
        if not w:
            continue
        if w[0] != "symfunction_short":
            key.setdefault(w[0], w[1:])
            continue
        t = int(w[2])
        el = sorted((w[3:4] if t == 20 else w[3:5]), key=z.get)
        num = [float(x) for x in w[3 + len(el):-1]]
        rows[w[1]].append(((t, w[-1], [z[e] for e in el], num[1], num[0], num[2:]), (t, el, num, w[-1])))
    return float(key["conv_length"][0]), {e: [f for _, f in sorted(r, key=lambda x: x[0])] for e, r in rows.items()}


def _values(s, length, functions):
    x = np.asarray(s.positions) * length
    el = np.array(s.elements)
    out = []
    for i in range(len(el)):
        d = np.delete(x, i, 0) - x[i]
        e = np.delete(el, i)
        r = np.linalg.norm(d, axis=1)
        angle = np.arccos(np.clip((d @ d.T) / np.outer(r, r), -1.0, 1.0))
        row, largest = [], []
        for t, pair, num, sub in functions[el[i]]:
            w = _part(r, num[0] * length, num[1] * length, sub.endswith("a"))
            if t == 20:
                row.append((w * (e == pair[0])).sum())
                continue
            k = _part(angle, *np.radians(num[2:]), False)
            np.fill_diagonal(k, 0.0)
            row.append((w * (e == pair[0])) @ k @ (w * (e == pair[1])) * (0.5 if pair[0] == pair[1] else 1.0))
        out.append(np.array(row))
    return out


@pytest.mark.parametrize("atoms", [2, 3, 40, 66, 150])
def test_values_and_forces(atoms):
    f = read_structures(os.path.join(MODEL, "input.data"))[0]
    near = np.argsort(np.linalg.norm(f.positions - f.positions.mean(0), axis=1))[:atoms]
    s = Structure(f.positions[near], [f.elements[k] for k in near])
    m = H.gpu_mode(MODEL)
    b = m.batch([s])
    b.setPositions(s.positions)
    b.evaluate()
    counts = np.diff(b.neighbors()["offset"])
    assert counts.max() <= 64 if atoms <= 40 else counts.max() > 64
    length, functions = _functions()
    want = _values(s, length, functions)
    got = H.unscaled_from_files(MODEL, s, b.symmetryFunctions())
    got = np.split(got, np.cumsum([len(w) for w in want])[:-1])
    size = {e: np.max([np.abs(w) for w, x in zip(want, s.elements) if x == e], axis=0) for e in set(s.elements)}
    for g, w, e in zip(got, want, s.elements):
        assert np.all(np.abs(g - w) <= 1e-12 * np.maximum(size[e], 1.0))
    forces = b.forces()
    for a, c in ((0, 0), (atoms - 1, 1), (atoms // 2, 2)):
        energy = []
        for sign in (1.0, -1.0):
            x = s.positions.copy()
            x[a, c] += sign * 1e-4
            b.setPositions(x)
            b.evaluate()
            energy.append(b.energies()[0])
        assert abs(forces[a, c] + (energy[0] - energy[1]) / 2e-4) <= 1e-6
