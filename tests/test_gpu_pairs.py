"""The pair kernels of the symmetry-function passes (sf_pairs.cuh) against the
C restatement of the reference, for every form a model's groups can take
there: zeta powers of two up to 4 and 16 and other integers, one to three
widths, lambda other than +-1 (and beyond 1, where terms vanish), shifted
radial functions, every kind of cutoff function, angular cutoffs below the
list's; and for atoms of every tier of the stage (from none to more than 384
neighbours); and the stored derivatives
(k_pair_derivatives.cu) through the forces contracted from them.

Tolerances: those of the other parity tests (energies 1e-10 relative, forces
1e-10 of the largest component), and for the mixed form its budget of
1 meV/atom and 30 meV/Angstrom.
"""
import numpy as np
import pytest

from n2p2_b200 import Mode, Structure, water
from n2p2_b200.scaling import collect_statistics, write_scaling
from tests import helpers as H

pytestmark = pytest.mark.gpu

HA_TO_MEV = 27211.386
HA_BOHR_TO_MEV_A = 27211.386 / 0.529177


def _lines(angular, radial=((0.01, 0.0), (0.3, 1.5)), rc_radial=12.0):
    """angular: (type, eta, lambda, zeta, rc) for every element pair of every element."""
    out = []
    for ec in ("H", "O"):
        for e1 in ("H", "O"):
            out += [f"symfunction_short {ec} 2 {e1} {eta} {rs} {rc_radial}" for eta, rs in radial]
        for e1, e2 in (("H", "H"), ("H", "O"), ("O", "O")):
            out += [f"symfunction_short {ec} {t} {e1} {e2} {eta} {lam} {zeta} {rc}" for t, eta, lam, zeta, rc in angular]
    return out


def _grid(t, etas, zetas, lams=(-1, 1), rc=12.0):
    return [(t, e, la, z, rc) for e in etas for la in lams for z in zetas]


FORMS = {
    "zeta4": ("6 0.0", _grid(3, (0.01, 0.03), (1, 2, 4))),
    "one_eta": ("6 0.0", _grid(3, (0.02,), (1, 4), (1,))),
    "three_etas": ("6 0.0", _grid(3, (0.004, 0.01, 0.025), (4,)) + _grid(9, (0.01,), (1, 2))),
    "zeta16": ("6 0.0", _grid(3, (0.01, 0.03), (1, 4)) + _grid(9, (0.001, 0.01), (1, 2, 4, 16))),
    "narrow16": ("6 0.0", _grid(3, (0.01,), (8, 16)) + _grid(9, (0.01,), (2,), (1,))),
    "inner_radius": ("6 0.2", _grid(3, (0.01, 0.03), (1, 4))),
    "tanh": ("2 0.0", _grid(3, (0.01, 0.03), (1, 4)) + _grid(9, (0.01,), (8,))),
    "cosine": ("1 0.2", _grid(3, (0.01,), (2, 16))),
    "hard": ("0 0.0", _grid(3, (0.05,), (1, 2))),
    "integers": ("6 0.0", _grid(3, (0.01, 0.03), (1, 3, 6)) + _grid(9, (0.01,), (1, 2, 3, 5, 7, 11))),
    "lambdas": ("6 0.0", _grid(3, (0.01,), (1, 2), (-1, 0.5, 1))),
    "lambda_beyond": ("6 0.0", _grid(3, (0.01,), (1, 3), (-1.5, 1))),
    "general_zeta": ("6 0.0", _grid(3, (0.01, 0.03), (1, 2.5)) + _grid(9, (0.01, 0.02, 0.05), (1, 1.5))),
    "general_shift": ("3 0.0", _grid(3, (0.01, 0.03), (1, 4), rc="12.0 1.0") + _grid(9, (0.01,), (2,))),
    "short_angular": ("6 0.0", _grid(3, (0.01, 0.03), (1, 4), rc=8.0) + _grid(9, (0.02,), (2,), rc=6.0)),
}


@pytest.fixture(scope="module")
def structures():
    def box(n, seed, f=1.0):
        s = water.water_box(n, seed=seed, sigma=0.08)
        return Structure(s.positions * f, s.elements, box=s.box * f)
    m = water.water_box(32, seed=3)
    return [box(33, 1), box(40, 2), box(40, 4, 0.92), box(48, 5, 0.8), box(48, 6, 0.62),
            Structure(m.positions[:3], m.elements[:3]), Structure(m.positions[:1], m.elements[:1]),
            Structure(m.positions[:7], m.elements[:7])]


def _model(tmp_path, cutoff, lines, structures):
    d = tmp_path
    (d / "input.nn").write_text(water.input_nn_text(lines, nodes=(8, 8), cutoff=cutoff))
    m = Mode(0)
    m.initialize()
    m.loadSettingsFile(str(d / "input.nn"))
    m.setupGeneric()
    m.setupSymmetryFunctionScalingNone()
    write_scaling(str(d / "scaling.data"), collect_statistics(m, structures))
    m.close()
    rng = np.random.default_rng(5)
    n = len(lines) // 2
    for z in (1, 8):
        water.write_weights(str(d / f"weights.{z:03d}.data"), water.random_weights([n, 8, 8, 1], rng))
    return str(d)


@pytest.mark.parametrize("form", FORMS)
def test_forms_and_tiers(form, structures, tmp_path):
    from oracle import port
    cutoff, angular = FORMS[form]
    d = _model(tmp_path, cutoff, _lines(angular), structures)
    ref = [port.PortModel(d).evaluate(s) for s in structures]
    counts = np.concatenate([np.diff(r["nbr_offset"]) for r in ref])
    assert counts.min() == 0 and counts.max() > 384
    for a, b in ((1, 128), (129, 160), (161, 384)):
        assert ((counts >= a) & (counts <= b)).any()
    natoms = np.array([s.numAtoms for s in structures])
    start = np.concatenate([[0], np.cumsum(natoms)])
    for precision in ("fp64", "mixed"):
        m = H.gpu_mode(d, precision=precision)
        b = m.batch(structures)
        b.setPositions(np.concatenate([s.positions for s in structures]))
        for shape in range(4 if precision == "fp64" else 3):   # 3: with stored dG/dr
            if shape < 3:
                b.setShapes(shape, shape)
            b.evaluate(forces=True, storeDGdr=shape == 3, graph=False)
            E, F = b.energies(), b.forces()
            for k, r in enumerate(ref):
                f = F[start[k]:start[k + 1]]
                de, df = abs(E[k] - r["energy"]), np.abs(f - r["forces"]).max()
                if precision == "fp64":
                    assert de <= 1e-10 * abs(r["energy"]), (form, shape, k)
                    assert df <= 1e-10 * np.abs(r["forces"]).max() + 1e-13, (form, shape, k)
                else:
                    assert de / natoms[k] * HA_TO_MEV <= 1.0 and df * HA_BOHR_TO_MEV_A <= 30.0, (form, shape, k)
        b.close()
        m.close()
