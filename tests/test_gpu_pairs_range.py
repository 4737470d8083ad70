"""The ends of the pair kernels' range of functions (sf_pairs.cuh): zeta up to
32, groups with zeta 1 to 4 alone and beside others, Gaussians that underflow
inside the cutoff (eta r^2 log2 e beyond the exponent range of a double,
shifted and not, radial, narrow and wide) and shifts far out.  They run there
(no candidate_masks stage, which only the general kernels have), with the C
restatement's energies and forces.

Tolerances: those of the other parity tests, 1e-10 of the energy and of the
largest force component."""
import numpy as np
import pytest

from n2p2_b200 import Mode, water
from n2p2_b200.scaling import collect_statistics, write_scaling
from tests import helpers as H

pytestmark = pytest.mark.gpu

PAIRS = (("H", "H"), ("H", "O"), ("O", "O"))
RADIAL = [(0.01, 0.0), (0.3, 1.5)]
PLAIN = [(3, 0.01, 1, 4)]
# cutoff 12: eta r_c^2 log2 e is 208 eta
FORMS = {
    "zeta31": (RADIAL, PLAIN + [(3, 0.01, 1, 31), (9, 0.01, -1, 31)]),
    "zeta32": (RADIAL, PLAIN + [(3, 0.01, 1, 32), (3, 0.01, -1, 32), (9, 0.02, 1, 32), (9, 0.02, 1, 16)]),
    "cubic": (RADIAL, [(3, e, la, z) for e in (0.01, 0.03) for la in (-1, 1) for z in (1, 3)] +
              [(9, 0.02, 0.5, z) for z in (2, 3, 4)]),
    "cubic_beside": (RADIAL, [(3, 0.01, la, z) for la in (-1, 1) for z in (3, 4)] + [(9, 0.02, 1, 7), (9, 0.05, -1, 3)]),
    "at_1000": (RADIAL + [(4.8, 0.0), (4.82, 0.0)], PLAIN),
    "wide_radial": (RADIAL + [(6.0, 0.0), (20.0, 0.0), (30.0, 2.0)], PLAIN),
    "far_shift": (RADIAL + [(2.0, 9.0), (4.0, 6.0), (3.0, 11.5)], PLAIN),
    "wide_narrow": (RADIAL, PLAIN + [(3, 5.0, 1, 2), (3, 8.0, -1, 1)]),
    "wide_wide": (RADIAL, PLAIN + [(9, 7.0, 1, 1), (9, 7.0, -1, 3)]),
}


def _model(d, radial, angular, structures):
    lines = []
    for ec in ("H", "O"):
        for e1 in ("H", "O"):
            lines += [f"symfunction_short {ec} 2 {e1} {eta} {rs} 12.0" for eta, rs in radial]
        for e1, e2 in PAIRS:
            lines += [f"symfunction_short {ec} {t} {e1} {e2} {eta} {lam} {zeta} 12.0" for t, eta, lam, zeta in angular]
    (d / "input.nn").write_text(water.input_nn_text(lines, nodes=(8, 8)))
    m = Mode(0)
    m.initialize()
    m.loadSettingsFile(str(d / "input.nn"))
    m.setupGeneric()
    m.setupSymmetryFunctionScalingNone()
    write_scaling(str(d / "scaling.data"), collect_statistics(m, structures))
    m.close()
    rng = np.random.default_rng(5)
    for z in (1, 8):
        water.write_weights(str(d / f"weights.{z:03d}.data"), water.random_weights([len(lines) // 2, 8, 8, 1], rng))
    return str(d)


@pytest.mark.parametrize("form", FORMS)
def test_range(form, tmp_path):
    from oracle import port
    structures = [water.water_box(33, seed=1, sigma=0.08), water.water_box(40, seed=2, sigma=0.08)]
    d = _model(tmp_path, *FORMS[form], structures)
    ref = [port.PortModel(d).evaluate(s) for s in structures]
    m = H.gpu_mode(d)
    b = m.batch(structures)
    b.setPositions(np.concatenate([s.positions for s in structures]))
    for store in (False, True):
        b.evaluate(forces=True, storeDGdr=store, graph=False)
        E, F, a = b.energies(), b.forces(), 0
        for k, r in enumerate(ref):
            f = F[a:a + structures[k].numAtoms]
            a += structures[k].numAtoms
            assert abs(E[k] - r["energy"]) <= 1e-10 * abs(r["energy"]), (form, k)
            assert np.abs(f - r["forces"]).max() <= 1e-10 * np.abs(r["forces"]).max(), (form, k)
    assert "candidate_masks" not in dict(b.profileStages(forces=True))
