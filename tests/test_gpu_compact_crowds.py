"""The block shapes of the staged compact kernels in large batches: an atom
gets one warp up to 64 neighbours (32 in the weighted types) where no atom of
the batch has more and the batch fills the SMs with one-warp blocks, up to 20
elsewhere, and four warps above.  A cluster around each limit has the same
symmetry functions and forces alone, in a crowd of small molecules and in one
that holds a larger structure too.

The shapes differ in the order of sums of at most P = 65 64 / 2 terms (symmetry
functions: none negative), so a function differs by at most 2 P eps of its
unscaled value, 9.3e-13; forces by the other parity tests' 1e-10 of the largest
component."""
import os

import numpy as np
import pytest

from n2p2_b200 import Structure, read_structures
from tests import helpers as H

pytestmark = pytest.mark.gpu

MODELS = {"wide": ("examples", "Anisole_SCAN"), "narrow": ("models", "scan_narrow"), "weighted": ("models", "qm9_weighted")}


def _cluster(frame, atoms):
    near = np.argsort(np.linalg.norm(frame.positions - frame.positions.mean(0), axis=1))[:atoms]
    return Structure(frame.positions[near], [frame.elements[k] for k in near])


def _frame(model, d):
    s = read_structures(os.path.join(d, "input.data"))
    if model != "weighted":
        return s[0]
    x, e = [], []   # molecules on a grid of 7 bohr: up to 80 atoms within the cutoff
    for k, m in enumerate(s[:12]):
        x.append(m.positions - m.positions.mean(0) + 7.0 * np.array([k % 2, k // 2 % 2, k // 4]))
        e += list(m.elements)
    return Structure(np.concatenate(x), e)


@pytest.mark.parametrize("atoms", [20, 21, 22, 32, 33, 34, 64, 65, 66])
@pytest.mark.parametrize("model", MODELS)
def test_cluster_in_a_crowd(model, atoms):
    d = os.path.join(H.GOLDEN, *MODELS[model])
    frame = _frame(model, d)
    s = _cluster(frame, atoms)
    assert s.numAtoms == atoms
    crowd = [_cluster(frame, 12)] * 150
    assert atoms + 12 * 150 >= 12 * 148   # 12 one-warp blocks on each of the 148 SMs
    m = H.gpu_mode(d)

    def run(structs):
        b = H.gpu_batch(m, structs)
        n = s.numAtoms
        k = sum(m.numSymmetryFunctions(e) for e in b.elements[:n])
        G = H.unscaled_from_files(d, s, b.symmetryFunctions()[:k])
        return G, b.forces()[:n], int(np.diff(b.neighbors()["offset"])[:n].max())
    G, F, most = run([s])
    assert most > 0
    for others in (crowd, crowd + [_cluster(frame, 80)]):
        g, f, _ = run([s] + others)
        assert np.all(np.abs(g - G) <= 9.3e-13 * np.maximum(np.abs(G), 1e-3 * np.abs(G).max()))
        assert np.abs(f - F).max() <= 1e-10 * np.abs(F).max()
