"""Per-atom results (symmetry functions, dE/dG) read back in pieces by several
threads equal those of the small batches that take the single copy, bit for
bit: elements with different numbers of functions (27 and 30), a batch of
several pieces per thread and one of just over the limit."""
import os

import numpy as np
import pytest

from n2p2_b200 import Structure, read_structures
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [3, 40])
def test_pieces_equal_single_copy(frames):
    d = os.path.join(H.GOLDEN, "examples", "H2O_RPBE-D3")
    f = read_structures(os.path.join(d, "input.data"))[0]
    rng = np.random.default_rng(1)
    kinds = [Structure(f.positions + rng.normal(scale=0.02, size=f.positions.shape), f.elements, box=f.box)
             for _ in range(3)]
    m = H.gpu_mode(d)

    def results(structs):
        b = m.batch(structs)
        b.setPositions(np.concatenate([s.positions for s in structs]))
        b.evaluate(forces=True)
        return b.symmetryFunctions(), b.dEdG()
    one = [results([k]) for k in kinds]
    G, D = results([kinds[k % 3] for k in range(frames)])
    assert G.size > 65536 and one[0][0].size < 65536
    assert np.array_equal(G, np.concatenate([one[k % 3][0] for k in range(frames)]))
    assert np.array_equal(D, np.concatenate([one[k % 3][1] for k in range(frames)]))
