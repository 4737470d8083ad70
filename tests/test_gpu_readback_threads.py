"""Symmetry functions and dE/dG of one evaluated batch read by several host
threads at once (the library calls release the interpreter lock) equal what
one thread reads, bit for bit; the batch is large enough for the copy in
pieces through the batch's staging."""
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from n2p2_b200 import Structure, read_structures
from tests import helpers as H

pytestmark = pytest.mark.gpu


def test_two_threads_read_one_batch():
    d = os.path.join(H.GOLDEN, "examples", "H2O_RPBE-D3")
    f = read_structures(os.path.join(d, "input.data"))[0]
    rng = np.random.default_rng(2)
    structs = [Structure(f.positions + rng.normal(scale=0.02, size=f.positions.shape), f.elements, box=f.box)
               for _ in range(40)]
    m = H.gpu_mode(d)

    def batch():
        b = m.batch(structs)
        b.setPositions(np.concatenate([s.positions for s in structs]))
        b.evaluate(forces=True)
        return b
    alone = batch()
    G, D = alone.symmetryFunctions(), alone.dEdG()
    assert G.size > 16 * 65536
    b = batch()
    with ThreadPoolExecutor(4) as pool:   # the first reads allocate the staging
        for _ in range(10):
            reads = [pool.submit(b.symmetryFunctions if k % 2 else b.dEdG) for k in range(4)]
            for k, r in enumerate(reads):
                assert np.array_equal(r.result(), G if k % 2 else D)
