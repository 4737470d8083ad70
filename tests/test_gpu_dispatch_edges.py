"""Both sides of the limits that send few atoms (or a structure of many) to
another kernel: neighbour search of up to 512 atoms and reverse entries of up
to 2,048 by blocks per atom; energy of a structure of more than 4,096 atoms by
its block.  Lists and forces of a structure have the same bits in every batch;
an energy is the sum of its atoms' to the rounding of a sum in any order, n eps
times the sum of their sizes."""
import math

import numpy as np
import pytest

from n2p2_b200 import Structure, water
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _batch(total):
    """Water boxes of 96 atoms, molecules of 3 and a cluster of the remainder."""
    box = [water.water_box(32, seed=k, sigma=0.08) for k in range(3)]
    molecule = [Structure(box[0].positions[k:k + 3], box[0].elements[k:k + 3]) for k in range(0, 96, 3)]
    out = [box[k % 3] for k in range((total - 8) // 96)]
    left = total - 96 * len(out)
    while left > 5:
        out.append(molecule[left % 32])
        left -= 3
    b = box[1]
    return out + ([Structure(b.positions[:left], b.elements[:left])] if left else [])


@pytest.mark.parametrize("total", [511, 512, 513, 2047, 2048, 2049])
def test_lists_and_forces_around_the_limits(total):
    structs = _batch(total)
    m = H.gpu_mode(H.WATER40)
    b = H.gpu_batch(m, structs)
    assert b.numAtoms == total
    b.evaluate(forces=True)   # the second search: into the stride of the first
    nb, F, off, a = b.neighbors(), b.forces(), None, 0
    alone = {}
    for s in structs:
        if id(s) not in alone:
            x = H.gpu_batch(m, [s])
            alone[id(s)] = (x.neighbors(), x.forces())
        ref, f = alone[id(s)]
        got = H.split_neighbors(nb, a, a + s.numAtoms)
        for k in ("offset", "index", "d", "dr"):
            assert np.array_equal(got[k], ref[k]), (total, a, k)
        assert np.array_equal(F[a:a + s.numAtoms], f)
        a += s.numAtoms


@pytest.mark.parametrize("atoms", [4095, 4096, 4097, 4352])
def test_energy_sum_around_the_limit(atoms):
    big = water.water_box(1500, seed=4, sigma=0.08)
    s = Structure(big.positions[:atoms], big.elements[:atoms], box=big.box)
    small = water.water_box(32, seed=1)
    b = H.gpu_batch(H.gpu_mode(H.WATER40), [small, s, small, s])
    E, e, a = b.energies(), b.atomicEnergies(), 0
    for k, n in enumerate((small.numAtoms, atoms, small.numAtoms, atoms)):
        own = e[a:a + n]
        a += n
        assert abs(E[k] - math.fsum(own)) <= n * np.finfo(float).eps * np.abs(own).sum()
    assert E[1] == E[3] and E[0] == E[2]
