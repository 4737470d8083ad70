"""A first-tier shape that was measured on another batch of the same class
gives way to the smallest one that holds the batch's largest neighbour count
(one atom beyond the stage costs the next tier's kernel); the same when new
positions outgrow it.  Results do not depend on the shape."""
import json

import numpy as np
import pytest

from n2p2_b200 import Structure, water
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _most(b):
    return int(np.diff(b.neighbors()["offset"]).max())


def _smallest_from_cache(b, path):
    """A cache entry for the batch's class that says 128, 128, read back by the tuner."""
    b.autotune(useCache=True)
    cache = json.load(open(path))
    for entry in cache.values():
        entry["values"] = entry["forces"] = 0
    path.write_text("{\n" + ",\n".join(f'  "{k}": {json.dumps(v)}' for k, v in cache.items()) + "\n}\n")
    r = b.autotune(useCache=True)
    assert r["from_cache"]
    return r["values"], r["forces"]


@pytest.mark.parametrize("scale,shape", [(1.0, 0), (0.95, 1), (0.9, 2), (0.8, 0)])
def test_cached_shape_fits_the_batch(scale, shape, tmp_path, monkeypatch):
    monkeypatch.setenv("N2P2_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    m = H.gpu_mode(H.WATER40)
    s = water.water_box(110, seed=3, sigma=0.1)
    s = Structure(s.positions * scale, s.elements, box=s.box * scale)
    b = H.gpu_batch(m, [s])
    low, high = {0: (0, 128), 1: (129, 160), 2: (161, 192)}[shape] if scale > 0.85 else (193, 384)
    assert low <= _most(b) <= high
    assert _smallest_from_cache(b, tmp_path / "tune.json") == (shape, shape)


def test_positions_that_outgrow_the_shape(monkeypatch, tmp_path):
    monkeypatch.setenv("N2P2_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    m = H.gpu_mode(H.WATER40)
    s = water.water_box(110, seed=3, sigma=0.05)
    near = s.positions - s.box.sum(axis=0) / 2
    r = np.linalg.norm(near, axis=1)
    dense = s.positions.copy()   # atoms around the centre drawn in
    dense[r < 12.0] -= 0.25 * near[r < 12.0]
    b = H.gpu_batch(m, [s])
    assert _smallest_from_cache(b, tmp_path / "tune.json") == (0, 0)
    b.evaluate()
    assert _most(b) <= 128
    b.setPositions(dense)
    for _ in range(3):   # with the old shape, then with the one that holds them
        b.evaluate()
        E, F = b.energies(), b.forces()
    assert 128 < _most(b) <= 160
    fresh = H.gpu_batch(m, [Structure(dense, s.elements, box=s.box)])
    assert np.array_equal(E, fresh.energies()) and np.array_equal(F, fresh.forces())
