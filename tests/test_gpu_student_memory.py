"""A student benchmark gives its device memory back: two in a row, as the full
bench runs them, need no more than one."""
import gc
import os

import pytest

from n2p2_b200 import student
from tests import helpers as H

pytestmark = pytest.mark.gpu


def test_benchmark_releases_its_memory():
    torch = pytest.importorskip("torch")
    model = os.path.join(H.GOLDEN, "models", "student_water56")

    def free_after():
        out = student.benchmark(model, H.WATER56, num=24, steps=1, warmup=1)
        assert out["value"] > 0
        return torch.cuda.mem_get_info()[0]
    gc.collect()
    gc.disable()
    try:
        first = free_after()
        second = free_after()
    finally:
        gc.enable()
    assert first - second <= 64 << 20   # its batches hold about 0.5 GB
