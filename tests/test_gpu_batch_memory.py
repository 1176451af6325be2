"""An FP64 batch whose energy records do not fit the memory that is left: an error from the run, and nothing lost."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered
from test_gpu_out_of_memory import memory_left

pytestmark = pytest.mark.gpu


def make(md):
    n, box = 60000, 43.0
    rng = np.random.default_rng(2)
    systems = [(jittered(n, box, k), box, rng.standard_normal((3, n)), None) for k in range(4)]
    return md.Batch(systems, cutoff=2.5, skin=0.3, dt=0.002, precision=md.PREC_FP64, energy_every=1, chunk_steps=4)


def test_run_without_room_for_the_records(md):
    want = make(md)
    want_rec = want.run(4)
    b = make(md)
    with memory_left(64 << 20):  # the records take 123 MB
        with pytest.raises(md.MDError, match="out of memory"):
            b.run(4)
    launches = b.info()["launches"]
    for x, y in zip(b.run(4), want_rec):
        assert np.array_equal(x, y)
    assert np.array_equal(b.state_hashes(), want.state_hashes())
    assert b.info()["launches"] > launches
