"""All-pairs forces of a few particles (one launch up to 32): the oracle's bits on both sides of the line"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import MODE_ALL_PAIRS, OForceField
from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 16, 31, 32, 33])
@pytest.mark.parametrize("box,rc", [(6.0, 3.0), (6.0, 1.1), (40.0, 2.5)])
def test_few_particles_match_the_oracle(md, oracle, n, box, rc):
    pos = jittered(n, 6.0, n)
    s = md.System.from_arrays(pos, box)
    ff = md.LennardJonesForceField(1.0, 1.0, rc)
    os_, off = oracle.system(pos, box), OForceField(oracle, 1.0, 1.0, rc)
    for _ in range(2):
        pe = ff.compute_forces(s)
        assert pe == off.forces(os_, None, MODE_ALL_PAIRS)
        assert ff.virial == off.virial and ff.inside_pairs == off.inside
        assert np.array_equal(s.forces(), os_.state().force)
