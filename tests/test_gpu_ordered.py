"""The serial sums computed in parallel (md_ordered.cuh): every result equals the one-after-another sum bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import MODE_ALL_PAIRS, OForceField

pytestmark = pytest.mark.gpu


def jittered(n: int, box: float, seed: int) -> np.ndarray:
    """n sites of a simple cubic lattice filling the box, each displaced by up to a sixth of the spacing"""
    side = int(np.ceil(n ** (1.0 / 3.0)))
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    g = g[np.sort(rng.permutation(len(g))[:n])]
    pos = np.zeros((n, 4))
    pos[:, :3] = (g + 0.5 + rng.uniform(-1 / 6, 1 / 6, size=g.shape)) * (box / side)
    return pos


@pytest.mark.parametrize("n,box,rc", [(1, 6.0, 2.5), (2, 6.0, 2.5), (31, 6.0, 3.0), (33, 6.0, 2.5), (129, 6.0, 3.0),
                                      (1025, 11.0, 2.5), (4097, 17.0, 2.5),
                                      (8100, 20.0, 10.0)])  # the last: more pairs than one pass of records holds
def test_all_pairs_sums_bit_exact(md, oracle, n, box, rc):
    pos = jittered(n, box, n)
    s = md.System.from_arrays(pos, box)
    ff = md.LennardJonesForceField(1.0, 1.0, rc)
    pe = ff.compute_forces(s)
    os_, off = oracle.system(pos, box), OForceField(oracle, 1.0, 1.0, rc)
    assert pe == off.forces(os_, None, MODE_ALL_PAIRS)
    assert ff.virial == off.virial and ff.inside_pairs == off.inside
    assert n < 8100 or ff.inside_pairs > 1 << 24
    assert np.array_equal(s.forces(), os_.state().force)
