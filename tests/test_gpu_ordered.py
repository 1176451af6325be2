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


def serial(x: np.ndarray) -> float:
    """0.0 + x[0] + x[1] + ... one after another (numpy's cumulative sum is that loop)"""
    return float(np.cumsum(np.concatenate([[0.0], x]))[-1])


STREAMS = {
    "positive": lambda r, n: r.uniform(0.1, 2.0, n),
    "mixed signs": lambda r, n: r.standard_normal(n) * r.standard_normal(n) - 0.1,
    "walk": lambda r, n: r.standard_normal(n),  # crosses zero and binades again and again
    "halfway": lambda r, n: np.round(r.uniform(0, 1024, n)) / 2.0 ** 22 + 2.0 ** -30 * (r.integers(0, 2, n)),
    "scales": lambda r, n: np.ldexp(r.standard_normal(n), r.integers(-40, 40, n)),
    "mostly zero": lambda r, n: np.where(r.integers(0, 50, n) == 0, r.standard_normal(n), 0.0),
}


@pytest.mark.parametrize("kind", STREAMS)
@pytest.mark.parametrize("n", [1, 7, 8, 1023, 1025, 512 * 1024, 513 * 1024 + 1, 2200 * 1024 - 5])
def test_blocked_sum_bit_exact(md, kind, n):
    """The blocked kinetic-energy sum of any values (unit velocities, signed masses): 1,024 values at a time in order,
    then the block sums in order, as one chain up to 512 of them and through ordered_sum above"""
    x = STREAMS[kind](np.random.default_rng(n), n)
    vel = np.zeros((3, n))
    vel[0] = 1.0
    s = md.System.from_arrays(np.zeros((n, 4)), 10.0, vel=vel, mass=2.0 * x)
    blocks = np.array([serial(x[k:k + 1024]) for k in range(0, n, 1024)])
    assert s.kinetic_energy() == serial(blocks)
