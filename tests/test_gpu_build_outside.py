"""Lists of positions outside the box, where a particle's cell is the clamped one: the oracle's rows, also with 3 cells a
side, where the frames of neighbouring cells do not always name a pair's nearest image."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ONeighbourList

pytestmark = pytest.mark.gpu

KEYS = ("offsets", "neighbours", "rev_offsets", "rev_pairs")


def check(md, oracle, pos, box, rc=2.5, skin=0.3):
    n = len(pos)
    onl = ONeighbourList(oracle, rc, skin, reverse=True)
    onl.build(oracle.system(pos, box))
    want = onl.get(n)
    for variant in (-1, 0):
        s = md.System.from_arrays(pos, box)
        nl = md.NeighbourList(rc, skin, reverse_index=True)
        nl.set_build_variant(variant)
        nl.build(s)
        got = nl.download()
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), (variant, k)


def test_one_pair_across_the_box(md, oracle):
    """The pair's frames are 5.91 apart, its nearest images 2.59"""
    pos = np.zeros((2, 4))
    pos[:, :3] = [[2.843, 4.25, 4.25], [8.75, 4.25, 4.25]]
    check(md, oracle, pos, 8.5)


# 8.4: cells of exactly r_l; 9.6, 10.0: 3 cells a side; 12.0: 4
@pytest.mark.parametrize("box", [8.4, 8.5, 9.6, 12.0])
@pytest.mark.parametrize("beyond", [0.0, 1e-7, 1e-3, 0.4, 2.0])
def test_outside_positions(md, oracle, box, beyond):
    n = 900
    rng = np.random.default_rng(int(1e4 * box + 1e8 * beyond))
    pos = np.zeros((n, 4))
    pos[:, :3] = rng.uniform(0.0, box, size=(n, 3))
    # a fifth of the coordinates at or just past either face
    at = rng.random((n, 3)) < 0.2
    edge = np.where(rng.random((n, 3)) < 0.5, box + rng.uniform(0, 1, (n, 3)) * beyond, -rng.uniform(0, 1, (n, 3)) * beyond)
    pos[:, :3] = np.where(at, edge, pos[:, :3])
    check(md, oracle, pos, box)


def test_batch_replica_with_outside_positions(md):
    """A batch's first list against the single system's, by the forces and energies it gives"""
    rng = np.random.default_rng(5)
    systems = []
    for box in (8.5, 12.0):
        n = int(0.5 * box ** 3)
        side = int(np.ceil(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        pos = np.zeros((n, 4))
        pos[:, :3] = (g + 0.5 + rng.uniform(-0.1, 0.1, g.shape)) * (box / side)
        pos[:, 0] += np.where(pos[:, 0] < 0.6, box, 0.0)  # the same sites, named past the upper face
        systems.append((pos, box, None, None))
    pe, w, _, inside = md.Batch(systems, cutoff=2.5, skin=0.3, precision=md.PREC_FP64, energy_every=1).energy()
    for r, (pos, box, _, _) in enumerate(systems):
        s = md.System.from_arrays(pos, box)
        nl = md.NeighbourList(2.5, 0.3)
        nl.set_build_variant(0)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5)
        assert (ff.compute_forces(s, nl), ff.virial, ff.inside_pairs) == (pe[r], w[r], inside[r])
