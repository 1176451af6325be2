"""MD_PREC_FP64 with the tile kernel pinned on lists without tiles: the other kernels' forces, energies and inside-cutoff
count, from the first force call on."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


def forces(md, s, nl):
    ff = md.LennardJonesForceField(1.0, 1.0, 2.5)
    out = []
    for _ in range(2):
        out.append((ff.compute_forces(s, nl), ff.virial, ff.inside_pairs))
    return out, s.forces()


def expect(md, pos, box):
    s = md.System.from_arrays(pos, box)
    nl = md.NeighbourList(2.5, 0.3)
    nl.set_force_variant(md.PREC_FP64, 0)
    nl.build(s)
    return forces(md, s, nl)


# a box under 3 cells per side; 3 cells of 27 too full for a tile
@pytest.mark.parametrize("n,box", [(500, 8.0), (9000, 9.0)])
def test_pinned_without_tiles(md, n, box):
    pos = jittered(n, box, n)
    s = md.System.from_arrays(pos, box)
    nl = md.NeighbourList(2.5, 0.3)
    nl.set_force_variant(md.PREC_FP64, 1)
    nl.build(s)
    assert not nl.layout()["use_tiles"]
    got, want = forces(md, s, nl), expect(md, pos, box)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])


def test_tiles_lost_at_a_rebuild(md):
    n, box = 9000, 30.0
    s = md.System.from_arrays(jittered(n, box, 1), box)
    nl = md.NeighbourList(2.5, 0.3)
    nl.set_force_variant(md.PREC_FP64, 1)
    nl.build(s)
    forces(md, s, nl)
    assert nl.layout()["use_tiles"] and nl.force_variant(md.PREC_FP64) == 1
    pos = jittered(n, 9.0, 2)
    s.upload(pos=pos)
    nl.build(s)
    assert not nl.layout()["use_tiles"]
    got = forces(md, s, nl)
    want = expect(md, pos, box)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
