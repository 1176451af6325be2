"""The list builds at the edges of their paths: the half list and the reverse index equal the oracle's, from the
automatic build and from the thread-per-particle one, and a batch replica's first forces equal the single system's."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ONeighbourList

pytestmark = pytest.mark.gpu

# (particles, box, cutoff, skin, spread beyond the box)
CASES = {
    "no cells, 2": (2, 8.0, 3.0, 0.2, 0.0),
    "no cells, 31": (31, 8.0, 3.0, 0.2, 0.0),
    "no cells, 33": (33, 8.0, 3.0, 0.2, 0.0),
    "no cells, 500": (500, 8.64, 3.0, 0.2, 0.0),
    "3 cells a side": (700, 9.6, 2.9, 0.3, 0.0),
    "4 cells a side, odd": (1201, 13.0, 2.9, 0.3, 0.0),
    "mostly empty cells": (200, 40.0, 2.5, 0.3, 0.0),
    "cells of more than 32": (3000, 9.0, 2.5, 0.3, 0.0),
    "more candidates than the shared memory holds": (9000, 9.0, 2.5, 0.3, 0.0),
    "positions outside the box": (1500, 12.0, 2.5, 0.3, 0.4),
    "wide grid": (40000, 42.0, 2.5, 0.3, 0.0),
}


@pytest.mark.parametrize("case", CASES)
def test_lists_equal_the_oracle(md, oracle, case):
    n, box, rc, skin, beyond = CASES[case]
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4))
    pos[:, :3] = rng.uniform(-beyond, box + beyond, size=(n, 3))
    os_ = oracle.system(pos, box)
    onl = ONeighbourList(oracle, rc, skin, reverse=True)
    onl.build(os_)
    want = onl.get(n)
    for variant in (-1, 0):
        s = md.System.from_arrays(pos, box)
        nl = md.NeighbourList(rc, skin, reverse_index=True)
        nl.set_build_variant(variant)
        nl.build(s)
        got = nl.download()
        for k in ("offsets", "neighbours", "rev_offsets", "rev_pairs"):
            assert np.array_equal(got[k], want[k]), (variant, k)


@pytest.mark.parametrize("precision", ["PREC_FP64", "PREC_FP32FX"])
@pytest.mark.parametrize("n", [33, 500, 1201])
def test_batch_replicas_equal_single_systems(md, precision, n):
    """Replicas with and without cells in one batch against the same systems alone: energies and forces"""
    from test_gpu_ordered import jittered

    prec = getattr(md, precision)
    systems = [(jittered(m, L, m + k), L, None, None) for k, (m, L) in enumerate([(n, 8.0), (300, 7.0), (n + 700, 13.0)])]
    b = md.Batch(systems, cutoff=2.5, skin=0.3, precision=prec, energy_every=1)
    pe, w, _, inside = b.energy()
    for r, (pos, box, _, _) in enumerate(systems):
        s = md.System.from_arrays(pos, box)
        nl = md.NeighbourList(2.5, 0.3, reverse_index=True)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, prec)
        assert ff.compute_forces(s, nl) == pe[r] and ff.virial == w[r] and ff.inside_pairs == inside[r]
        assert np.array_equal(b.download(r)["force"], s.forces())
