"""MD_PREC_FP64's branch-free force kernels (variant 2) over the sizes where their shape changes: the branchy kernel's
(variant 0) forces, energies and inside count bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 31, 500, 2047, 8192, 8193, 24576, 24577, 72000, 72001, 118001])
def test_fp64_variants_agree(md, n):
    box = max(6.0, (n / 0.8) ** (1.0 / 3.0))
    s = md.System.from_arrays(jittered(n, box, n), box)
    ff = md.LennardJonesForceField(1.0, 1.0, 2.5)
    nl = md.NeighbourList(2.5, 0.3, reverse_index=True)
    nl.build(s)
    got = {}
    for v in (0, 2):
        nl.set_force_variant(md.PREC_FP64, v)
        pe = ff.compute_forces(s, nl)
        assert nl.force_variant(md.PREC_FP64) == v
        got[v] = (pe, ff.virial, ff.inside_pairs, s.forces())
    assert got[0][:3] == got[2][:3]
    assert np.array_equal(got[0][3], got[2][3])
