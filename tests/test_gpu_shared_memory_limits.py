"""Systems whose long cutoffs need different amounts of shared memory from the same kernels, used in turn in one process."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


def make(md, box, rc, chunk):
    n = int(0.8 * box ** 3)
    s = md.System.from_arrays(jittered(n, box, 3), box, vel=np.random.default_rng(4).standard_normal((3, n)))
    s.set_graph(chunk)
    nl = md.NeighbourList(rc, 0.3)
    nl.build(s)
    ff = md.LennardJonesForceField(1.0, 1.0, rc, md.PREC_FP32FX)
    ff.compute_forces(s, nl)
    return s, ff, nl


def test_systems_of_different_cutoffs_in_turn(md):
    """The first system captures again after the second, which needs less, has captured the same step kernel"""
    out = []
    for chunk in (16, 0):
        a, b = make(md, 19.0, 4.4, chunk), make(md, 16.0, 3.6, chunk)
        pe = [md.VelocityVerletIntegrator(dt).run(*x, 32)[0]
              for dt, x in ((0.002, a), (0.002, b), (0.001, a), (0.001, b))]
        if chunk:
            assert a[0].graph_info()["launches"] == 4 and b[0].graph_info()["launches"] == 4
        out.append((np.concatenate(pe), a[0].positions(), b[0].positions()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
