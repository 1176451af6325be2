"""Both sides of lines in the rules on size: FP64's threads per particle (4 up to 48,000) and the cells of which the graphs'
step kernel adds up the counts directly (up to 16,384)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [48000, 48001])
def test_fp64_lanes_agree_with_one_thread(md, n):
    box = (n / 0.8) ** (1.0 / 3.0)
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


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FX32"])
@pytest.mark.parametrize("n,cells", [(4000, 25), (4000, 26), (300000, 25), (300000, 26)])  # 15,625 and 17,576 cells
def test_graphs_equal_the_host_loop(md, n, cells, prec):
    box = 2.801 * cells
    vel = 2.5 * np.random.default_rng(n).standard_normal((3, n))
    out = []
    for chunk in (16, 0):
        s = md.System.from_arrays(jittered(n, box, n), box, vel=vel)
        s.set_graph(chunk)
        nl = md.NeighbourList(2.5, 0.3)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, getattr(md, prec))
        ff.compute_forces(s, nl)
        rec = md.VelocityVerletIntegrator(0.002).run(s, ff, nl, 48)
        info = s.graph_info()
        assert (info["launches"] == 3) == (chunk > 0) and info["recoveries"] == 0, info
        assert nl.rebuild_count > 3
        out.append((*rec, nl.rebuild_count, *(s.download()[k] for k in ("pos", "vel", "force", "ids"))))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
