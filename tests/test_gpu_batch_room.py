"""Batches whose cells outgrow the room that the list build first had for their candidates: more room where the shared memory
has it, captured once; where it has none, the graphs stay."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_build_nonuniform import droplet, pos4, uniform

pytestmark = pytest.mark.gpu


# r_l = 7.8 with 370 particles a cell: 8,000 candidates of which the shared memory holds about 3,500; a droplet in a large box
@pytest.mark.parametrize("system,rc,most", [(lambda: uniform(10000, 0.77), 7.5, 1), (lambda: droplet(3000, 0.02), 2.5, 2)])
def test_graphs_are_captured_once(md, system, rc, most):
    p, box = system()
    vel = 0.5 * np.random.default_rng(1).standard_normal((3, len(p)))
    b = md.Batch([(pos4(p), box, vel, None)], cutoff=rc, skin=0.3, dt=0.002, precision=md.PREC_FP32FX, chunk_steps=20)
    b.run(40)
    settled = b.graph_info()["captured"]
    b.run(160)
    info = b.graph_info()
    assert b.rebuilds().min() > 3
    assert info["captured"] - settled <= most, info
    s = md.System.from_arrays(pos4(p), box, vel=vel)
    nl = md.NeighbourList(rc, 0.3)
    nl.set_build_variant(0)
    nl.build(s)
    ff = md.LennardJonesForceField(1.0, 1.0, rc, md.PREC_FP32FX)
    ff.compute_forces(s, nl)
    md.VelocityVerletIntegrator(0.002).run(s, ff, nl, 200)
    assert np.array_equal(s.positions(), b.download(0)["pos"])
