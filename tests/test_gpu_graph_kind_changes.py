"""A run whose cells thin out until the graphs' step kernel builds the list another way, with every chunk run again on the host
path in between (its builds measure the cells): the host loop's bits, and the next graphs have what the new kind needs"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_build_nonuniform import lattice, pos4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32FX"])
def test_full_cells_that_thin_out(md, prec):
    n, box, side = 8000, 36.5, 19.0
    p = lattice(n, (side, side, side), 1) + (box - side) / 2
    vel = (1.1 * (p - box / 2)).T.copy()  # homogeneous expansion
    out = []
    for chunk in (8, 0):
        s = md.System.from_arrays(pos4(p), box, vel=vel)
        s.set_graph(chunk, test_rerun=chunk > 0)
        nl = md.NeighbourList(2.5, 0.3)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, getattr(md, prec))
        ff.compute_forces(s, nl)
        vv = md.VelocityVerletIntegrator(0.003)
        rec = list(vv.run(s, ff, nl, 240))
        info = s.graph_info()
        assert (info["recoveries"] > 5) == (chunk > 0), info
        s.set_graph(chunk)
        rec += vv.run(s, ff, nl, 32)
        out.append((*rec, *(s.download()[k] for k in ("pos", "vel", "force", "ids"))))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    cells = np.minimum((out[0][6][:, :3] / box * 13).astype(int), 12)
    count = np.zeros((13, 13, 13), int)
    np.add.at(count, tuple(cells.T), 1)
    assert count.max() < 18  # thinned out
