"""Thermostatted FP64 runs through md_run's graphs (the kinetic kernels scale, sum and record there) at the block edges of the
kinetic sum: the host loop's bits, with a partial chunk at the end."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_kinetic_sum import kinetic
from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thermostat", ["rescale", "bussi"])
@pytest.mark.parametrize("n", [500, 1023, 1024, 1025, 2049])
def test_graphs_equal_the_host_loop(md, thermostat, n):
    box, steps = max(8.5, (n / 0.8) ** (1.0 / 3.0)), 40
    vel = np.random.default_rng(n).standard_normal((3, n))
    r1 = np.random.default_rng(1).standard_normal(steps)
    chi2 = np.random.default_rng(2).chisquare(3 * n - 4, steps)
    out = []
    for chunk, record in ((16, True), (16, False), (0, True)):
        s = md.System.from_arrays(jittered(n, box, n), box, vel=vel)
        s.set_graph(chunk)
        nl = md.NeighbourList(2.5, 0.3)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, md.PREC_FP64)
        ff.compute_forces(s, nl)
        pe, ke, w = md.VelocityVerletIntegrator(0.002).run(
            s, ff, nl, steps, thermostat=thermostat, rescale_every=3, rescale_temperature=1.1, bussi_temperature=1.1,
            bussi_tau=0.2, bussi_r1=r1, bussi_chi2=chi2, record=record)
        info = s.graph_info()
        assert info["launches"] == (3 if chunk else 0) and info["recoveries"] == 0, info
        out.append((pe, ke, w, s.download()))
    graph, silent, host = out
    for k in range(3):
        assert np.array_equal(graph[k], host[k])
    assert graph[1][-1] == kinetic(graph[3]["vel"], np.ones(n))
    for other in (silent, host):
        for k in ("pos", "vel", "force", "ids"):
            assert np.array_equal(graph[3][k], other[3][k]), k
