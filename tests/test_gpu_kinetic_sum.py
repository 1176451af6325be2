"""Kinetic energies and the thermostats' factors at the block edges of their kernels (one block, several, and more than one
launch adds in order), against the reference's blocked serial sum evaluated with numpy: the same bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kinetic(vel, mass):
    """deterministicSum over 0.5 m v^2 (blocks of 1,024 added one after another, then the blocks)"""
    e = (0.5 * mass) * ((vel[0] * vel[0] + vel[1] * vel[1]) + vel[2] * vel[2])
    blocks = [np.cumsum(e[k:k + 1024])[-1] for k in range(0, len(e), 1024)]
    return float(np.cumsum(blocks)[-1])


@pytest.mark.parametrize("n", [2, 1023, 1024, 1025, 4097, 524288, 524289])
def test_kinetic_energy_and_rescale(md, n):
    rng = np.random.default_rng(n)
    box = float((n / 0.3) ** (1.0 / 3.0)) + 6.0
    pos = np.zeros((n, 4))
    pos[:, :3] = rng.uniform(0.0, box, size=(n, 3))
    vel, mass = rng.standard_normal((3, n)), rng.uniform(0.5, 2.0, n)
    s = md.System.from_arrays(pos, box, vel=vel, mass=mass)
    want = kinetic(vel, mass)
    assert s.kinetic_energy() == want
    assert s.kinetic_energy() == want  # the block count is back at zero
    s.rescale_velocities(1.7)
    vel = vel * np.sqrt(1.7 / ((2.0 * want) / (3.0 * n - 3.0)))
    assert np.array_equal(s.download()["vel"], vel)
    assert s.kinetic_energy() == kinetic(vel, mass)


@pytest.mark.parametrize("thermostat", ["rescale", "bussi"])
@pytest.mark.parametrize("n", [500, 1024, 2049])
def test_thermostatted_run_equals_steps(md, thermostat, n):
    """md_run's graphs (factor, scaling and record in the kinetic kernels) against the host loop without records"""
    from test_gpu_ordered import jittered

    box = max(6.0, (n / 0.8) ** (1.0 / 3.0))
    vel = np.random.default_rng(n).standard_normal((3, n))
    steps = 24
    r1 = np.random.default_rng(1).standard_normal(steps)
    chi2 = np.random.default_rng(2).chisquare(3 * n - 4, steps)
    out = []
    for chunk, record in ((16, True), (0, True), (0, False)):
        s = md.System.from_arrays(jittered(n, box, n), box, vel=vel)
        s.set_graph(chunk)
        nl = md.NeighbourList(2.5, 0.3)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, md.PREC_FP64)
        ff.compute_forces(s, nl)
        pe, ke, w = md.VelocityVerletIntegrator(0.002).run(
            s, ff, nl, steps, thermostat=thermostat, rescale_every=3, rescale_temperature=1.1, bussi_temperature=1.1,
            bussi_tau=0.2, bussi_r1=r1, bussi_chi2=chi2, record=record)
        out.append((ke, s.download()))
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][0][-1] == kinetic(out[0][1]["vel"], np.ones(n))
    for other in out[1:]:
        for k in ("pos", "vel", "force"):
            assert np.array_equal(out[0][1][k], other[1][k]), k
