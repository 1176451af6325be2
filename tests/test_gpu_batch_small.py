"""Batches of small replicas (resorted by a block each) and of replicas one particle past that: trajectories, records and
rebuild counts equal the same systems run alone, with the energies of every step or some summed beside the next steps."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["PREC_FP64", "PREC_FP32FX"])
@pytest.mark.parametrize("most,every", [(500, 1), (1023, 3), (1024, 1), (1025, 1)])
def test_replicas_equal_single_runs(md, precision, most, every):
    prec, steps = getattr(md, precision), 60
    rng = np.random.default_rng(most)
    systems = []
    for n, density in ((most, 0.8), (2, 0.01), (33, 0.1), (300, 0.85), (257, 0.02)):
        box = max(6.0, (n / density) ** (1.0 / 3.0))
        systems.append((jittered(n, box, n), box, rng.standard_normal((3, n)) * 1.4, np.linspace(0.5, 2.0, n)))
    b = md.Batch(systems, cutoff=2.5, skin=0.2, dt=0.003, precision=prec, energy_every=every)
    pe, w, ke = b.run(steps)
    assert b.rebuilds().max() > 3
    for r, (pos, box, vel, mass) in enumerate(systems):
        s = md.System.from_arrays(pos, box, vel=vel, mass=mass)
        nl = md.NeighbourList(2.5, 0.2)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, prec)
        ff.compute_forces(s, nl)
        spe, ske, sw = md.VelocityVerletIntegrator(0.003).run(s, ff, nl, steps)
        assert np.array_equal(pe[:, r], spe[every - 1::every]), r
        assert np.array_equal(w[:, r], sw[every - 1::every]), r
        assert np.array_equal(ke[:, r], ske[every - 1::every]), r
        got, want = b.download(r), s.download()
        for k in ("pos", "vel", "force", "ids"):
            assert np.array_equal(got[k], want[k]), (r, k)
