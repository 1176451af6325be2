"""Steps of lists with 3 cells a side and more whose cells are too full for the shared-memory tiles (long cutoffs, dense
systems): the forces of every step belong to the step's positions."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_build_nonuniform import pos4, uniform

pytestmark = pytest.mark.gpu


def make(md, prec, n, density, rc):
    p, box = uniform(n, density)
    vel = 0.8 * np.random.default_rng(n).standard_normal((3, n))
    s = md.System.from_arrays(pos4(p), box, vel=vel)
    nl = md.NeighbourList(rc, 0.3)
    nl.build(s)
    layout = nl.layout()
    assert not layout["use_tiles"] and layout["segments_per_column"] >= 3
    ff = md.LennardJonesForceField(1.0, 1.0, rc, prec)
    ff.compute_forces(s, nl)
    return s, nl, ff


def by_id(s):
    d = s.download()
    o = np.argsort(d["ids"])
    return d["pos"][o, :3], d["vel"][:, o]


# 27 cells of 370 particles; 64 of 312
@pytest.mark.parametrize("n,density,rc", [(10000, 0.77, 6.5), (20000, 1.0, 5.5)])
@pytest.mark.parametrize("prec", ["PREC_FP32FX", "PREC_FP32", "PREC_FX32", "PREC_FX64"])
def test_steps_use_the_positions_they_reached(md, prec, n, density, rc):
    p = getattr(md, prec)
    vv = md.VelocityVerletIntegrator(0.002)
    s, nl, ff = make(md, p, n, density, rc)
    t, tl, tf = make(md, p, n, density, rc)
    r, rl, rf = make(md, md.PREC_FP64, n, density, rc)
    pe, _, _ = vv.run(s, ff, nl, 24)
    one_by_one = [vv.step(t, tf, tl) for _ in range(24)]
    want, _, _ = vv.run(r, rf, rl, 24)
    assert np.array_equal(pe, one_by_one)
    assert nl.rebuild_count == tl.rebuild_count == rl.rebuild_count
    # single-precision pair terms, 24 steps: the energies of 64-bit terms to about their own rounding
    assert np.abs(pe - want).max() < 1e-5 * np.abs(want).max()
    (xs, vs), (xr, vr) = by_id(s), by_id(r)
    d = xs - xr
    d -= s.box * np.round(d / s.box)
    assert np.abs(d).max() < 1e-4 and np.abs(vs - vr).max() < 1e-2
    f = s.forces()
    ff.compute_forces(s, nl)  # the same list, frames made from the positions
    assert np.array_equal(f, s.forces())
