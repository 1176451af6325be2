"""The fixed-point and float modes' force kernels over the sizes where their threads per particle change: variant 2's
bits equal the thread-per-particle variant 0's, and a run with the fused kicks and drift equals single steps."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["PREC_FP32FX", "PREC_FP32"])
@pytest.mark.parametrize("n", [700, 4096, 4097, 24576, 24577])
def test_variants_agree(md, precision, n):
    box = (n / 0.8) ** (1.0 / 3.0)
    prec = getattr(md, precision)
    s = md.System.from_arrays(jittered(n, box, n), box)
    ff = md.LennardJonesForceField(1.0, 1.0, 2.5, prec)
    nl = md.NeighbourList(2.5, 0.3)
    nl.build(s)
    got = []
    for v in (0, 2):
        nl.set_force_variant(prec, v)
        pe = ff.compute_forces(s, nl)
        got.append((pe, ff.virial, ff.inside_pairs, s.forces()))
    assert got[0][:3] == got[1][:3] and np.array_equal(got[0][3], got[1][3])


@pytest.mark.parametrize("precision", ["PREC_FP32FX", "PREC_FP32", "PREC_FX64", "PREC_FX32"])
@pytest.mark.parametrize("n", [33, 500, 4096, 4097])
def test_fused_run_equals_steps(md, precision, n):
    """20 steps of md_run (kick, drift, frames and half-skin test in the force kernel) against md_step_list"""
    box = max(6.0, (n / 0.8) ** (1.0 / 3.0))
    prec = getattr(md, precision)
    vel = np.random.default_rng(n).standard_normal((3, n))
    vv = md.VelocityVerletIntegrator(0.002)
    out = []
    for one_by_one in (False, True):
        s = md.System.from_arrays(jittered(n, box, n), box, vel=vel, mass=np.linspace(0.5, 2.0, n))
        nl = md.NeighbourList(2.5, 0.3)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, prec)
        ff.compute_forces(s, nl)
        if one_by_one:
            pe = np.array([vv.step(s, ff, nl) for _ in range(20)])
        else:
            pe = vv.run(s, ff, nl, 20)[0]
        out.append((pe, s.download(), nl.rebuild_count))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][2] == out[1][2]
    for k in ("pos", "vel", "force", "ids"):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k


@pytest.mark.parametrize("n,box,rc", [(2, 6.0, 2.5), (33, 6.0, 2.5), (500, 8.3, 2.5), (1100, 11.0, 4.0)])
def test_small_boxes_match_batch_replicas(md, n, box, rc):
    """Boxes without cells: 8 threads per particle against the batch engine's kernel for them (FP32FX)"""
    pos = jittered(n, box, n)
    s = md.System.from_arrays(pos, box)
    nl = md.NeighbourList(rc, 0.3)
    nl.build(s)
    ff = md.LennardJonesForceField(1.0, 1.0, rc, md.PREC_FP32FX)
    pe = ff.compute_forces(s, nl)
    b = md.Batch([(pos, box, None, None)], cutoff=rc, skin=0.3, precision=md.PREC_FP32FX)
    assert pe == b.energy()[0][0]
    assert np.array_equal(s.forces(), b.download(0)["force"])
