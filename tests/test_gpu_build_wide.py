"""Lists of long rows (18 to 24 words of candidates a cell): the build that writes 24 words at a time, from the list build,
from md_run's graphs and from the batch engine."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ONeighbourList
from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_cell", [26.0, 28.5, 34.0])
def test_lists_equal_the_oracle(md, oracle, per_cell):
    box = 13.1 * 3.2
    n = int(per_cell * 13 ** 3) + 1
    pos = np.zeros((n, 4))
    pos[:, :3] = np.random.default_rng(n).uniform(0.0, box, size=(n, 3))
    os_ = oracle.system(pos, box)
    onl = ONeighbourList(oracle, 3.0, 0.2, reverse=True)
    onl.build(os_)
    want = onl.get(n)
    s = md.System.from_arrays(pos, box)
    nl = md.NeighbourList(3.0, 0.2, reverse_index=True)
    nl.build(s)
    got = nl.download()
    for k in ("offsets", "neighbours", "rev_offsets", "rev_pairs"):
        assert np.array_equal(got[k], want[k]), k


def test_graph_run_equals_host_loop(md):
    n, box = 61000, 41.8
    vel = np.random.default_rng(3).standard_normal((3, n)) * 1.3
    out = []
    for chunk in (16, 0):
        s = md.System.from_arrays(jittered(n, box, 3), box, vel=vel)
        s.set_graph(chunk)
        nl = md.NeighbourList(3.0, 0.2)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 3.0, md.PREC_FP32FX)
        ff.compute_forces(s, nl)
        pe = md.VelocityVerletIntegrator(0.004).run(s, ff, nl, 40)[0]
        out.append((pe, s.download(), nl.rebuild_count))
    assert out[0][2] == out[1][2] > 2
    assert np.array_equal(out[0][0], out[1][0])
    for k in ("pos", "vel", "force", "ids"):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k


def test_batch_replicas_equal_single_systems(md):
    systems = [(jittered(n, L, n), L, None, None) for n, L in ((1800, 12.9), (5500, 19.3))]  # 4 and 6 cells a side
    b = md.Batch(systems, cutoff=3.0, skin=0.2, precision=md.PREC_FP32FX)
    pe = b.energy()[0]
    for r, (pos, box, _, _) in enumerate(systems):
        s = md.System.from_arrays(pos, box)
        nl = md.NeighbourList(3.0, 0.2)
        nl.build(s)
        assert md.LennardJonesForceField(1.0, 1.0, 3.0, md.PREC_FP32FX).compute_forces(s, nl) == pe[r]
        assert np.array_equal(b.download(r)["force"], s.forces())
