"""The list build kernels on the kinds of cells that their rule sends them (few full cells, long cutoffs, nearly empty boxes), and
batches on both sides of their rule on thin replicas: the thread-per-particle build's rows, the single systems' trajectories."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_build_nonuniform import KEYS, droplet, pos4, rows, slab, uniform

pytestmark = pytest.mark.gpu

CASES = {
    "tiles, droplet": (lambda: droplet(40000), 5.2), "8 warps, small droplet": (lambda: droplet(20000), 5.2),
    "8 warps, slab": (lambda: slab(40000), 4.0), "8 warps, liquid": (lambda: uniform(60000, 0.85), 3.1),
    "4 warps, droplet": (lambda: droplet(60000), 2.5), "4 warps, slab": (lambda: slab(60000), 2.5),
    "warps and a list, nearly empty": (lambda: droplet(30000, 0.01), 4.0),
    "tiles, large and nearly empty": (lambda: droplet(200000, 0.01), 2.5),
}


@pytest.mark.parametrize("case", CASES)
def test_rows_equal_the_thread_build(md, case):
    make, rc = CASES[case]
    p, box = make()
    (got, layout), (want, _) = rows(md, p, box, rc, -1), rows(md, p, box, rc, 0)
    assert layout["use_tiles"]
    for k in KEYS:
        assert np.array_equal(got[k], want[k]), k


# particles a cell: 1.5 and 2.7 (threads), 3.4 (cells); droplets in much empty space (cells)
@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32FX"])
def test_batches_of_thin_replicas(md, prec):
    p = getattr(md, prec)
    cases = [uniform(2000, 0.06), uniform(2000, 0.1), uniform(2000, 0.14), droplet(1500, 0.05), droplet(900, 0.01)]
    vels = [1.3 * np.random.default_rng(k).standard_normal((3, len(q))) for k, (q, _) in enumerate(cases)]
    b = md.Batch([(pos4(q), L, v, None) for (q, L), v in zip(cases, vels)], cutoff=2.5, skin=0.3, dt=0.003, precision=p,
                 energy_every=20, chunk_steps=20)
    pe, w, ke = b.run(100)
    assert b.rebuilds().min() > 3
    for r, ((q, L), v) in enumerate(zip(cases, vels)):
        s = md.System.from_arrays(pos4(q), L, vel=v)
        nl = md.NeighbourList(2.5, 0.3)
        nl.set_build_variant(0)
        nl.build(s)
        ff = md.LennardJonesForceField(1.0, 1.0, 2.5, p)
        ff.compute_forces(s, nl)
        spe, ske, sw = md.VelocityVerletIntegrator(0.003).run(s, ff, nl, 100)
        assert np.array_equal(spe[19::20], pe[:, r]) and np.array_equal(sw[19::20], w[:, r]), r
        assert np.array_equal(s.positions(), b.download(r)["pos"]), r
