"""The adjoint at the edges of its kernels' groups of threads: sizes that fill no whole warp or 1,024-particle block,
boxes without cells and cells of more than 32 particles, against the CPU adjoint bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import OAdjoint
from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,cutoff,skin", [(2, 6.0, 2.5, 0.3), (33, 6.0, 2.5, 0.3), (257, 7.0, 2.5, 0.3),
                                               (1025, 11.0, 2.5, 0.3), (1500, 12.2, 3.6, 0.4)])
def test_adjoint_sizes(md, oracle, n, box, cutoff, skin):
    pos = jittered(n, box, n)
    vel = np.random.default_rng(n).standard_normal((3, n))
    gpu = md.Adjoint(pos, box, vel, cutoff=cutoff, skin=skin, dt=0.002, steps=7, checkpoint_every=3)
    cpu = OAdjoint(oracle, pos, box, vel, rc=cutoff, skin=skin, dt=0.002, steps=7, every=3)
    mu, mp, u, w, k = gpu.forward(record=True)
    cu, cp, ou, ow, ok = cpu.forward()
    assert (mu, mp) == (cu, cp)
    assert np.array_equal(u, ou) and np.array_equal(w, ow) and np.array_equal(k, ok)
    for g in ((1.0, 0.0), (0.0, 1.0), (0.4, -0.9), (0.0, 0.0)):
        a, b = gpu.backward(*g), cpu.backward(*g)
        for key in ("d_epsilon", "d_sigma"):
            assert a[key] == b[key], (g, key)
        for key in ("d_pos", "d_vel"):
            assert np.array_equal(a[key], b[key]), (g, key)
