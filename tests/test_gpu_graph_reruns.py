"""Chunks of md_run's graphs that run again on the host path: everything a chunk restores is what it started from."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_graph import make, start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32FX"])
def test_histogram_of_chunks_without_samples(md, prec):
    """A g(r) sample every 40 steps and chunks of 16: most chunks that run again take none."""
    p = getattr(md, prec)
    st, box = start(md, temperature=1.5)
    out = []
    for chunk, rerun in ((16, True), (0, False)):
        s, nl, ff = make(md, st, box, p)
        s.set_graph(chunk, test_rerun=rerun)
        rdf = md.RadialDistribution(2.5, 50)
        md.VelocityVerletIntegrator(0.005).run(s, ff, nl, 160, rdf=rdf, rdf_every=40)
        out.append((rdf.histogram(), rdf.values(), s.download(), s.graph_info()))
    (ha, ga, sa, ia), (hb, gb, sb, _) = out
    assert ia["recoveries"] > 3, ia
    assert np.array_equal(ha, hb) and hb.sum() > 0
    assert np.array_equal(ga, gb)
    assert np.array_equal(sa["pos"], sb["pos"])
