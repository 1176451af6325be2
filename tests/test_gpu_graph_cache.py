"""The graphs a system keeps: md_run_prepare captures each kind of chunk once, and the run launches those."""
from __future__ import annotations

import pytest

from test_gpu_graph import make, start

pytestmark = pytest.mark.gpu


# three chunks: MD_PREC_FP64's are alike; the float modes' first begins with its own drift and the last ends without one
@pytest.mark.parametrize("prec,kinds", [("PREC_FP64", 1), ("PREC_FX32", 3), ("PREC_FP32FX", 3)])
def test_prepared_graphs_are_the_ones_launched(md, prec, kinds):
    st, box = start(md)
    s, nl, ff = make(md, st, box, getattr(md, prec))
    s.set_graph(16)
    integ = md.VelocityVerletIntegrator(0.005)
    integ.prepare(s, ff, nl, 48)
    assert s.graph_info()["graphs"] == kinds
    integ.run(s, ff, nl, 48)
    info = s.graph_info()
    assert info["graphs"] == kinds and info["launches"] == 3, info
