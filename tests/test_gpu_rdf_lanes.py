"""g(r) histograms with several threads per particle, at rows of every remainder and particle counts around a block:
the counts equal numpy's over all pairs."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box", [(2, 6.0), (33, 6.0), (63, 6.5), (64, 6.5), (65, 6.5), (700, 9.6)])
def test_histogram_equals_numpy(md, n, box):
    pos = jittered(n, box, n)
    s = md.System.from_arrays(pos, box)
    nl = md.NeighbourList(2.5, 0.3)
    nl.build(s)
    rdf = md.RadialDistribution(2.5, 100)
    rdf.sample(s, nl)
    p = s.download()["pos"][:, :3]
    a, b = np.triu_indices(n, 1)
    d = p[a] - p[b]
    d -= box * np.rint(d / box)
    r2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    k = (np.sqrt(r2[r2 < 2.5 * 2.5]) / (2.5 / 100)).astype(np.int64)
    assert np.array_equal(rdf.histogram(), np.bincount(k[k < 100], minlength=100).astype(float))
