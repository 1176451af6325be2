"""Chunks of md_run's graphs that run again on the host path: everything a chunk restores is what it started from."""
from __future__ import annotations

import threading
import time

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


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FX32"])
def test_step_kernel_that_gives_up(md, prec):
    """Barriers of a device rebuild that wait in vain end by themselves within a second; the run's bits are the host
    loop's, and the system's graphs work afterwards."""
    p = getattr(md, prec)
    st, box = start(md, cells=10, temperature=1.5)
    integ = md.VelocityVerletIntegrator(0.005)
    out = []
    for chunk in (16, 0):
        s, nl, ff = make(md, st, box, p)
        s.set_graph(chunk, test_give_up=chunk > 0)
        t = time.perf_counter()
        pe, ke, _ = integ.run(s, ff, nl, 48)
        seconds = time.perf_counter() - t
        given_up = s.graph_info()["recoveries"]
        assert (given_up > 0) == (chunk > 0)
        if given_up:
            print(f"{seconds / given_up:.2f} s for a chunk that gives up")
            assert seconds < 1.0 * given_up + 2.0
        s.set_graph(chunk)
        pe2, ke2, _ = integ.run(s, ff, nl, 48)
        assert s.graph_info()["recoveries"] == given_up
        out.append((pe, ke, pe2, ke2, *(s.download()[k] for k in ("pos", "vel", "force", "ids"))))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_two_threads_two_systems(md):
    """Two systems' graphs at once: each step kernel asks for every SM"""
    st, box = start(md, temperature=1.5)
    cases = [(md.PREC_FP64, 0.005), (md.PREC_FX32, 0.004)]

    def run(k, out):
        s, nl, ff = make(md, st, box, cases[k][0])
        for _ in range(4):
            pe, ke, _ = md.VelocityVerletIntegrator(cases[k][1]).run(s, ff, nl, 256)
        out[k] = (pe, ke, s.positions(), s.graph_info()["recoveries"])

    alone, together = [None, None], [None, None]
    for k in range(2):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, together)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert alone[k][3] == 0 and together[k][3] == 0
        for x, y in zip(alone[k][:3], together[k][:3]):
            assert np.array_equal(x, y)
