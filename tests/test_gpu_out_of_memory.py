"""A call that runs out of device memory reports it and leaves nothing behind: the next calls work."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

from test_gpu_ordered import jittered

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def memory_left(nbytes: int):
    """The device with only nbytes free"""
    import torch

    torch.cuda.init()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - nbytes, dtype=torch.uint8, device="cuda")
    yield
    del hog
    torch.cuda.empty_cache()


def forces(md):
    box = 20.0
    s = md.System.from_arrays(jittered(6400, box, 1), box)
    nl = md.NeighbourList(2.5, 0.3)
    nl.build(s)
    ff = md.LennardJonesForceField(1.0, 1.0, 2.5)
    return ff.compute_forces(s, nl), s.forces()


def test_next_call_after_a_failed_allocation(md):
    want = forces(md)
    with memory_left(64 << 20):
        with pytest.raises(md.MDError, match="out of memory"):
            md.System(4_000_000, 100.0)
        with pytest.raises(md.MDError, match="out of memory"):
            md.Adjoint(np.zeros((1_000_000, 4)), 100.0, np.zeros((3, 1_000_000)))
    got = forces(md)
    assert got[0] == want[0] and np.array_equal(got[1], want[1])
