"""List builds of cells that hold more than a warp's 32 particles (long cutoffs), at sizes where every candidate slot counts:
the rows of the cell build equal the thread-per-particle build's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(n: int, box: float, seed: int) -> np.ndarray:
    """n sites of a simple cubic lattice filling the box, each displaced by up to a twelfth of the spacing"""
    side = int(np.ceil((n - 1e-9) ** (1.0 / 3.0)))
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    g = g[rng.permutation(len(g))[:n]]
    pos = np.zeros((n, 4))
    pos[:, :3] = (g + 0.5 + rng.uniform(-1 / 12, 1 / 12, size=g.shape)) * (box / side)
    return pos


@pytest.mark.parametrize("n,rl", [(32000, 3.6), (200000, 4.0), (864000, 4.0), (500000, 4.5)])
def test_rows_equal_the_other_builds(md, n, rl):
    box = (n / 0.8442) ** (1.0 / 3.0)
    pos = lattice(n, box, n)
    lists = []
    for variant in (-1, 0):
        s = md.System.from_arrays(pos, box)
        nl = md.NeighbourList(rl - 0.3, 0.3, reverse_index=True)
        nl.set_build_variant(variant)
        nl.build(s)
        lists.append(nl.download())
    for k in ("offsets", "neighbours", "rev_offsets", "rev_pairs"):
        assert np.array_equal(lists[0][k], lists[1][k]), k
