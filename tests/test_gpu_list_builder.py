"""The list builder's chunks of 128 joined candidates: its entries against a
brute-force count of the pairs within the cut-off, for cases whose warps
span several columns, whose stencils are cut by the lattice's edges, and
whose runs end inside a chunk."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,hdr", [((1, 1, 5), 1.2), ((5, 3, 2), 1.2), ((2, 9, 31), 1.3), ((40, 3, 3), 1.0),
                                      ((12, 11, 13), 1.5)])
@pytest.mark.parametrize("skin", [0.0, 0.05])
def test_list_entries_are_the_pairs_within_the_cut_off(lq, cuda, size, hdr, skin):
    """neighbor_entries counts a target's own slot too.  With a skin, a pair
    beyond 2h that lies two columns apart is not listed; pairs within a
    float rounding of the cut-off may fall on either side."""
    from scipy.spatial import cKDTree

    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, hdr=hdr, seed=93, jitter_frac=0.1)
    s = lq.Simulation(c.par, *c.arrays())
    s.set_skin(skin)
    s.step(1)
    material, boundary = s.neighbor_entries()
    # the lists were built at the initial positions
    x, nb, h = c.pospres[:, :3].astype(np.float64), c.par.npb, float(c.par.h)
    col = np.floor(0.5 * c.pospres[:, :2] / np.float32(h)).astype(int)

    def count(targets, sources, cut):
        i, j = [], []
        for t, near in zip(targets, cKDTree(x[sources]).query_ball_point(x[targets], cut)):
            i += [t] * len(near)
            j += [sources[k] for k in near]
        i, j = np.array(i, int), np.array(j, int)
        return int(np.sum(np.all(np.abs(col[i] - col[j]) <= 1, axis=1)))

    assert not s.health().any()     # every particle lies in the lattice
    soil, wall, every = np.arange(nb, c.par.np), np.arange(nb), np.arange(c.par.np)
    cut = (2.0 + skin) * h
    for got, targets, sources in ((material, soil, every), (boundary, wall, soil)):
        low, high = count(targets, sources, cut * (1 - 2e-6)), count(targets, sources, cut * (1 + 2e-6))
        assert low <= got <= high, (got, low, high)
