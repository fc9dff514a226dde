"""The in-cell ordering of the search (k_cell_order) where its forms meet:
cells of 1, 31, 32, 33, 127, 128, 129 and 300 particles in reversed, random
and sorted order, against the oracle's stable sort."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import copy_from_ptr, dev, par_dev, sync

pytestmark = pytest.mark.gpu

SIZES = (1, 0, 31, 32, 0, 33, 127, 128, 129, 300, 2)


@pytest.mark.parametrize("order", ["sorted", "reversed", "random"])
def test_cells_of_every_size_are_in_stable_order(lq, orc, cuda, order):
    from loquat_b200 import cases

    c = cases.small_column(nsx=16, nsy=6, nsz=12)
    par = c.par
    rng = np.random.default_rng(5)
    h2 = 2.0 * float(par.h)
    cells = [(k % par.cell_num_x, (k // 3) % par.cell_num_y, (2 * k) % par.cell_num_z) for k in range(len(SIZES))]
    pos = []
    for n, cell in zip(SIZES, cells):
        pos.append((np.array(cell) + rng.uniform(0.2, 0.8, (n, 3))) * h2)
    pos = np.concatenate(pos)
    n = len(pos)
    if order == "reversed":
        pos = pos[::-1]
    elif order == "random":
        pos = pos[rng.permutation(n)]
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = pos
    par = par.copy()
    par.np, par.npb, par.npm = n, n // 3, n - n // 3
    want = orc.grid_float(par, x, par.npb)
    g = lq.Grid(n, par.ncell)
    xd, pd = dev(x), par_dev(par)
    g.neighbor_search(par, pd, xd)
    sync()
    a = g.arrays()
    for name, m in (("part_cel", n), ("part_idx", n), ("cell_beg", par.ncell), ("cell_end", par.ncell)):
        assert np.array_equal(copy_from_ptr(a[name], m), want[name]), (order, name)
    g.close()
