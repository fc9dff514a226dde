"""The in-cell ordering of the search (k_cell_order) where its forms meet: grids
on both sides of the 2^18 cells at which a warp takes 16 instead of 8, with
neighbouring cells that hold up to 4, 8, 16 and 32 particles each (as many lanes
a cell), up to 128, and more (a lane a cell), and all of these among one
another.  Keys, order and bounds against the oracle's stable sort."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import copy_from_ptr, dev, par_dev, sync

pytestmark = pytest.mark.gpu

FILLS = {"one": (1,), "to 4": (0, 1, 2, 3, 4, 0, 0), "to 8": (0, 5, 8, 1), "to 16": (16, 9, 0, 3, 15),
         "to 32": (17, 32, 0, 31, 1), "to 128": (33, 0, 127, 128, 4), "more": (129, 0, 300, 141, 2, 700),
         "mixed": (4, 0, 17, 129, 1, 8, 64, 0, 0, 16, 5)}


@pytest.mark.parametrize("cells", [(6, 5, 40), (40, 40, 90)])
@pytest.mark.parametrize("fill", list(FILLS))
def test_cells_of_every_width_are_in_stable_order(lq, orc, cuda, fill, cells):
    from loquat_b200 import cases

    par = cases.small_column(nsx=4, nsy=4, nsz=4).par.copy()
    h2 = 2.0 * float(par.h)
    par.domain_size_x, par.domain_size_y, par.domain_size_z = ((k - 0.5) * h2 for k in cells)
    lq.initialize_parameters(par)
    assert (par.ncell > 1 << 18) == (cells[0] == 40)
    rng = np.random.default_rng(5)
    nz = par.cell_num_z
    pos = []
    for k in range(2 * nz):       # two whole columns of cells, at the far end
        n = FILLS[fill][k % len(FILLS[fill])]
        cell = (par.cell_num_x - 1, par.cell_num_y - 1 - k // nz, k % nz)
        pos.append((np.array(cell) + rng.uniform(0.2, 0.8, (n, 3))) * h2)
    pos = np.concatenate(pos)
    n = len(pos)
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = pos[rng.permutation(n)]
    par.np, par.npb, par.npm = n, n // 3, n - n // 3
    want = orc.grid_float(par, x, par.npb)
    g = lq.Grid(n, par.ncell)
    g.neighbor_search(par, par_dev(par), dev(x))
    sync()
    a = g.arrays()
    for name, m in (("part_cel", n), ("part_idx", n), ("cell_beg", par.ncell), ("cell_end", par.ncell)):
        assert np.array_equal(copy_from_ptr(a[name], m), want[name]), (fill, name)
    g.close()
