"""A caller's grid may mark an empty cell by equal bounds instead of -1 (the
reference's loops run from begin to end): interaction, boundary pass and stress
filter give the same bits with every mark."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import dev, host, par_dev, rel_l2, sorted_state, sync, zeros

pytestmark = pytest.mark.gpu


def rates_and_stresses(lq, par, st, beg, end):
    pd = par_dev(par)
    d = [dev(a) for a in st]
    rates = [zeros((par.np, 4)), zeros((par.np, 4)), zeros((par.np, 6))]
    b, e = dev(beg), dev(end)
    lq.particle_interaction(par, pd, *d, *rates, b, e)
    wall, filtered, cache = d[3].clone(), d[3].clone(), zeros((par.np, 6))
    lq.adami_boundary(par, pd, d[0], d[1], wall, b, e)
    lq.stress_regularization(par, pd, d[0], d[1], filtered, cache, b, e)
    sync()
    return [host(r)[par.npb:] for r in rates] + [host(wall), host(filtered)[par.npb:]]


@pytest.mark.parametrize("mark", ["zeros", "ends", "running"])
def test_empty_cells_by_equal_bounds(lq, orc, cuda, mark):
    c = cases.small_column(nsx=9, nsy=5, nsz=7, velocity_noise=0.05, seed=74)
    par = c.par
    g, st = sorted_state(orc, c)
    rng = np.random.default_rng(75)
    st[3][par.npb:] += (1e2 * rng.standard_normal((par.npm, 6))).astype(np.float32)
    beg, end = np.array(g["cell_beg"]), np.array(g["cell_end"])
    want = rates_and_stresses(lq, par, st, beg, end)
    empty = beg == -1
    if mark == "zeros":
        beg[empty] = end[empty] = 0
    elif mark == "ends":
        beg[empty] = end[empty] = par.np
    else:   # a plain exclusive scan of the counts
        counts = np.where(empty, 0, end - beg)
        end = np.cumsum(counts).astype(np.int32)
        beg = (end - counts).astype(np.int32)
    got = rates_and_stresses(lq, par, st, beg, end)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b), (mark, k, rel_l2(a, b))
