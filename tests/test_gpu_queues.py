"""Kernels that hand work on through queues.

* Model 3: the particles whose first trial sub-step fails, through the queue,
  against the oracle, for the smallest and the default cap of sub-steps and
  particle counts that end inside a warp.  Bounds: those of ten steps in
  test_gpu_vw; a particle whose error estimate lies at the tolerance (1e-5)
  may take another number of sub-steps, which changes it by no more.
* Drop-in Adami and stress filter on a caller's grid whose cells do not
  follow one another in the slots (each cell's particles are contiguous,
  the cells in any order) against the oracle on the same grid, with
  test_gpu_operators' bounds."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import dev, host, par_dev, rel_l2, sorted_state, sync, zeros
from test_gpu_operators import TOL_ADAMI, TOL_SHEPARD
from test_gpu_vw import TOL_VW, pair, vw_errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 2, 3, 64])
@pytest.mark.parametrize("size,mixed", [((3, 3, 3), False), ((17, 5, 9), True)])
def test_queued_substeps_vs_oracle(lq, orc, cuda, size, mixed, cap):
    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, model=3, velocity_noise=0.05, seed=61,
                           vw=cases.vw_row(tol=1e-5, max_substeps=cap)).with_ids()
    sim, osim = pair(lq, orc, c, mixed)
    sim.step(3)
    osim.step(3)
    e = vw_errors(sim.download(), osim.get(), c.par.npb)
    for k, tol in TOL_VW[10].items():
        assert e[k] < tol, (k, e)
    assert not sim.health().any()


@pytest.mark.parametrize("size", [(2, 1, 2), (9, 5, 7), (16, 6, 12)])
def test_cells_in_any_order_vs_oracle(lq, orc, cuda, size):
    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, velocity_noise=0.05, seed=62)
    par = c.par
    g, st = sorted_state(orc, c)
    rng = np.random.default_rng(63)
    st[3][par.npb:] += (1e2 * rng.standard_normal((par.npm, 6))).astype(np.float32)
    beg, end = np.array(g["cell_beg"]), np.array(g["cell_end"])
    full = np.flatnonzero((beg >= par.npb) & (end > beg))
    slots, at = [], par.npb
    for cell in rng.permutation(full):
        b, e = beg[cell], end[cell]
        slots.append(np.arange(b, e))
        beg[cell], end[cell] = at, at + (e - b)
        at += e - b
    assert at == par.np
    order = np.concatenate([np.arange(par.npb)] + slots)
    st = [np.ascontiguousarray(a[order]) for a in st]
    pd, x, v, b, e = par_dev(par), dev(st[0]), dev(st[1]), dev(beg), dev(end)
    s_a, s_f, cache = dev(st[3]), dev(st[3]), zeros((par.np, 6))
    lq.adami_boundary(par, pd, x, v, s_a, b, e)
    lq.stress_regularization(par, pd, x, v, s_f, cache, b, e)
    sync()
    want = orc.adami(par, st[0], st[1], st[3], beg, end)
    assert rel_l2(host(s_a)[: par.npb], want[: par.npb]) < TOL_ADAMI
    want = orc.shepard(par, st[0], st[1], st[3], beg, end)
    assert rel_l2(host(s_f)[par.npb:], want[par.npb:]) < TOL_SHEPARD
