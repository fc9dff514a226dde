"""Carried lists and the cut-off: interactions on one grid, at positions that
do not change, with another smoothing length than the call before.  The rates
against those from lists built afresh; the tolerance is that of the same pairs
in another order (test_gpu_identities.py)."""
from __future__ import annotations

import pytest

from loquat_b200 import cases
from helpers import dev, host, par_dev, rel_l2, sync

pytestmark = pytest.mark.gpu
TOL = 1e-4


@pytest.mark.parametrize("factor", [1.12, 0.9])
def test_other_smoothing_length_builds_other_lists(lq, cuda, factor):
    import torch

    from cuda.bindings import runtime as rt

    c = cases.small_column(velocity_noise=0.05, seed=72)
    n, nb = c.par.np, c.par.npb
    other = c.par.copy()
    other.hdr *= factor
    lq.initialize_parameters(other)
    grid = lq.Grid(n, max(c.par.ncell, other.ncell))
    state = [dev(a) for a in c.arrays()]
    f4, t2 = torch.empty_like(state[0]), torch.empty_like(state[3])
    rates = [torch.zeros(n, 4, device="cuda"), torch.zeros(n, 4, device="cuda"), torch.zeros(n, 6, device="cuda")]
    for par in (c.par, other):
        pd = par_dev(par)
        grid.neighbor_search(par, pd, state[0], state[2])
        for x in state:
            grid.sort_float4(n, x, f4) if x.shape[1] == 4 else grid.sort_tensor2d(n, x, t2)
        a = grid.arrays()
        lq.particle_interaction(par, pd, *state, *rates, a["cell_beg"], a["cell_end"])
    sync()
    got = [host(r)[nb:].copy() for r in rates]
    beg, end = (torch.empty(other.ncell, dtype=torch.int32, device="cuda") for _ in range(2))
    for src, dst in ((a["cell_beg"], beg), (a["cell_end"], end)):
        rt.cudaMemcpy(dst.data_ptr(), src, 4 * other.ncell, rt.cudaMemcpyKind.cudaMemcpyDeviceToDevice)
    lq.particle_interaction(other, pd, *state, *rates, beg, end)
    sync()
    grid.close()
    for g, r, name in zip(got, rates, ("acceleration", "spin", "strain rate")):
        assert rel_l2(g, host(r)[nb:]) < TOL, (factor, name, rel_l2(g, host(r)[nb:]))
