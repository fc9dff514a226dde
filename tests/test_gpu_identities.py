"""The particle identities of a drop-in grid, by which the interaction carries
its neighbour lists: a grid that is searched with fewer particles than it was
sized for, before or between searches over all of them, and a grid whose
first search runs on a stream that the default stream does not hold up.  The
rates from the carried lists (a build, then a reuse with other velocities)
against those from lists built afresh for copies of the grid's bounds.  Both
add the same pairs in another order: about 100 terms of unit roundoff 6e-8,
of which up to 16 times their sum's size cancels."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import dev, host, par_dev, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-4


def poison(nbytes):
    """Fills and frees device allocations of a size, so that the next ones
    of that size are likely to hold no zeros."""
    from cuda.bindings import runtime as rt

    held = []
    for _ in range(16):
        err, p = rt.cudaMalloc(nbytes)
        assert int(err) == 0
        rt.cudaMemset(p, 0x7F, nbytes)
        held.append(p)
    rt.cudaDeviceSynchronize()
    for p in held:
        rt.cudaFree(p)


@pytest.mark.parametrize("order", ["fewer first", "fewer between", "busy default stream"])
def test_carried_lists_after_the_identities_restart(lq, cuda, order):
    import torch

    from cuda.bindings import runtime as rt

    c = cases.small_column(velocity_noise=0.05, seed=71)
    par, n, nb = c.par, c.par.np, c.par.npb
    pd = par_dev(par)
    few = par.copy()
    few.np, few.npb, few.npm = nb // 2, nb // 2, 0
    pd_few = par_dev(few)
    lq.interaction_reserve(par)
    state = [dev(a) for a in c.arrays()]
    f4, t2 = torch.empty_like(state[0]), torch.empty_like(state[3])
    rates = [torch.zeros(n, 4, device="cuda"), torch.zeros(n, 4, device="cuda"), torch.zeros(n, 6, device="cuda")]
    beg, end = (torch.empty(par.ncell, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    poison(4 * n)
    stream = torch.cuda.Stream()
    s = stream.cuda_stream
    with torch.cuda.stream(stream):
        if order == "busy default stream":
            with torch.cuda.stream(torch.cuda.default_stream()):
                torch.cuda._sleep(800_000_000)      # less than half a second
        grid = lq.Grid(n, par.ncell)

        def search(p, d):
            grid.neighbor_search(p, d, state[0], state[2], stream=s)

        def sort():
            for a in state:
                if a.shape[1] == 4:
                    grid.sort_float4(n, a, f4, stream=s)
                else:
                    grid.sort_tensor2d(n, a, t2, stream=s)

        if order == "fewer first":
            search(few, pd_few)
        search(par, pd)
        sort()
        if order == "fewer between":
            a = grid.arrays()
            lq.particle_interaction(par, pd, *state, *rates, a["cell_beg"], a["cell_end"], stream=s)
            search(few, pd_few)
            search(par, pd)
            sort()
        a = grid.arrays()
        for src, dst in ((a["cell_beg"], beg), (a["cell_end"], end)):
            rt.cudaMemcpyAsync(dst.data_ptr(), src, 4 * par.ncell, rt.cudaMemcpyKind.cudaMemcpyDeviceToDevice, s)
        builds, reuses = lq.interaction_stats()
        for turn in range(2):
            if turn:
                state[1][nb:, :3] *= -0.7
            lq.particle_interaction(par, pd, *state, *rates, a["cell_beg"], a["cell_end"], stream=s)
            stream.synchronize()
            got = [host(r)[nb:].copy() for r in rates]
            if turn:
                b, u = lq.interaction_stats()
                assert (b - builds, u - reuses) == (1, 1)
                break
        lq.particle_interaction(par, pd, *state, *rates, beg.data_ptr(), end.data_ptr(), stream=s)
        stream.synchronize()
    torch.cuda.synchronize()
    grid.close()
    for g, w, name in zip(got, [host(r)[nb:] for r in rates], ("acceleration", "spin", "strain rate")):
        assert rel_l2(g, w) < TOL, (order, name, rel_l2(g, w))
