"""lq_grid_sort_float4 / _tensor2d: the array and its cache after the call
against the permutation of the grid's search, for counts that end inside a
block and, from 148 x 4 blocks of 256 on, inside a thread's second turn."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1, 1), (3, 4, 5), (40, 21, 19), (67, 41, 53), (111, 63, 91)])
def test_arrays_follow_the_search(lq, cuda, size):
    import torch

    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, seed=23)
    lq.initialize_parameters(c.par)
    n = c.par.np
    rng = np.random.default_rng(24)
    order = rng.permutation(n)
    pos, idep = (torch.as_tensor(np.ascontiguousarray(np.asarray(a)[order]), device="cuda")
                 for a in (c.arrays()[0], c.arrays()[2]))
    par_dev = torch.from_numpy(np.frombuffer(c.par.to_bytes(), dtype=np.uint8).copy()).cuda()
    grid = lq.Grid(n, c.par.ncell)
    grid.neighbor_search(c.par, par_dev, pos, idep)
    ids = torch.arange(n, device="cuda", dtype=torch.int32)
    tag = ids.view(torch.float32)[:, None].repeat(1, 4).contiguous()    # bit patterns: no arithmetic
    tag_cache = torch.zeros_like(tag)
    t2 = torch.rand(n, 6, device="cuda")
    t2_cache = torch.zeros_like(t2)
    before = t2.clone()
    torch.cuda.synchronize()
    grid.sort_float4(n, tag, tag_cache)
    grid.sort_tensor2d(n, t2, t2_cache)
    torch.cuda.synchronize()
    perm = tag.view(torch.int32)
    assert torch.equal(perm[:, :1].expand(n, 4), perm)
    p = perm[:, 0].long()
    assert torch.equal(torch.sort(p).values, torch.arange(n, device="cuda"))
    assert torch.equal(tag_cache.view(torch.int32), perm)
    assert torch.equal(t2, before[p]) and torch.equal(t2_cache, t2)
    want = pos[p]
    grid.sort_float4(n, pos, tag_cache)
    torch.cuda.synchronize()
    assert torch.equal(pos, want)
    grid.close()
