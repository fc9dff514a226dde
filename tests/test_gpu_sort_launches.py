"""The array sorts are plain launches: none that must have all its blocks on
the device at once, which would wait for a caller's resident kernel and for
another stream's sort (a cooperative launch).  Read from a captured graph's
kernel nodes; replayed, the graph sorts.  Counts around the 8192 elements up to
which one cluster of blocks does it."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import dev, par_dev, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 8191, 8192, 8193, 36000])
@pytest.mark.parametrize("width", [4, 6])
def test_captured_sort_has_no_cooperative_launch(lq, cuda, width, n):
    import torch

    from cuda.bindings import runtime as rt

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]

    c = cases.small_column(nsx=40, nsy=21, nsz=25, seed=76)
    order = np.random.default_rng(77).permutation(c.par.np)[:n]
    par = c.par.copy()
    par.np, par.npb, par.npm = n, n // 2, n - n // 2
    grid = lq.Grid(n, par.ncell)
    grid.neighbor_search(par, par_dev(par), dev(c.pospres[order]))
    data = torch.rand(n, width, device="cuda")
    want, cache = data.clone(), torch.empty_like(data)
    ids = torch.arange(n, device="cuda", dtype=torch.float32)[:, None].repeat(1, 4).contiguous()
    sort = grid.sort_float4 if width == 4 else grid.sort_tensor2d
    grid.sort_float4(n, ids, torch.empty_like(ids))
    sync()
    stream = torch.cuda.Stream()
    s = stream.cuda_stream
    ok(rt.cudaStreamBeginCapture(s, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    sort(n, data, cache, stream=s)
    graph = ok(rt.cudaStreamEndCapture(s))
    count = ok(rt.cudaGraphGetNodes(graph))[-1]
    nodes = ok(rt.cudaGraphGetNodes(graph, count))[0]
    kernels = [x for x in nodes if ok(rt.cudaGraphNodeGetType(x)) == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel]
    assert kernels
    for k in kernels:
        v = ok(rt.cudaGraphKernelNodeGetAttribute(k, rt.cudaLaunchAttributeID.cudaLaunchAttributeCooperative))
        assert v.cooperative == 0
    ex = ok(rt.cudaGraphInstantiate(graph, 0))
    rt.cudaGraphLaunch(ex, s)
    stream.synchronize()
    rt.cudaGraphExecDestroy(ex)
    rt.cudaGraphDestroy(graph)
    grid.close()
    assert torch.equal(data, want[ids[:, 0].long()])
