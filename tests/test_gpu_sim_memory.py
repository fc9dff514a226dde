"""A simulation's device memory: no more than its arrays at one copy of each,
so the largest particle set that fits does not shrink unnoticed.  Per
particle: three states of 96 bytes (128 mixed) of which the stage buffer
shares the object words and the scratch state the stage's records, the
records, the rates, the build positions, the search's key, rank and order, and
a list (192 entries and a count; a boundary particle's also its place among the
targets, a soil particle's its place in the tile order)."""
from __future__ import annotations

import pytest

from loquat_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
def test_bytes_per_particle(lq, cuda, mixed):
    import torch

    c = cases.cylinder_collapse(dr=0.003)       # 2.2 M particles, whose records are 115 MB
    par = c.par
    warm = lq.Simulation(par, *c.arrays(), mixed=mixed)     # what the library loads once
    warm.step(1)
    warm.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = lq.Simulation(par, *c.arrays(), mixed=mixed)
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    per = 3 * 96 - 16 + (96 if mixed else 0) + 52 + 56 + 16 + 3 * 4 + 193 * 4
    need = par.np * per + par.npb * 4 + par.npm * 4 + 2 * 4 * par.ncell
    # about 40 allocations in whole 2 MiB pages
    assert used <= need + 40 * (2 << 20), (used - need) / (1 << 20)
