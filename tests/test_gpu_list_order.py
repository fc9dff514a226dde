"""The stages' lists in bank order (k_list_arrange) and filled up to groups of
four: lists that end inside a group, that fit one piece of the reordering
(96 entries), that take two, and that overflow the stored 192, one- and
two-level, against the oracle.  The bounds are those of the drop-in
sequence's ten steps: FP32 sums of up to 200 terms against FP64."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("hdr", [0.85, 1.2, 1.5, 1.8])
@pytest.mark.parametrize("wide", [0.0, 0.15])
def test_ordered_lists_of_every_length_vs_oracle(lq, orc, cuda, hdr, mixed, wide):
    c = cases.small_column(nsx=13, nsy=7, nsz=11, hdr=hdr, velocity_noise=0.05, shepard=4, seed=31).with_ids()
    s = lq.Simulation(c.par, *c.arrays(), mixed=mixed)
    s.set_skin(0.03)
    s.set_wide_skin(wide)
    s.step(10)
    got = by_id(s.download())
    material, _ = s.neighbor_entries()
    mean = material / c.par.npm
    assert {0.85: 10 < mean < 40, 1.2: 40 < mean < 96, 1.5: mean > 70, 1.8: mean > 96}[hdr]
    o = orc.OracleSim(c.par, *c.arrays())
    o.step(10)
    want = by_id(o.get())
    o.close()
    m = slice(c.par.npb, c.par.np)
    assert rel_l2(got[0][m, :3], want[0][m, :3]) < 1e-6
    assert rel_l2(got[1][m, :3], want[1][m, :3]) < 1e-4
    assert rel_l2(got[1][m, 3], want[1][m, 3]) < 1e-6
    assert rel_l2(got[3][m], want[3][m]) < 1e-4
    assert np.array_equal(s.health()[:3], [0, 0, 0])
