"""The kernels that small cases take: the pair kernel with a team of lanes
per target (shape 0 up to 8192 targets) against the thread-per-target form,
bit for bit, where the target count ends inside a block, a warp or a team's
batch; and the list-driven Adami with eight, four and one lane per target
against the oracle, for walls whose targets end inside a warp."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("size", [(1, 1, 1), (3, 3, 5), (16, 6, 12), (9, 5, 7), (32, 16, 16), (33, 16, 16)])
def test_team_and_thread_forms_agree_bit_for_bit(lq, cuda, size, mixed):
    """32 x 16 x 16 = 8192 targets take teams, one layer more threads.  A
    single particle's filter divides zero by zero: NaN in every form."""
    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, velocity_noise=0.2, shepard=3, seed=91, hdr=1.2 + 0.1 * (nx % 3))
    c.par.artificial_pressure, c.par.artificial_pressure_coefficient = int(nx == 9), 0.3
    lq.initialize_parameters(c.par)
    runs = []
    for shape in (0, 8, 3):
        s = lq.Simulation(c.par, *c.arrays(), mixed=mixed)
        s.set_pair_shape(shape)
        s.step(8)
        runs.append(s.download())
    for other in runs[1:]:
        for x, y in zip(runs[0], other):
            assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("size", [(2, 1, 3), (7, 5, 9), (21, 10, 6), (131, 127, 3), (241, 239, 3)])
def test_wall_stress_vs_oracle(lq, orc, cuda, size):
    """One step's boundary stress: eight lanes per target to 32768 targets,
    four for the 131 x 127 floor's (about 3 layers of it), one for the
    241 x 239 floor's.  The bound is the operator test's (FP32 sums of up to
    60 terms, relative L2)."""
    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, velocity_noise=0.02, seed=92).with_ids()
    s = lq.Simulation(c.par, *c.arrays(), mixed=True)
    s.step(1)
    got = by_id(s.download())
    o = orc.OracleSim(c.par, *c.arrays())
    o.step(1)
    want = by_id(o.get())
    o.close()
    b = slice(0, c.par.npb)
    assert rel_l2(got[3][b], want[3][b]) < 1e-5
