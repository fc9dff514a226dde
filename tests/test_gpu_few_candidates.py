"""Drop-in boundary pass and stress filter where a target has few candidates
(cells of about one particle: short smoothing lengths, sheets one particle
thick), on both sides of the number up to which they are summed untested,
against the oracle with test_gpu_operators' bounds."""
from __future__ import annotations

import numpy as np
import pytest

from loquat_b200 import cases
from helpers import dev, host, par_dev, rel_l2, sorted_state, sync, zeros
from test_gpu_operators import TOL_ADAMI, TOL_SHEPARD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(9, 1, 7), (12, 5, 9)])
@pytest.mark.parametrize("hdr", [0.4, 0.55, 0.7, 0.9])
def test_few_candidates_vs_oracle(lq, orc, cuda, hdr, size):
    nx, ny, nz = size
    c = cases.small_column(nsx=nx, nsy=ny, nsz=nz, hdr=hdr, velocity_noise=0.05, seed=78)
    par = c.par
    g, st = sorted_state(orc, c)
    rng = np.random.default_rng(79)
    st[3][par.npb:] += (1e2 * rng.standard_normal((par.npm, 6))).astype(np.float32)
    pd, x, v, b, e = par_dev(par), dev(st[0]), dev(st[1]), dev(g["cell_beg"]), dev(g["cell_end"])
    wall, filtered, cache = dev(st[3]), dev(st[3]), zeros((par.np, 6))
    lq.adami_boundary(par, pd, x, v, wall, b, e)
    lq.stress_regularization(par, pd, x, v, filtered, cache, b, e)
    sync()
    want = orc.adami(par, st[0], st[1], st[3], g["cell_beg"], g["cell_end"])
    assert rel_l2(host(wall)[: par.npb], want[: par.npb]) < TOL_ADAMI
    want = orc.shepard(par, st[0], st[1], st[3], g["cell_beg"], g["cell_end"])
    assert rel_l2(host(filtered)[par.npb:], want[par.npb:]) < TOL_SHEPARD
