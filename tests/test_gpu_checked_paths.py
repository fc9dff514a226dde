"""The bounds-checked build (test_gpu_checked.py) over the paths that run there
do not reach: the drop-in step with carried and with fresh lists, the array
sorts on both sides of the one-cluster form, lists in bank order by more than
one piece, few targets by teams, and the model-3 queue from one entry to
several blocks, with many sub-steps each.  No run may count a violation."""
from __future__ import annotations

from test_gpu_checked import CHECKED, ROOT

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import loquat_b200 as lq
from loquat_b200 import cases
from loquat_b200.dropin import ReferenceStep
for nsx, carry in ((6, True), (16, True), (16, False), (40, True)):
    c = cases.small_column(nsx=nsx, nsy=nsx // 2, nsz=nsx // 2, velocity_noise=0.3, shepard=4, seed=81).with_ids()
    seq = ReferenceStep(c.par, *c.arrays(), carry=carry)
    seq.step(12)
    seq.close()
r, u = lq.interaction_stats()
assert r >= 3 and u >= 10, (r, u)
for hdr, shape in ((1.2, 0), (1.35, 9), (1.7, 0)):      # lists of 60 to more than 96 entries, then overflowing ones
    c = cases.small_column(nsx=24, nsy=18, nsz=24, hdr=hdr, velocity_noise=0.3, seed=82)
    for mixed in (False, True):
        s = lq.Simulation(c.par, *c.arrays(), mixed=mixed)
        s.set_pair_shape(shape)
        s.step(12)
        s.close()
for size, tol in (((1, 1, 1), 1e-4), ((5, 3, 4), 1e-6), ((24, 8, 12), 1e-6)):
    c = cases.small_column(nsx=size[0], nsy=size[1], nsz=size[2], model=3, velocity_noise=0.05, seed=83,
                           vw=cases.vw_row(tol=tol))
    s = lq.Simulation(c.par, *c.arrays(), mixed=True)
    s.set_hypoplastic(c.meta["hypoplastic"])
    s.step(12)
    s.close()
print("VIOLATIONS", lq.bounds_violations())
"""


def test_reworked_paths_count_no_bounds_violation(cuda):
    from loquat_b200 import build

    srcs = list((ROOT / "loquat_b200" / "csrc").iterdir()) + list((ROOT / "include").iterdir())
    if not CHECKED.exists() or CHECKED.stat().st_mtime < max(p.stat().st_mtime for p in srcs):
        build.build_checked()      # a checked library older than the sources tests other code
    env = dict(os.environ, LOQUAT_B200_LIB=str(CHECKED), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, env=env, timeout=600, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "VIOLATIONS 0" in r.stdout, r.stdout
