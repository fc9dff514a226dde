"""The interaction's working arrays are ready when the call that allocates them
returns: the counts of list builds and reuses, zeroed on the default stream,
hold what calls on another stream counted although the default stream was busy
meanwhile.  A child process, whose first allocation it is."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

SCRIPT = r"""
import sys
sys.path.insert(0, "tests")
import torch
import loquat_b200 as lq
from loquat_b200 import cases
from helpers import dev, par_dev
c = cases.small_column(seed=73)
n, pd = c.par.np, par_dev(c.par)
state = [dev(a) for a in c.arrays()]
f4, t2 = torch.empty_like(state[0]), torch.empty_like(state[3])
rates = [torch.zeros(n, 4, device="cuda"), torch.zeros(n, 4, device="cuda"), torch.zeros(n, 6, device="cuda")]
grid = lq.Grid(n, c.par.ncell)
stream = torch.cuda.Stream()
s = stream.cuda_stream
torch.cuda.synchronize()
grid.neighbor_search(c.par, pd, state[0], state[2], stream=s)
for x in state:
    (grid.sort_float4 if x.shape[1] == 4 else grid.sort_tensor2d)(n, x, f4 if x.shape[1] == 4 else t2, stream=s)
a = grid.arrays()
stream.synchronize()
torch.cuda._sleep(800_000_000)          # less than half a second
lq.interaction_reserve(c.par)
for _ in range(3):
    lq.particle_interaction(c.par, pd, *state, *rates, a["cell_beg"], a["cell_end"], stream=s)
stream.synchronize()
torch.cuda.synchronize()
print("STATS", *lq.interaction_stats())
"""


def test_counts_survive_a_busy_default_stream(lq, cuda):
    env = dict(os.environ, PYTHONPATH=str(ROOT), CUDA_MODULE_LOADING="EAGER")   # no waits to load kernels
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, env=env, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "STATS 1 2" in r.stdout, r.stdout
