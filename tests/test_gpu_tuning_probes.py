"""The first unsteady launch of a process times the launch shapes that it may choose, and no
other: the shape for few seeds is chosen by their number."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch
from pars_gb300 import native, workloads as W
c = native.Context(0)
xyz, offset, spacing, t0, dt = W.double_gyre_slices(8, 3)
j = native.BatchJob()
j.field, j.integrator, j.stage_mode = c.upload_unsteady_field(xyz, offset, spacing, t0, dt), native.RUNGE_KUTTA_4, native.STAGES_RESAMPLED
j.max_steps, j.step_size = 4, 0.02
seeds = torch.full((64, 4), 0.3, device="cuda")
torch.cuda.synchronize()
j.seeds, j.seed_count = seeds.data_ptr(), len(seeds)
before = c.launch_count()
steps = c.batch_advect([j])
print(steps[0], c.launch_count() - before)
"""


def test_the_shape_for_few_seeds_is_not_timed():
    out = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env={**os.environ, "PYTHONPATH": ROOT}, capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    # three shapes twice, then the launch itself
    assert out.stdout.split() == ["256", "7"]
