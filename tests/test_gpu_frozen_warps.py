"""Frozen curves on either side of 16 and of 20 warps per SM, where the kernel that traces them
changes: the same bits as the oracle."""
import numpy as np
import pytest

from test_gpu_narrow_warps import _seeds
from test_gpu_parity import compare, gpu_curves

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps,extra", [(16, 0), (16, 1), (20, 0), (20, 1)])
def test_frozen_curves_match_the_oracle(ctx, port, warps, extra):
    import torch
    from pars_gb300 import native, workloads as W
    f = W.abc_field(17)
    p = _seeds(native.PARTICLE_DTYPE, 32 * warps * torch.cuda.get_device_properties(0).multi_processor_count + extra, 12)
    h = ctx.upload_field(f)
    s = ctx.trace(h, p, 2, 0, 0.05)
    expected = port.trace_single(f, p, 2, 0.05, "rgb", 0.5)
    assert s["steps"] == expected.steps
    compare(gpu_curves(ctx, s, "rgb"), expected.batches)
    ctx.release_field(h)
