"""Unsteady launches of few and of many seeds take different launch shapes: the same
bits either way, and the continuous engine changes over between its jobs."""
import numpy as np
import pytest

from test_gpu_pools import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [("few", "many", "few"), ("many", "few", "many")])
def test_results_do_not_depend_on_the_launch_shape(ctx, order):
    import torch
    from pars_gb300 import native, workloads as W
    xyz, offset, spacing, t0, dt = W.double_gyre_slices(24, 5)
    field = ctx.upload_unsteady_field(xyz, offset, spacing, t0, dt)
    # either side of 12 warps of seeds per SM, the most that the shape for few seeds holds
    fill = 12 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    count = {"few": fill, "many": fill + 1}
    p = torch.rand((fill + 1, 4), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    p[:, :3] *= torch.tensor((2.0, 1.0, 1.0), device="cuda")
    p[:, 3] = 0.0
    ends = {}
    for name in order:
        seeds = p[: count[name]].contiguous()
        batch, engine = (_job(native, torch, field, seeds, 40, native.STAGES_RESAMPLED) for _ in range(2))
        torch.cuda.synchronize()
        total = ctx.batch_advect([batch[0]])[0]
        ctx.engine_submit(engine[0])
        done, left = [], 1
        while left:
            finished, left = ctx.engine_advance(16)
            done += finished
        assert [d[1] for d in done] == [total]
        assert torch.equal(batch[1], engine[1]) and torch.equal(batch[2], engine[2])
        ends[name] = batch[1]
    assert torch.equal(ends["few"], ends["many"][:fill])
    ctx.release_field(field)
