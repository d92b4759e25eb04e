"""Unsteady jobs that join the continuous engine while another one's particles are parked: the
launch shape goes by the seeds of all of them, with the same bits as jobs of their own."""
import pytest

from test_gpu_pools import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, "many"), (4000, "many", 31), ("many", 4000), (300, 300, "many", "many")])
def test_jobs_joining_parked_ones(ctx, counts):
    import torch
    from pars_gb300 import native, workloads as W
    xyz, offset, spacing, t0, dt = W.double_gyre_slices(24, 5)
    field = ctx.upload_unsteady_field(xyz, offset, spacing, t0, dt)
    # one seed more than 12 warps per SM hold, the most that take the shape for few seeds
    many = 12 * 32 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    g = torch.Generator(device="cuda").manual_seed(7)
    alone, joined, totals = [], [], []
    for n in counts:
        p = torch.rand((many if n == "many" else n, 4), generator=g, device="cuda")
        p[:, :3] *= torch.tensor((2.0, 1.0, 1.0), device="cuda")
        p[:, 3] = 0.0
        alone.append(_job(native, torch, field, p, 50, native.STAGES_RESAMPLED) + (p,))
        joined.append(_job(native, torch, field, p, 50, native.STAGES_RESAMPLED) + (p,))
    torch.cuda.synchronize()
    for j in alone:
        totals.append(ctx.batch_advect([j[0]])[0])
    done, tickets = {}, []
    for j in joined:
        tickets.append(ctx.engine_submit(j[0]))
        finished, left = ctx.engine_advance(8)   # the job's particles are parked when the next joins
        done.update(finished)
        assert left
    while left:
        finished, left = ctx.engine_advance(8)
        done.update(finished)
    assert [done[t] for t in tickets] == totals
    for a, b in zip(alone, joined):
        assert torch.equal(a[1], b[1]) and torch.equal(a[2], b[2])
    ctx.release_field(field)
