"""Seed pools of the batched engine: a job's results are the same bits whether it
is alone in a launch (a warp's seeds run to the end), beside a large job (lanes
refilled as particles end) or on the continuous engine, at the edges of a pool."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _job(native, torch, field, seeds, steps, stages):
    j = native.BatchJob()
    j.field, j.integrator, j.stage_mode, j.max_steps, j.step_size = field, native.RUNGE_KUTTA_4, stages, steps, 0.02
    end = torch.full((len(seeds), 4), float("nan"), dtype=torch.float32, device="cuda")
    count = torch.full((len(seeds),), -1, dtype=torch.int32, device="cuda")
    j.seeds, j.seed_count = seeds.data_ptr(), len(seeds)
    j.end_positions, j.end_steps = end.data_ptr(), count.data_ptr()
    return j, end, count


@pytest.mark.parametrize("kind", ["steady", "unsteady", "frozen"])
def test_results_do_not_depend_on_the_pool_size(ctx, kind):
    import torch
    from pars_gb300 import native, workloads as W
    stages = native.STAGES_FROZEN if kind == "frozen" else native.STAGES_RESAMPLED
    if kind == "unsteady":
        xyz, offset, spacing, t0, dt = W.double_gyre_slices(24, 5)
        field, extent = ctx.upload_unsteady_field(xyz, offset, spacing, t0, dt), (2.0, 1.0, 1.0)
    else:
        f = W.abc_field(24, noise_sigma=0.01, seed=3)
        field, extent = ctx.upload_field(f), (2 * np.pi,) * 3
    g = torch.Generator(device="cuda").manual_seed(5)

    def seeds(n):
        p = torch.rand((n, 4), generator=g, device="cuda")
        p[:, :3] *= torch.tensor(extent, device="cuda")
        p[:, 3] = 0.0
        return p

    # 4 M seeds: many rounds a lane on any GPU
    big = seeds(4 << 20)
    for n in (1, 31, 32, 33, 255, 257, 5000):
        s = seeds(n)
        alone, with_big, engine = (_job(native, torch, field, s, 60, stages) for _ in range(3))
        torch.cuda.synchronize()
        total = ctx.batch_advect([alone[0]])[0]
        filler = _job(native, torch, field, big, 2, stages)
        assert ctx.batch_advect([with_big[0], filler[0]])[0] == total
        ctx.engine_submit(engine[0])
        done, left = [], 1
        while left:
            finished, left = ctx.engine_advance(16)
            done += finished
        assert [d[1] for d in done] == [total] and int(alone[2].sum()) == total and int(alone[2].min()) >= 0
        for other in (with_big, engine):
            assert torch.equal(alone[1], other[1]) and torch.equal(alone[2], other[2]), n
    ctx.release_field(field)
