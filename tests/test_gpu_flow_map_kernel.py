"""The flow-map kernel at the edges of its work division: fewer seeds than a
warp, a few more, ragged shapes, a lattice larger than the flow map, and enough
seeds that lanes take several; frozen stages equal the oracle's flow map bit for
bit for every integrator, re-sampled ones stay within 1e-3 cells of FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (3, 2, 5), (2, 3, 11), (4, 4, 9), (17, 5, 33)]


def _field(shape, seed):
    from pars_gb300 import workloads as W
    rng = np.random.default_rng(seed)
    h = np.float32(0.25)
    base = np.array([0.7, -0.4, 0.55])
    xyz = (base + 0.4 * rng.normal(size=(*shape, 3))).astype(np.float32)
    return W.Field(xyz, np.array([0.5, -1.0, 0.0], np.float32), np.full(3, h, np.float32))


@pytest.mark.parametrize("integrator", range(8))
def test_flow_maps_of_small_and_ragged_grids(ctx, port, integrator):
    from pars_gb300 import native
    for k, shape in enumerate(SHAPES):
        f = _field(shape, 10 * integrator + k)
        h = ctx.upload_field(f)
        for iterations in (0, 1, 2, 30):
            fm, steps = ctx.flow_map_generate(h, iterations, 1.0, integrator, native.STAGES_FROZEN, 0.05)
            expected, expected_steps = port.flow_map(f, iterations, 1.0, integrator, 0.05)
            assert steps == expected_steps
            if iterations > 1:
                assert np.array_equal(ctx.download_field(fm), expected)
            ctx.release_field(fm)
        fm, steps = ctx.flow_map_generate(h, 21, 1.0, integrator, native.STAGES_RESAMPLED, 0.02)
        got = ctx.download_field(fm).reshape(-1, 3).astype(np.float64)
        ctx.release_field(fm)
        ijk = np.stack(np.unravel_index(np.arange(len(got)), shape), -1).astype(np.float32)
        start = (f.offset + ijk * f.spacing).astype(np.float32).astype(np.float64)
        end, steps64, _ = port.advect_fp64(f, start, 20, integrator=integrator, mode=1, step=0.02)
        ctx.release_field(h)
        cell = float(f.spacing[0])
        err = np.linalg.norm(got - end, axis=1) / cell
        # a step taken or not at a face moves the end point by a step; counts decide whether one was
        if steps == int(steps64.sum()):
            assert err.max() <= 1e-3, (shape, err.max())
        else:
            assert np.mean(err <= 1e-3) > 0.9, shape


def test_many_seeds_per_lane_equal_few(ctx, port):
    """A lattice with more than refill_from_rounds seeds a lane (lanes refilled one
    by one) against its strided part (a warp's seeds run to the end)."""
    from pars_gb300 import native, workloads as W
    f = W.abc_field(120, noise_sigma=0.01, seed=4)
    h = ctx.upload_field(f)
    for integrator, stages in ((2, native.STAGES_FROZEN), (4, native.STAGES_RESAMPLED), (7, native.STAGES_RESAMPLED)):
        fm, _ = ctx.flow_map_generate(h, 41, 1.0, integrator, stages, 0.02)       # 1.7 M seeds
        fine = ctx.download_field(fm)
        ctx.release_field(fm)
        fm, _ = ctx.flow_map_generate(h, 41, 0.5, integrator, stages, 0.02)       # 216 k seeds at every other vertex
        coarse = ctx.download_field(fm)
        ctx.release_field(fm)
        # spacing / 0.5 = 2 h exactly; index * 2 h and 2 index * h round alike
        assert np.array_equal(coarse, fine[::2, ::2, ::2][:60, :60, :60])
    ctx.release_field(h)
