"""Flow maps of few steps run one seed per thread, those of many steps take seeds from a
counter: the same bits on either side of both changes, and from small lattices as from
large ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", range(8))
def test_frozen_maps_on_either_side_equal_the_oracle(ctx, port, integrator):
    from pars_gb300 import native, workloads as W
    rng = np.random.default_rng(integrator)
    for shape in [(2, 2, 2), (3, 2, 11), (17, 5, 33)]:
        xyz = (np.array([0.7, -0.4, 0.55]) + 0.4 * rng.normal(size=(*shape, 3))).astype(np.float32)
        f = W.Field(xyz, np.array([0.5, -1.0, 0.0], np.float32), np.full(3, np.float32(0.25)))
        h = ctx.upload_field(f)
        for iterations in (16, 17, 96, 97):
            fm, steps = ctx.flow_map_generate(h, iterations, 1.0, integrator, native.STAGES_FROZEN, 0.005)
            expected, expected_steps = port.flow_map(f, iterations, 1.0, integrator, 0.005)
            assert steps == expected_steps
            assert np.array_equal(ctx.download_field(fm), expected)
            ctx.release_field(fm)
        ctx.release_field(h)


@pytest.mark.parametrize("iterations", [16, 17, 96, 97])
@pytest.mark.parametrize("integrator,frozen", [(0, True), (2, True), (6, True), (1, False), (4, False), (6, False), (7, False)])
def test_large_lattices_equal_small_ones(ctx, integrator, frozen, iterations):
    """More than six seeds a lane (1.7 M) and fewer (216 k at every other vertex)."""
    from pars_gb300 import native, workloads as W
    f = W.abc_field(120, noise_sigma=0.01, seed=4)
    h = ctx.upload_field(f)
    maps = []
    for scale in (1.0, 0.5):
        fm, _ = ctx.flow_map_generate(h, iterations, scale, integrator, native.STAGES_FROZEN if frozen else native.STAGES_RESAMPLED, 0.02)
        maps.append(ctx.download_field(fm))
        ctx.release_field(fm)
    assert np.array_equal(maps[1], maps[0][::2, ::2, ::2][:60, :60, :60])
    ctx.release_field(h)
