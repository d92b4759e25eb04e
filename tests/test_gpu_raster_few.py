"""Scenes of few capsules drawn onto the screen: a warp takes as few capsules as give every
warp some, large capsules start at fewer pixels and their slices are cut into parts, and
the frames of small images go through one launch together.  Images equal the oracle's."""
import numpy as np
import pytest

from test_gpu_raster_refused import VIEW, _spheres

pytestmark = pytest.mark.gpu


def _open(ctx, batches, radius, size):
    ctx.ray_tracer_clear_volume()
    ctx.ray_tracer_set_integral_curves_host(batches, radius)
    ctx.ray_tracer_set_image_size(*size)
    ctx.ray_tracer_set_camera(*VIEW)


def _check(ctx, port, batches, radius, size, frames, view=VIEW):
    expected, _ = port.render(batches, radius, view, size, frames=frames)
    diff = np.any(ctx.ray_tracer_serialize() != expected, axis=-1)
    assert not diff.any(), int(diff.sum())


@pytest.mark.parametrize("size,frames", [((70, 41), 5), ((70, 41), 65), ((1000, 700), 5), ((2100, 999), 2)])
@pytest.mark.parametrize("count,radius", [(1, 1.5), (3, 0.8), (40, 0.3), (300, 0.02)])
def test_frames_go_together(ctx, port, size, frames, count, radius):
    """All frames in one launch, in launches of two and a rest, and one at a time."""
    batches = _spheres(count, radius, count, 1.0)
    for calls in ([frames], [frames - 1, 1]):
        _open(ctx, batches, radius, size)
        for n in calls:
            ctx.ray_tracer_trace(n)
        _check(ctx, port, batches, radius, size, frames)


@pytest.mark.parametrize("radius", [0.004, 0.06])
def test_capsules_per_warp(ctx, port, radius):
    """Capsule counts at which a warp takes twice as many, and at which large ones start later."""
    import torch
    warps = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    for count in (1, 16384, 16385, 2 * warps - 1, 2 * warps, 4 * warps + 3):
        batches = _spheres(count, radius, 5, 1.5)
        _open(ctx, batches, radius, (333, 250))
        ctx.ray_tracer_trace(1)
        _check(ctx, port, batches, radius, (333, 250), 1)


def test_a_scene_looked_at_again(ctx, port):
    """Drawn first; its next view builds the tree where the walk alone is the cheaper way."""
    batches, radius, size = _spheres(700, 0.55, 1, 0.5), 0.55, (640, 480)
    _open(ctx, batches, radius, size)
    other = ((0.5, 0.2, -6.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0))
    builds = []
    for view in (VIEW, other, VIEW):
        ctx.ray_tracer_set_camera(*view)
        ctx.profile_reset()
        ctx.profile_enable(True)
        ctx.ray_tracer_trace(2)
        builds.append((ctx.profile_get("bvh_build")[1] > 0, ctx.profile_get("raster")[1] > 0))
        ctx.profile_enable(False)
        _check(ctx, port, batches, radius, size, 2, view)
    assert builds == [(False, True), (True, True), (False, False)]
