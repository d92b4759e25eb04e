"""Walks through the tree beside a volume: shading in the walk's own launch (all frames in
one, or one for each) and in a launch of its own give the oracle's bytes."""
import numpy as np
import pytest

from test_gpu_raster_refused import _spheres

pytestmark = pytest.mark.gpu

SIZE = (1280, 1024)


@pytest.mark.parametrize("frames", [1, 3])
@pytest.mark.parametrize("count", [16, 17, 2048, 2049])
def test_walks_with_a_volume(ctx, port, count, frames):
    batches = _spheres(count, 0.05, count, 0.5)
    # a camera inside the first capsule, which covers the whole image: the tree is built
    view = (tuple(batches[0][0][0, :3]), (0.2, 0.1, 1.0), (0.0, 1.0, 0.0))
    rng = np.random.default_rng(count)
    volume = (rng.uniform(-0.2, 1.0, (7, 6, 5)).astype(np.float32), (-1.0, -1.5, -0.5), (0.4, 0.5, 0.3))
    ctx.ray_tracer_set_volume(*volume)
    ctx.ray_tracer_set_integral_curves_host(batches, 0.05)
    ctx.ray_tracer_set_image_size(*SIZE)
    ctx.ray_tracer_set_camera(*view)
    ctx.profile_reset()
    ctx.profile_enable(True)
    ctx.ray_tracer_trace(frames)
    walks, shaded = ctx.profile_get("tree_hits")[1], ctx.profile_get("render")[1]
    ctx.profile_enable(False)
    assert (walks, shaded) == {16: (0, 1), 17: (0, frames), 2048: (0, frames), 2049: (frames, frames)}[count]
    got = ctx.ray_tracer_serialize()
    ctx.ray_tracer_clear_volume()
    expected, _ = port.render(batches, 0.05, view, SIZE, frames=frames, volume=volume)
    diff = np.any(got != expected, axis=-1)
    assert not diff.any(), int(diff.sum())
