"""Long thin segments through the walk of the tree: its boxes hold every hit of the capsule
test, whose rounding grows with the segment's length."""
import numpy as np
import pytest

from test_gpu_raster_thin import SIZE, scene, view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1e-4, 1e-3, 1e-2])
@pytest.mark.parametrize("length", [0.05, 0.5, 2.0, 6.0])
def test_thin_segments_of_the_tree_equal_the_oracle(ctx, port, length, radius):
    for seed in range(3):
        batches = scene(seed, length, radius)
        ctx.ray_tracer_clear_volume()
        ctx.ray_tracer_set_integral_curves_host(batches, radius)
        ctx.ray_tracer_set_image_size(*SIZE)
        # a camera in the middle of a segment: the whole image belongs to it, so the tree is
        # built, and serves the scene's later views
        v = batches[0][0]
        ctx.ray_tracer_set_camera(tuple(0.5 * (v[0, :3] + v[1, :3])), tuple(v[1, :3] - v[0, :3]), (0.05, 1.0, 0.1))
        ctx.ray_tracer_trace(1)
        ctx.ray_tracer_set_camera(*view(length))
        ctx.profile_reset()
        ctx.profile_enable(True)
        ctx.ray_tracer_trace(1)
        drawn, rendered = ctx.profile_get("raster")[1], ctx.profile_get("render")[1]
        ctx.profile_enable(False)
        assert drawn == 0 and rendered == 1
        expected, _ = port.render(batches, radius, view(length), SIZE)
        diff = np.any(ctx.ray_tracer_serialize() != expected, axis=-1)
        assert not diff.any(), (seed, int(diff.sum()), np.argwhere(diff)[:3].tolist())
