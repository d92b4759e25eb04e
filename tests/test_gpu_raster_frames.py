"""Calls of several frames draw every capsule in every frame: a capsule's rectangle gains or
loses a row or a column with a frame's jitter, so it may be small enough for one warp in one
frame and cut into slices in the next, or need one slice more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VIEW = ((0.0, 0.0, -6.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0))
SLICE = 2048


def _trace(ctx, batches, radius, size, calls):
    ctx.ray_tracer_clear_volume()
    ctx.ray_tracer_set_integral_curves_host(batches, radius)
    ctx.ray_tracer_set_image_size(*size)
    ctx.ray_tracer_set_camera(*VIEW)
    for frames in calls:
        ctx.ray_tracer_trace(frames)
    return ctx.ray_tracer_serialize()


@pytest.mark.parametrize("frames", [2, 3, 8])
def test_a_rectangle_that_grows_past_a_slice_is_drawn(ctx, port, frames):
    """2016 pixels in the first frame, 2064 in the second."""
    v = np.array([[-0.2, 0.1, 0.0, 0.0], [0.2, -0.05, 0.0, 0.0]], np.float32)
    batches = [(v, np.ones((2, 4), np.float32), np.zeros(1, np.int32))]
    expected, _ = port.render(batches, 1.09, VIEW, (160, 121), frames=frames)
    assert np.array_equal(_trace(ctx, batches, 1.09, (160, 121), [frames]), expected)


@pytest.mark.parametrize("slices", [1, 2, 3])
def test_rectangles_around_a_multiple_of_a_slice(ctx, port, slices):
    """Capsules at the depths where their rectangles have about that many slices, some cut by
    the image's edges; one call of four frames equals four calls."""
    rng = np.random.default_rng(slices)
    width, height, radius, count = 1200, 900, 0.1, 60
    focal = height / (2 * np.tan(np.radians(34.0)))
    side = np.sqrt(SLICE * slices) + np.linspace(-3.0, 3.0, count)
    # a grid of cells, so that few hide behind others
    cell = rng.permutation(count)
    px = (cell % 10 + 0.5) * width / 10 - width / 2 + rng.uniform(-8, 8, count)
    py = (cell // 10 + 0.5) * height / 6 - height / 2 + rng.uniform(-8, 8, count)
    px[:3], py[3:6] = -width / 2, height / 2
    # (off the axis a rectangle is wider by 1 + slope)
    z = radius * (1 + 2 * focal / side * np.sqrt((1 + abs(px) / focal) * (1 + abs(py) / focal)))
    v = np.zeros((2 * count, 4), np.float32)
    v[0::2, :3] = v[1::2, :3] = np.stack([px * z / focal, py * z / focal, z - 6.0], -1)
    v[1::2, 1] += np.float32(0.01)
    batches = [(v, rng.uniform(0, 1, (2 * count, 4)).astype(np.float32), np.arange(0, 2 * count - 1, 2, dtype=np.int32))]
    expected, _ = port.render(batches, radius, VIEW, (width, height), frames=4)
    for calls in ([4], [1, 1, 1, 1], [3, 1]):
        diff = np.any(_trace(ctx, batches, radius, (width, height), calls) != expected, axis=-1)
        assert not diff.any(), (calls, int(diff.sum()))
