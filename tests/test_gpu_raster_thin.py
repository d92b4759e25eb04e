"""Long thin segments: the capsule test's discriminant cancels terms of the segment's length
squared, so its hits reach farther from the axis than the radius.  Capsules drawn onto the
screen keep all of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZE = (1080, 1920)


def scene(seed, length, radius):
    """Forty segments of one length, in a box of its size, colours by segment."""
    rng = np.random.default_rng(seed)
    count = 40
    centre = rng.uniform(-1, 1, (count, 3)) * max(1.0, 0.4 * length)
    along = rng.normal(size=(count, 3))
    along *= 0.5 * length / np.linalg.norm(along, axis=1, keepdims=True)
    v = np.zeros((2 * count, 4), np.float32)
    v[0::2, :3], v[1::2, :3] = centre - along, centre + along
    c = np.repeat(rng.uniform(0.2, 1, (count, 4)), 2, axis=0).astype(np.float32)
    return [(v, c, np.arange(0, 2 * count - 1, 2, dtype=np.int32))]


def view(length):
    eye = np.array([0.3, -0.2, -(1.5 + 1.6 * max(1.0, length))])
    return tuple(eye), tuple(-eye / np.linalg.norm(eye)), (0.05, 1.0, 0.1)


@pytest.mark.parametrize("radius", [1e-4, 1e-3, 1e-2])
@pytest.mark.parametrize("length", [0.05, 0.5, 2.0, 6.0])
def test_thin_segments_drawn_equal_the_oracle(ctx, port, length, radius):
    for seed in range(3):
        batches = scene(seed, length, radius)
        ctx.ray_tracer_clear_volume()
        ctx.ray_tracer_set_integral_curves_host(batches, radius)
        ctx.ray_tracer_set_image_size(*SIZE)
        ctx.ray_tracer_set_camera(*view(length))
        ctx.profile_reset()
        ctx.profile_enable(True)
        ctx.ray_tracer_trace(1)
        drawn, walked = ctx.profile_get("raster")[1], ctx.profile_get("tree_hits")[1]
        ctx.profile_enable(False)
        assert drawn == 1 and walked == 0
        got = ctx.ray_tracer_serialize()
        expected, _ = port.render(batches, radius, view(length), SIZE)
        diff = np.any(got != expected, axis=-1)
        assert not diff.any(), (seed, int(diff.sum()), np.argwhere(diff)[:3].tolist())
