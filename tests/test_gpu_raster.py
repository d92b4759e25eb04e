"""Capsules drawn onto the screen (no tree): images equal the CPU restatement byte
for byte where the conservative rectangles could go wrong -- capsules at and
beyond the image's edges, around and behind the camera, larger than a slice of
pixels, degenerate, wide angles off the axis, a camera far away, jittered frames,
ragged image sizes -- and where the scene falls back to the tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(seed, count, extent, length):
    rng = np.random.default_rng(seed)
    start = rng.uniform(-extent, extent, (count, 3))
    step = rng.normal(size=(count, 3)) * length
    v = np.zeros((2 * count, 4), np.float32)
    v[0::2, :3], v[1::2, :3] = start, start + step
    v[20] = v[21]                                                   # no length
    c = rng.uniform(0, 1, (2 * count, 4)).astype(np.float32)
    return [(v, c, np.arange(0, 2 * count - 1, 2, dtype=np.int32))]


VIEWS = {
    "front": ((0.0, 0.0, -6.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0)),
    "oblique": ((4.0, 3.0, -2.5), (-0.8, -0.55, 0.6), (0.1, 1.0, -0.2)),
    "close": ((0.1, 0.05, -1.25), (0.1, 0.0, 1.0), (0.0, 1.0, 0.0)),
    "inside": ((0.0, 0.1, 0.0), (0.3, 0.2, 1.0), (0.0, 1.0, 0.0)),
    "away": ((0.0, 0.0, -3.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0)),
    "far": ((0.0, 0.0, -500.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0)),
}


@pytest.mark.parametrize("view", sorted(VIEWS))
@pytest.mark.parametrize("radius", [0.001, 0.02, 0.4])
def test_images_equal_the_oracle(ctx, port, view, radius):
    for seed, (count, length, size, frames) in enumerate([(400, 0.05, (97, 61), 1), (37, 1.5, (160, 121), 3), (1, 0.5, (33, 250), 2)]):
        batches = _scene(seed, max(count, 11), 1.0, length)
        if count == 1:
            batches = [(batches[0][0][:2], batches[0][1][:2], np.zeros(1, np.int32))]
        ctx.ray_tracer_clear_volume()
        ctx.ray_tracer_set_integral_curves_host(batches, radius)
        ctx.ray_tracer_set_image_size(*size)
        ctx.ray_tracer_set_camera(*VIEWS[view])
        ctx.ray_tracer_trace(frames)
        got = ctx.ray_tracer_serialize()
        expected, _ = port.render(batches, radius, VIEWS[view], size, frames=frames)
        diff = np.any(got != expected, axis=-1)
        assert not diff.any(), (seed, int(diff.sum()), np.argwhere(diff)[:3].tolist())


def test_equal_distances_keep_the_smaller_segment_and_frames_accumulate(ctx, port):
    """The same segment twice, in two colours: the first one's colour; one call of
    four frames equals four calls of one; a new camera starts again."""
    v = np.array([[-1, 0, 0, 0], [1, 0.2, 0, 0], [-1, 0, 0, 0], [1, 0.2, 0, 0]], np.float32)
    c = np.array([[1, 0, 0, 1], [1, 0, 0, 1], [0, 1, 0, 1], [0, 1, 0, 1]], np.float32)
    for order in ([0, 2], [2, 0]):
        batches = [(v, c, np.array(order, np.int32))]
        images = []
        for calls in ((4,), (1, 1, 1, 1)):
            ctx.ray_tracer_clear_volume()
            ctx.ray_tracer_set_integral_curves_host(batches, 0.3)
            ctx.ray_tracer_set_image_size(70, 41)
            ctx.ray_tracer_set_camera(*VIEWS["close"])
            ctx.ray_tracer_trace(1)
            ctx.ray_tracer_set_camera(*VIEWS["front"])
            for k in calls:
                ctx.ray_tracer_trace(k)
            assert ctx.ray_tracer_frames() == 4
            images.append(ctx.ray_tracer_serialize())
        expected, _ = port.render(batches, 0.3, VIEWS["front"], (70, 41), frames=4)
        assert np.array_equal(images[0], expected) and np.array_equal(images[1], expected)
        assert images[0][..., 0].max() > images[0][..., 1].max()


def test_every_srgb_code_is_the_thresholds_code(ctx, port):
    """One-frame images of a white sphere under many sizes reach most codes; each pixel's byte equals the oracle's."""
    v = np.array([[0, 0, 0, 0], [1e-3, 0, 0, 0]], np.float32)
    ramp = np.linspace(0.0, 1.3, 33)
    seen = set()
    for k in ramp:
        c = np.full((2, 4), k, np.float32)
        batches = [(v, c, np.zeros(1, np.int32))]
        ctx.ray_tracer_clear_volume()
        ctx.ray_tracer_set_integral_curves_host(batches, 1.5)
        ctx.ray_tracer_set_image_size(64, 64)
        ctx.ray_tracer_set_camera(*VIEWS["front"])
        ctx.ray_tracer_trace(1)
        got = ctx.ray_tracer_serialize()
        expected, _ = port.render(batches, 1.5, VIEWS["front"], (64, 64))
        assert np.array_equal(got, expected)
        seen |= set(got[..., :3].ravel().tolist())
    assert len(seen) > 150


@pytest.mark.parametrize("radius", [0.001, 0.01, 0.05])
def test_thin_segments_at_every_angle_equal_the_oracle(ctx, port, radius):
    """Bands along rows and columns: slopes through 0, 1 and infinity, both directions,
    some ending beyond the image."""
    angle = np.linspace(0, 2 * np.pi, 49)
    v = np.zeros((98, 4), np.float32)
    for k, (at, length) in enumerate(zip(angle, np.resize([0.3, 1.0, 3.0], 49))):
        centre = np.array([0.3 * np.cos(7 * at), 0.3 * np.sin(5 * at), 0.2 * np.sin(at)])
        along = np.array([np.cos(at), np.sin(at), 0.1 * np.cos(3 * at)]) * length
        v[2 * k, :3], v[2 * k + 1, :3] = centre, centre + along
    c = np.random.default_rng(3).uniform(0, 1, (98, 4)).astype(np.float32)
    batches = [(v, c, np.arange(0, 97, 2, dtype=np.int32))]
    view = ((0.0, 0.0, -3.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0))
    ctx.ray_tracer_clear_volume()
    ctx.ray_tracer_set_integral_curves_host(batches, radius)
    ctx.ray_tracer_set_image_size(301, 233)
    ctx.ray_tracer_set_camera(*view)
    ctx.ray_tracer_trace(2)
    expected, _ = port.render(batches, radius, view, (301, 233), frames=2)
    assert np.array_equal(ctx.ray_tracer_serialize(), expected)
