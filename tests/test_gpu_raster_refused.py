"""Scenes at the limits of the drawing onto the screen: many large capsules, each cut into
slices, and scenes that are left to the tree because one capsule or all together cover too
much.  Those launch nothing per frame that draws nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VIEW = ((0.0, 0.0, -6.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0))


def _spheres(count, radius, seed, depth):
    rng = np.random.default_rng(seed)
    v = np.zeros((2 * count, 4), np.float32)
    v[0::2, :3] = v[1::2, :3] = rng.uniform(-1, 1, (count, 3)) * (2.5, 2.0, depth)
    v[1::2, 0] += np.float32(0.01)
    return [(v, rng.uniform(0, 1, (2 * count, 4)).astype(np.float32), np.arange(0, 2 * count - 1, 2, dtype=np.int32))]


def _trace(ctx, batches, radius, size, frames):
    ctx.ray_tracer_clear_volume()
    ctx.ray_tracer_set_integral_curves_host(batches, radius)
    ctx.ray_tracer_set_image_size(*size)
    ctx.ray_tracer_set_camera(*VIEW)
    ctx.profile_reset()
    ctx.profile_enable(True)
    ctx.ray_tracer_trace(frames)
    launches = {k: ctx.profile_get(k)[1] for k in ("raster", "bvh_build", "render")}
    ctx.profile_enable(False)
    return ctx.ray_tracer_serialize(), launches


@pytest.mark.parametrize("frames", [1, 3])
@pytest.mark.parametrize("scene", ["drawn", "covered", "around"])
def test_large_capsules(ctx, port, scene, frames):
    if scene == "drawn":       # about 6000 pixels each
        batches, radius, size = _spheres(700, 0.55, 1, 0.5), 0.55, (640, 480)
    elif scene == "covered":   # far more pixels than the tree's walk is worth
        batches, radius, size = _spheres(3000, 0.9, 2, 0.5), 0.9, (640, 480)
    else:                      # one capsule beside the camera covers the whole image
        batches, radius, size = _spheres(40, 0.05, 3, 0.5), 0.05, (1280, 1024)
        batches[0][0][6:8, 2] = [-7.0, -5.0]
        batches[0][0][6:8, :2] = 0.4
    got, launches = _trace(ctx, batches, radius, size, frames)
    if scene == "drawn":
        # (640 x 480: up to six frames go through one launch)
        assert launches == {"raster": 1, "bvh_build": 0, "render": 1}
    else:
        assert launches["raster"] == 1 and launches["bvh_build"] >= 1 and launches["render"] == frames
    expected, _ = port.render(batches, radius, VIEW, size, frames=frames)
    diff = np.any(got != expected, axis=-1)
    assert not diff.any(), int(diff.sum())
