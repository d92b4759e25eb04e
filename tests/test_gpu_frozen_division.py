"""The frozen scheme's cell search divides by the spacing through its rounded
reciprocal and an exact remainder; the cells and weights, and so the sampled
velocities, are the reference's bits for every spacing and offset, also where
that path does not apply (spacings out of its range, points a hair from a grid
plane at the origin, points outside, infinities and NaNs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [
    (1.0, 0.5, 2.0), (np.nextafter(np.float32(2), np.float32(0)), 0.1, 1 / 3), (0.024639942, 0.09973310, 7.0e-7),
    (3.0e6, 1.0, 1.0), (2.0 ** -20, 2.0 ** 20, 1.7), (1.1754944e-30, 1.0, 1.0)])
def test_samples_are_the_references_bits(ctx, port, spacing):
    from pars_gb300 import workloads as W
    rng = np.random.default_rng(7)
    n = np.array([9, 6, 12])
    h = np.array(spacing, np.float32)
    for offset in (np.zeros(3, np.float32), (np.array([1.7, -3.1, 100.0]) * h).astype(np.float32)):
        f = W.Field(rng.normal(size=(*n, 3)).astype(np.float32), offset, h)
        u = rng.uniform(-0.6, 1.05, (20000, 3)) * n                 # inside and outside
        u[:8000] = np.round(u[:8000]) + rng.choice([0.0, 1e-7, -1e-7, 6e-8], (8000, 3))   # next to the planes
        with np.errstate(over="ignore"):
            p = np.zeros((len(u) + 9, 4), np.float32)
            p[:len(u), :3] = (offset + u * h).astype(np.float32)
        p[len(u):len(u) + 6, :3] = offset + np.array([[0.0], [-0.0], [1e-13], [1e-30], [1e-42], [-1e-42]], np.float32) * np.ones(3, np.float32)
        p[len(u) + 6:, 0] = [np.inf, -np.inf, np.nan]
        hnd = ctx.upload_field(f)
        inside, v = ctx.sample(hnd, p)
        ctx.release_field(hnd)
        assert not inside[-3:].any()
        inside, v = inside[:-3], v[:-3]
        expected_inside, expected = port.field_sample(f, p[:-3])
        assert np.array_equal(inside, expected_inside.astype(bool))
        assert np.array_equal(v[inside].view(np.uint32), expected[inside].view(np.uint32))
