"""The FTLE kernel's largest eigenvalue against FP64 on the same FP32 flow map,
where closed forms go wrong: nearly isotropic, two nearly equal eigenvalues
(the larger or the smaller two), planar flows, strong anisotropy, large and
small scales, a constant map and non-finite positions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Relative error of lambda_max: each entry of J carries two roundings, C = J^T J
# doubles them and adds three, over three columns, and the eigen-solve adds a few
# ulps of |C|: 3 (2 * 2 + 3) + 3 = 24 units of 2^-24, halved by the logarithm of
# the square root; the logarithm itself within 2 ulps.
TOLERANCE = 0.5 * 24 * 2.0 ** -24


def _ftle64(p, h):
    flow = p.astype(np.float64)
    J = np.stack([np.gradient(flow, h, axis=a, edge_order=1) for a in range(3)], -1)
    return 0.5 * np.log(np.linalg.eigvalsh(np.einsum("...ki,...kj->...ij", J, J))[..., -1])


def _run(ctx, p, h):
    from pars_gb300 import workloads as W
    f = W.Field(p, np.zeros(3, np.float32), np.full(3, h, np.float32))
    hnd = ctx.upload_field(f)
    out = ctx.ftle_generate(hnd, 1.0, 0, shape=p.shape[:3])
    ctx.release_field(hnd)
    return out


@pytest.mark.parametrize("name,singular", [
    ("isotropic", (1.0, 1.0, 1.0)), ("near_isotropic", (1.0, 1.0 + 1e-5, 1.0 - 2e-5)), ("two_largest", (3.0, 3.0 + 1e-6, 0.2)),
    ("two_smallest", (5.0, 0.3, 0.3)), ("spread", (40.0, 1.0, 0.02)), ("generic", (2.0, 1.0, 0.5)), ("large", (2e12, 1e12, 3e11)),
    ("small", (2e-12, 1e-12, 1e-12))])
def test_linear_maps(ctx, name, singular):
    rng = np.random.default_rng(len(name))
    h = np.float32(0.125)
    x = np.stack(np.meshgrid(*[np.arange(5) * float(h)] * 3, indexing="ij"), -1)
    for _ in range(24):
        q, r = (np.linalg.qr(rng.normal(size=(3, 3)))[0] for _ in range(2))
        p = (x @ (q @ np.diag(singular) @ r).T).astype(np.float32)
        got, ref = _run(ctx, p, h), _ftle64(p, float(h))
        assert np.all(np.abs(got - ref) <= TOLERANCE + 2.0 ** -22 * np.abs(ref))


def test_planar_and_degenerate_maps(ctx):
    h = np.float32(0.25)
    x = np.stack(np.meshgrid(*[np.arange(6) * float(h)] * 3, indexing="ij"), -1)
    for m in ([[2, 0.3, 0], [-0.7, 0.9, 0], [0, 0, 1]], [[0.5, 0, 0], [0, 0.5, 0], [0, 0, 1]], [[1, 0, 0], [0, 1, 0], [0, 0, 1]],
              [[3, 0, 0], [0, 1, 0], [0, 0, 2]], [[0, 0, 0], [0, 2, 0], [0, 0, 1]]):
        p = (x @ np.array(m, float).T).astype(np.float32)
        ref = _ftle64(p, float(h))
        assert np.all(np.abs(_run(ctx, p, h) - ref) <= TOLERANCE + 2.0 ** -22 * np.abs(ref))
    p = np.zeros((4, 5, 6, 3), np.float32)
    assert np.all(np.isneginf(_run(ctx, p, h)))                   # C = 0
    p = x.astype(np.float32)
    p[3, 3, 3] = np.nan
    got = _run(ctx, p, h)
    touched = np.zeros(got.shape, bool)
    for a in range(3):
        for s in (-1, 1):
            i = [3, 3, 3]
            i[a] += s
            touched[tuple(i)] = True
    assert np.all(np.isnan(got[touched])) and np.all(np.isfinite(got[~touched]))


@pytest.mark.parametrize("shape", [(2, 64, 64), (3, 63, 65), (3, 64, 65), (5, 2, 2048), (4, 2, 2049), (66000, 2, 2)])
def test_planes_and_ragged_lattices_against_fp64(ctx, shape):
    """Either side of the change from CTAs by plane to one row over all vertices."""
    rng = np.random.default_rng(sum(shape))
    h = 0.25
    grid = np.stack(np.meshgrid(*[np.arange(n) * h for n in shape], indexing="ij"), -1)
    p = (grid + 0.1 * rng.normal(size=grid.shape)).astype(np.float32)
    got, expected = _run(ctx, p, h), _ftle64(p, h)
    # relative to lambda: the logarithm's absolute error, and two ulps of its value
    assert np.all(np.abs(got - expected) <= TOLERANCE + 2.0 ** -22 * np.abs(expected))
