"""Launches that leave lanes of each warp unused: the same bits as the oracle on
either side of every change of the lanes per warp."""
import numpy as np
import pytest

from test_gpu_parity import compare, gpu_curves

pytestmark = pytest.mark.gpu


def _edges():
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    fill = 12 * sms
    return [1, 4 * sms, 4 * sms + 1, 4 * fill, 4 * fill + 1, 8 * fill + 1, 16 * fill + 1]


def _seeds(dtype, n, iterations):
    p = np.zeros(n, dtype)
    p["position"][:, :3] = np.random.default_rng(n).uniform(0.2, 6.1, (n, 3)).astype(np.float32)
    p["remaining_iterations"] = iterations
    p["vector_field_index"] = -1
    return p


@pytest.mark.parametrize("edge", range(7))
def test_streamlines_match_the_oracle(ctx, port, edge):
    from pars_gb300 import native, workloads as W
    f = W.abc_field(17)
    p = _seeds(native.PARTICLE_DTYPE, _edges()[edge], 22)
    h = ctx.upload_field(f)
    s = ctx.trace(h, p, 2, 0, 0.05)
    expected = port.trace_single(f, p, 2, 0.05, "rgb", 0.5)
    assert s["steps"] == expected.steps
    compare(gpu_curves(ctx, s, "rgb"), expected.batches)
    ctx.release_field(h)


@pytest.mark.parametrize("edge", range(7))
def test_domain_matches_the_oracle(ctx, port, edge):
    from pars_gb300 import native, workloads as W
    f = W.abc_field(17)
    ranks = 8
    info = port.partition(ranks, 0, f.dims)
    p = _seeds(native.PARTICLE_DTYPE, _edges()[edge], 22)
    extent = (f.spacing * info["block"]).astype(np.float32)
    multi = np.minimum((p["position"][:, :3] / extent).astype(np.int64), info["grid"] - 1)
    owner = (multi[:, 0] * info["grid"][1] + multi[:, 1]) * info["grid"][2] + multi[:, 2]
    p = p[np.argsort(owner, kind="stable")]
    offsets = np.concatenate([[0], np.cumsum(np.bincount(owner, minlength=ranks))]).astype(np.int64)
    d = ctx.domain_create(f, ranks)
    s = ctx.trace_domain(d, p, offsets, 2, 0, 0.05)
    expected = port.trace_multi(f, ranks, offsets, p, 2, 0.05, "rgb", 0.5)
    assert s["steps"] == expected.steps
    compare(gpu_curves(ctx, s, "rgb"), expected.batches)
    ctx.domain_release(d)


@pytest.mark.parametrize("n", [5, 700])
def test_curves_on_a_large_field_do_not_depend_on_the_launch(ctx, n):
    """Re-sampled RK4 on a field of more than 32 MB fetches cells ahead in a launch of few
    particles; beside many others the same particles go through another kernel."""
    from pars_gb300 import native, workloads as W
    f = W.abc_field(132)
    h = ctx.upload_field(f)
    few = _seeds(native.PARTICLE_DTYPE, n, 40)
    few["position"][: n // 2, :3] *= np.float32(0.02)   # near the faces: cells clamped, curves that leave
    filler = _seeds(native.PARTICLE_DTYPE, 300000, 2)
    curves = []
    for p in (few, np.concatenate([few, filler])):
        s = ctx.trace(h, p, 2, 1, 0.2)
        curves.append(ctx.curves(s["batches"], vertices=True)[0]["vertices"])
    assert np.array_equal(curves[0], curves[1][: len(curves[0])])
    ctx.release_field(h)
