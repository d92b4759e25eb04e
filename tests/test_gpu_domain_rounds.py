"""A partitioned domain of more rounds than the first read of their sizes holds: curves
that circle around an edge where four blocks meet."""
import numpy as np
import pytest

from test_gpu_parity import compare, gpu_curves

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turns", [1, 70])
def test_circling_curves_match_the_oracle(ctx, port, turns):
    from pars_gb300 import native, workloads as W
    f = W.abc_field(17)
    centre = 8 * f.spacing[0]
    x = np.arange(17, dtype=np.float32) * f.spacing[0] - centre
    f.xyz = np.zeros((17, 17, 17, 3), np.float32)
    f.xyz[..., 0] = -x[None, :, None]
    f.xyz[..., 1] = x[:, None, None]
    ranks, step = 8, 0.005
    p = np.zeros(5, native.PARTICLE_DTYPE)
    p["position"][:, 0] = centre + np.linspace(0.1, 0.5, 5)
    p["position"][:, 1] = centre + 0.01
    p["position"][:, 2] = 1.0
    p["remaining_iterations"] = int(turns * 2 * np.pi / step) + 2
    p["vector_field_index"] = -1
    info = port.partition(ranks, 0, f.dims)
    multi = np.minimum((p["position"][:, :3] / (f.spacing * info["block"])).astype(np.int64), info["grid"] - 1)
    owner = (multi[:, 0] * info["grid"][1] + multi[:, 1]) * info["grid"][2] + multi[:, 2]
    p = p[np.argsort(owner, kind="stable")]
    offsets = np.concatenate([[0], np.cumsum(np.bincount(owner, minlength=ranks))]).astype(np.int64)
    d = ctx.domain_create(f, ranks)
    s = ctx.trace_domain(d, p, offsets, 2, 0, step)
    assert s["rounds"] > (255 if turns > 1 else 3)
    expected = port.trace_multi(f, ranks, offsets, p, 2, step, "rgb", 0.5)
    assert s["steps"] == expected.steps
    compare(gpu_curves(ctx, s, "rgb"), expected.batches)
    ctx.domain_release(d)
