"""A field keeps each vertex's neighbouring z component beside its own; a flow map
keeps residual codes there.  Both layouts give the same bits, and the FTLE of an
uploaded flow map reads no codes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Field:
    def __init__(self, xyz, spacing):
        self.xyz = np.ascontiguousarray(xyz, np.float32)
        self.dims = np.array(xyz.shape[:3], np.int32)
        self.offset = np.zeros(3, np.float32)
        self.spacing = np.asarray(spacing, np.float32)
        self.size = (self.dims * self.spacing).astype(np.float32)


@pytest.mark.parametrize("stages,integrator", [(0, 2), (0, 0), (0, 6), (1, 2), (1, 0), (1, 4), (1, 6)])
def test_a_flow_map_is_traced_as_its_upload(ctx, stages, integrator):
    from pars_gb300 import native, workloads as W
    base = W.abc_field(19)
    h = ctx.upload_field(base)
    flow, _ = ctx.flow_map_generate(h, 12, 1.0, 2, 1, 0.05)
    same = ctx.upload_field(_Field(ctx.download_field(flow), base.spacing))
    a, sa = ctx.flow_map_generate(flow, 40, 1.0, integrator, stages, 0.01)
    b, sb = ctx.flow_map_generate(same, 40, 1.0, integrator, stages, 0.01)
    assert sa == sb > 0 and np.array_equal(ctx.download_field(a), ctx.download_field(b))
    p = np.zeros(300, native.PARTICLE_DTYPE)
    p["position"][:, :3] = np.random.default_rng(1).uniform(0.3, 6.0, (300, 3)).astype(np.float32)
    p["remaining_iterations"], p["vector_field_index"] = 40, -1
    curves = []
    for field in (flow, same):
        s = ctx.trace(field, p, integrator, stages, 0.01)
        curves.append(ctx.curves(s["batches"], vertices=True))
    for x, y in zip(*curves):
        assert np.array_equal(x["vertices"], y["vertices"])
    for field in (h, flow, same, a, b):
        ctx.release_field(field)


def test_an_uploaded_flow_map_has_no_residuals(ctx):
    """Frozen flow maps store no codes, so their upload has the same FTLE."""
    from pars_gb300 import workloads as W
    base = W.abc_field(21)
    h = ctx.upload_field(base)
    flow, _ = ctx.flow_map_generate(h, 60, 1.0, 2, 0, 0.05)
    same = ctx.upload_field(_Field(ctx.download_field(flow), base.spacing))
    shape = tuple(int(n) for n in ctx.field_info(flow)["shape"])
    assert np.array_equal(ctx.ftle_generate(flow, 3.0, shape=shape), ctx.ftle_generate(same, 3.0, shape=shape))
    for field in (h, flow, same):
        ctx.release_field(field)
