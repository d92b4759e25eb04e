"""The flow-map kernel's step count beyond 32 bits in one warp: 32 particles that stay where
they are for 135 million steps each (about half a minute: nothing shorter reaches 2^32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_warp_of_more_than_2_to_32_steps(ctx):
    from pars_gb300 import native, workloads as W
    xyz = np.zeros((2, 2, 33, 3), np.float32)
    xyz[..., 0] = 1e-3
    h = ctx.upload_field(W.Field(xyz, np.ones(3, np.float32), np.ones(3, np.float32)))
    steps = (2 ** 32 + 2 ** 20) // 32
    flow, taken = ctx.flow_map_generate(h, steps + 1, 1.0, native.INTEGRATORS["adams_bashforth_2"], native.STAGES_RESAMPLED, 1e-20)
    ctx.release_field(flow)
    ctx.release_field(h)
    assert taken == 32 * steps
