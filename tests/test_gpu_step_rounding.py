"""Re-sampled Euler and Adams-Bashforth steps round alike in every kernel that takes them: end
positions (and streamlines) on a field of exact binary fractions, as checksums of the bits
that per-seed kernels of one particle per thread gave."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHECKSUMS = {
    "map euler 40 40": 0x6871ee70,
    "map euler 40 130": 0x852fdb0b,
    "map adams_bashforth_2 40 40": 0xf81dd964,
    "map adams_bashforth_2 40 130": 0x443c8b33,
    "map adams_bashforth_moulton_2 40 40": 0x91724519,
    "map adams_bashforth_moulton_2 40 130": 0x99d8af47,
    "curves euler 40 600": 0x67d53896,
    "curves adams_bashforth_2 40 600": 0xc138ced9,
    "curves euler 40 150000": 0x5ccaf4ba,
    "curves adams_bashforth_2 40 150000": 0x5904f6d5,
    "map euler 100 40": 0x10274309,
    "map euler 100 130": 0xfd8db2c4,
    "map adams_bashforth_2 100 40": 0x4cf6232b,
    "map adams_bashforth_2 100 130": 0xa9717d07,
    "map adams_bashforth_moulton_2 100 40": 0x6870c9d4,
    "map adams_bashforth_moulton_2 100 130": 0x62badca0,
    "curves euler 100 600": 0x9ecdc1a3,
    "curves adams_bashforth_2 100 600": 0xeba85c78,
    "curves euler 100 150000": 0xba72c27c,
    "curves adams_bashforth_2 100 150000": 0x2a59fac8,
}


def _field(edge):
    from pars_gb300 import workloads as W
    rng = np.random.default_rng(11)
    xyz = (rng.integers(-512, 513, (edge, edge, edge, 3)) + np.array([300, -200, 100])).astype(np.float32) / np.float32(256)
    return W.Field(xyz, np.array([0.5, -1.0, 2.0], np.float32), np.full(3, np.float32(0.25)))


def _crc(a):
    return zlib.crc32(np.ascontiguousarray(a).view(np.uint8).reshape(-1))


def results(ctx):
    from pars_gb300 import native
    out = {}
    for edge in (40, 100):
        h = ctx.upload_field(_field(edge))
        for name in ("euler", "adams_bashforth_2", "adams_bashforth_moulton_2"):
            for iterations in (40, 130):
                fm, _ = ctx.flow_map_generate(h, iterations, 1.0, native.INTEGRATORS[name], native.STAGES_RESAMPLED, 0.01)
                out[f"map {name} {edge} {iterations}"] = _crc(ctx.download_field(fm))
                ctx.release_field(fm)
        for count in (600, 150000):
            p = np.zeros(count, native.PARTICLE_DTYPE)
            p["position"][:, :3] = [0.5, -1.0, 2.0] + np.random.default_rng(count).integers(1, 256 * (edge - 1) // 4, (count, 3)) / 256.0
            p["remaining_iterations"], p["vector_field_index"] = 60, -1
            for name in ("euler", "adams_bashforth_2"):
                s = ctx.trace(h, p, native.INTEGRATORS[name], native.STAGES_RESAMPLED, 0.01)
                out[f"curves {name} {edge} {count}"] = _crc(ctx.curves(s["batches"], vertices=True)[0]["vertices"])
        ctx.release_field(h)
    return out


def test_steps_round_alike(ctx):
    got = results(ctx)
    assert got == CHECKSUMS, {k: (hex(v), k) for k, v in got.items() if CHECKSUMS.get(k) != v}
