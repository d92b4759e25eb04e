"""What a user of this framework has it do, as timed cases.

Each case is one pass through the public entry points of ``pars_gb300`` (the
Python binding, or the C functions of include/pars_gpu.h where a program passes
buffers of its own).  The flows are the ones of ``pars_gb300.workloads``: the
ABC flow with noise and the 3-D double gyre, here with amplitudes, phases and
noise drawn from the seed.  Kinds of case:

streamlines  trace, index, colour; the curves come back into pinned host
             buffers (a program that keeps or exports the curves).
image        the same, then the ray tracer; the image comes back (the reply
             of pars_service to a streamline request).
domain       a domain partitioned into blocks on one GPU, traced through all
             rounds, indexed, coloured and ray traced.
viewer       a resident scene (curves, maybe a volume) seen from the camera of
             the moment: set_camera, trace, serialize.
ftle         flow map and FTLE of a resident field; the FTLE stays on the GPU.
insitu       the allocation-free FTLE entry point, field and result on the GPU.
flow_map     a flow map with one of the higher-order integrators, downloaded.
ftle_stage   the FTLE stage alone, on a flow map of the caller's.
pathlines    a batch of unsteady fields advected in one call.
service      requests submitted to the two-lane service, replies collected.
"""
import ctypes
import math

import numpy as np
import torch

from pars_gb300 import native, workloads
from pars_gb300.requests import encode_settings

RK4_STEP_FLOPS = 330          # four trilinear samples and the weighted sum
FROZEN_STEP_FLOPS = 90        # one trilinear sample
UNSTEADY_STEP_FLOPS = 640     # four samples in two time slices each
STAGES = {"modified_midpoint": 3, "runge_kutta_cash_karp_54": 6, "runge_kutta_dormand_prince_5": 6,
          "runge_kutta_fehlberg_78": 13, "adams_bashforth_2": 1, "adams_bashforth_moulton_2": 2}


def listed():
    return [
        # The plain streamline workload: few curves, 1000 dependent steps, small
        # launches around them; latency is all of it.
        {"name": "streamlines_64", "kind": "streamlines", "flow": "abc", "nx": 64, "ny": 64, "nz": 64, "stride": 4,
         "steps": 1000, "stages": "resampled", "integrator": "runge_kutta_4", "color": "rgb", "parameter": 0.5},
        # A streamline request in the reference's own scheme (frozen stages, bit
        # for bit), on a ragged grid, replied to with an image.
        {"name": "image_reference", "kind": "image", "flow": "abc", "nx": 141, "ny": 97, "nz": 118, "stride": 6,
         "steps": 800, "stages": "frozen", "integrator": "runge_kutta_4", "color": "hsv_constant_s", "parameter": 0.75,
         "width": 960, "height": 540},
        # The largest requests of the served stream: long curves that stay in the
        # domain, a scene of many millions of capsules, a full-size image.
        {"name": "image_large", "kind": "image", "flow": "gyre", "nx": 198, "ny": 198, "nz": 198, "stride": 9,
         "steps": 1000, "stages": "resampled", "integrator": "runge_kutta_4", "color": "hsv_constant_s", "parameter": 0.75,
         "width": 1080, "height": 1920},
        # The partitioned domain, 64 blocks on one GPU, with clustered seeds.
        {"name": "domain_256", "kind": "domain", "n": 256, "ranks": 64, "seeds": 100000, "steps": 1000,
         "stages": "resampled", "color": "rgb", "parameter": 0.5, "width": 960, "height": 540},
        # A viewer moving its camera around curves inside a volume, at the
        # benchmark generator's image size.
        {"name": "viewer_volume", "kind": "viewer", "flow": "abc", "nx": 64, "ny": 64, "nz": 64, "stride": 4,
         "steps": 1000, "volume": True, "frames": 1, "width": 1080, "height": 1920},
        # The headline: FTLE of a 256^3 field, one seed per vertex, T = 5.
        {"name": "ftle_256", "kind": "ftle", "flow": "abc", "nx": 256, "ny": 256, "nz": 256, "steps": 500,
         "stages": "resampled", "integrator": "runge_kutta_4", "mode": "regular", "scale": 1.0},
        # The reference's FTLE (frozen stages) on a ragged grid.
        {"name": "ftle_reference", "kind": "ftle", "flow": "abc", "nx": 150, "ny": 128, "nz": 141, "steps": 300,
         "stages": "frozen", "integrator": "runge_kutta_4", "mode": "regular", "scale": 1.0},
        # A plugin inside a host application: the smallest call.
        {"name": "insitu_64", "kind": "insitu", "flow": "abc", "nx": 61, "ny": 64, "nz": 67, "steps": 120,
         "stages": "resampled", "integrator": "runge_kutta_4", "mode": "regular"},
        # A higher-order integrator with stages sampled where they fall.
        {"name": "flow_map_dopri5", "kind": "flow_map", "flow": "abc", "nx": 96, "ny": 90, "nz": 101, "steps": 200,
         "integrator": "runge_kutta_dormand_prince_5"},
        # The FTLE stage on a flow map that another program computed.
        {"name": "ftle_stage", "kind": "ftle_stage", "nx": 320, "ny": 300, "nz": 311, "mode": "regular"},
        # Pathlines: several unsteady fields of different sizes in one call.
        {"name": "pathlines_6", "kind": "pathlines", "fields": 6, "edge_lo": 32, "edge_hi": 128, "slices": 24,
         "seeds_lo": 4000, "seeds_hi": 120000, "steps": 400, "layout": 3},
        # A burst of mixed requests to the service.
        {"name": "service_16", "kind": "service", "requests": 16, "edge_lo": 75, "edge_hi": 160, "steps_lo": 200,
         "steps_hi": 1000, "seeds_lo": 1000, "seeds_hi": 12000, "voxels_hi": 500000, "width": 960, "height": 540, "layout": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A ragged grid: an edge spread over its logarithm, each axis within a quarter of it."""
    e = _log(rng, lo, hi)
    return {k: max(lo, min(hi, int(e * rng.uniform(0.8, 1.25)))) for k in ("nx", "ny", "nz")}


def draw(rng):
    """One more case.  Every kind, weighted towards the ones with most options."""
    kind = rng.choice(["streamlines", "image", "image", "domain", "viewer", "ftle", "ftle", "insitu", "flow_map", "ftle_stage",
                       "pathlines", "service"])
    stages = rng.choice(["frozen", "resampled"])
    integrators = ["runge_kutta_4"] * 3 + ["euler"] + sorted(STAGES)
    colours = ["rgb", "hsl_constant_s", "hsl_constant_l", "hsv_constant_s", "hsv_constant_v"]
    flow = rng.choice(["abc", "gyre"])
    color = {"color": rng.choice(colours), "parameter": round(rng.uniform(0.2, 0.9), 2)}
    view = dict(zip(("width", "height"), rng.choice([(960, 540), (640, 481), (1080, 1920), (333, 250)])))
    if kind in ("streamlines", "image"):
        grid = _grid(rng, 33, 198)
        smallest = min(grid.values())
        target = _log(rng, 512, 5000 if kind == "streamlines" else 12000)      # seeds
        stride = max(2, round((grid["nx"] * grid["ny"] * grid["nz"] / target) ** (1.0 / 3.0)))
        case = {"kind": kind, "flow": flow, **grid, "stride": min(stride, smallest // 4), "steps": _log(rng, 100, 1000), "stages": stages,
                "integrator": rng.choice(integrators), **color}
        return {**case, **view} if kind == "image" else case
    if kind == "domain":
        return {"kind": kind, "n": _log(rng, 64, 256), "ranks": rng.choice([8, 27, 64]), "seeds": _log(rng, 5000, 100000),
                "steps": _log(rng, 200, 1000), "stages": stages, **color, **view}
    if kind == "viewer":
        grid = _grid(rng, 48, 96)
        return {"kind": kind, "flow": flow, **grid, "stride": rng.choice([4, 5, 6]), "steps": _log(rng, 200, 1000),
                "volume": rng.random() < 0.5, "frames": rng.choice([1, 1, 2, 4]), **view}
    if kind == "ftle":
        return {"kind": kind, "flow": flow, **_grid(rng, 40, 200), "steps": _log(rng, 50, 400), "stages": stages,
                "integrator": rng.choice(["runge_kutta_4", "runge_kutta_4", "euler"]),
                "mode": rng.choice(["regular", "regular", "fractional_anisotropy"]), "scale": rng.choice([1.0, 1.0, 0.5])}
    if kind == "insitu":
        return {"kind": kind, "flow": flow, **_grid(rng, 24, 62), "steps": _log(rng, 20, 300), "stages": stages,
                "integrator": rng.choice(["runge_kutta_4", "runge_kutta_4", "euler"] + sorted(STAGES)),
                "mode": rng.choice(["regular", "fractional_anisotropy"])}
    if kind == "flow_map":
        return {"kind": kind, "flow": flow, **_grid(rng, 32, 101), "steps": _log(rng, 40, 250), "integrator": rng.choice(sorted(STAGES))}
    if kind == "ftle_stage":
        return {"kind": kind, **_grid(rng, 24, 310), "mode": rng.choice(["regular", "regular", "fractional_anisotropy"])}
    if kind == "pathlines":
        return {"kind": kind, "fields": rng.randint(2, 8), "edge_lo": 32, "edge_hi": _log(rng, 48, 128), "slices": rng.randint(2, 32),
                "seeds_lo": 1000, "seeds_hi": _log(rng, 4000, 120000), "steps": _log(rng, 100, 400), "layout": rng.randint(5, 99999)}
    return {"kind": "service", "requests": rng.randint(4, 16), "edge_lo": 64, "edge_hi": _log(rng, 80, 160), "steps_lo": 200,
            "steps_hi": _log(rng, 300, 1000), "seeds_lo": 1000, "seeds_hi": _log(rng, 2000, 12000),
            "voxels_hi": _log(rng, 20000, 500000), "width": view["width"], "height": view["height"], "layout": rng.randint(5, 99999)}


# ---- inputs --------------------------------------------------------------------------
def _uniform(generator, lo, hi, n):
    return (torch.rand(n, generator=generator, device="cuda", dtype=torch.float64) * (hi - lo) + lo).tolist()


def _extent(n, spacing):
    """shape * spacing in FP32, an ulp up where size / spacing would round below the shape (one seed per vertex)."""
    size = (np.array(n, np.float32) * spacing).astype(np.float32)
    return np.where(size / spacing < np.array(n, np.float32), np.nextafter(size, np.float32(np.inf)), size).astype(np.float32)


def _field(flow, n, seed):
    """A steady field of `flow` on the grid n: (xyz [nx, ny, nz, 3] FP32 on the
    GPU, offset, size, spacing).  ABC: [0, 2 pi] along the longest axis, the
    amplitudes and phases of the seed, N(0, 0.01) noise; gyre: one time slice
    on [0, 2] x [0, 1] x [0, 1]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.empty((*n, 3), dtype=torch.float32, device="cuda")
    if flow == "abc":
        h = 2.0 * math.pi / (max(n) - 1)
        spacing = np.full(3, h, np.float32)
        px, py, pz, a, b, c = _uniform(g, 0.0, 1.0, 6)
        x, y, z = (torch.arange(m, device="cuda", dtype=torch.float64) * h for m in n)
        x, y, z = (x + 0.5 * px)[:, None, None], (y + 0.5 * py)[None, :, None], (z + 0.5 * pz)[None, None, :]
        A, B, C = math.sqrt(3.0) * (0.95 + 0.1 * a), math.sqrt(2.0) * (0.95 + 0.1 * b), 0.95 + 0.1 * c
        out[..., 0] = A * torch.sin(z) + C * torch.cos(y)
        out[..., 1] = B * torch.sin(x) + A * torch.cos(z)
        out[..., 2] = C * torch.sin(y) + B * torch.cos(x)
        out.add_(torch.randn(out.shape, generator=g, device="cuda"), alpha=0.01)
    else:
        spacing = np.array([2.0 / (n[0] - 1), 1.0 / (n[1] - 1), 1.0 / (n[2] - 1)], np.float32)
        t, a = _uniform(g, 0.0, 10.0, 1)[0], 0.1 * (0.9 + 0.2 * _uniform(g, 0.0, 1.0, 1)[0])
        out[:] = _gyre(n, t, a)
    size = _extent(n, spacing)
    return out, np.zeros(3, np.float32), size, spacing


def _gyre(n, t, a):
    x = torch.linspace(0.0, 2.0, n[0], dtype=torch.float64, device="cuda")[:, None, None]
    y = torch.linspace(0.0, 1.0, n[1], dtype=torch.float64, device="cuda")[None, :, None]
    s = 0.25 * math.sin(0.2 * math.pi * t)
    f, df = s * x * x + (1.0 - 2.0 * s) * x, 2.0 * s * x + (1.0 - 2.0 * s)
    v = torch.zeros((*n, 3), dtype=torch.float32, device="cuda")
    v[..., 0] = -math.pi * a * torch.sin(math.pi * f) * torch.cos(math.pi * y)
    v[..., 1] = math.pi * a * torch.cos(math.pi * f) * torch.sin(math.pi * y) * df
    return v


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _step(case):
    return 0.05 if case.get("flow") == "gyre" else 0.01


def _flow_map_input(case, seed):
    """A smooth flow map as a caller might bring it: every vertex moved by a few
    displacement waves (amplitudes up to a cell's neighbourhood of folding)."""
    n = _shape(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    spacing = np.full(3, 2.0 * math.pi / (max(n) - 1), np.float32)
    h = float(spacing[0])
    x, y, z = (torch.arange(m, device="cuda", dtype=torch.float32) * h for m in n)
    p = torch.empty((*n, 3), dtype=torch.float32, device="cuda")
    ph = _uniform(g, 0.0, 2.0 * math.pi, 6)
    k = [int(round(v)) for v in _uniform(g, 2.0, 9.0, 6)]
    p[..., 0] = x[:, None, None] + 0.3 * torch.sin(k[0] * y + ph[0])[None, :, None] + 0.2 * torch.cos(k[1] * z + ph[1])[None, None, :]
    p[..., 1] = y[None, :, None] + 0.3 * torch.sin(k[2] * z + ph[2])[None, None, :] + 0.2 * torch.cos(k[3] * x + ph[3])[:, None, None]
    p[..., 2] = z[None, None, :] + 0.3 * torch.sin(k[4] * x + ph[4])[:, None, None] + 0.2 * torch.cos(k[5] * y + ph[5])[None, :, None]
    size = _extent(n, spacing)
    return p, np.zeros(3, np.float32), size, spacing


def _pathline_jobs(case, seed):
    """(slices [s, e, e, e, 3], spacing, dt, seeds [m, 4]) of every job; the sizes come from the case, the values from the seed."""
    rng = np.random.default_rng(case["layout"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    period, jobs = 10.0, []
    for _ in range(case["fields"]):
        e = int(np.exp(rng.uniform(np.log(case["edge_lo"]), np.log(case["edge_hi"]))))
        m = int(np.exp(rng.uniform(np.log(case["seeds_lo"]), np.log(case["seeds_hi"]))))
        slices = max(2, int(case["slices"] * rng.uniform(0.7, 1.3)))
        a = 0.1 * (0.9 + 0.2 * _uniform(g, 0.0, 1.0, 1)[0])
        dt = period / (slices - 1)
        xyz = torch.stack([_gyre((e, e, e), k * dt, a) for k in range(slices)])
        spacing = np.array([2.0 / (e - 1), 1.0 / (e - 1), 1.0 / (e - 1)], np.float32)
        seeds = torch.rand((m, 4), generator=g, device="cuda")
        seeds[:, 0] *= 2.0
        seeds[:, 3] = 0.0
        jobs.append((xyz, spacing, dt, seeds))
    return jobs


def _service_plan(case):
    """Datasets (flow, edge) and requests (kind, dataset, stride, steps) of the case: 70 % streamlines, 30 % FTLE."""
    rng = np.random.default_rng(case["layout"])
    datasets = []
    for k in range(3):
        datasets.append(("abc" if k == 0 else "gyre", int(np.exp(rng.uniform(np.log(case["edge_lo"]), np.log(case["edge_hi"]))))))
    requests = []
    for k in range(case["requests"]):
        d = int(rng.integers(0, 3))
        edge = datasets[d][1]
        kind = "ftle" if k % 10 in (2, 5, 8) else "streamlines"
        top = case["voxels_hi"] if kind == "ftle" else case["seeds_hi"]
        seeds = np.exp(rng.uniform(np.log(case["seeds_lo"]), np.log(top)))
        stride = max(1, int(np.ceil(edge / seeds ** (1.0 / 3.0))))
        requests.append((kind, d, stride, int(rng.integers(case["steps_lo"], case["steps_hi"] + 1))))
    return datasets, requests


# ---- state ----------------------------------------------------------------------------
class State:
    """What a program holds before the call; gives its handles back when dropped."""

    def __init__(self, case):
        self.case = dict(case)
        self.ctx = None
        self.fields = []
        self.domain = None
        self.own = False
        self.buffers = {}

    def pinned(self, name, count, dtype):
        """A pinned host buffer of `count` elements, kept."""
        b = self.buffers.get(name)
        if b is None or b.numel() != count:
            b = self.buffers[name] = torch.zeros(count, dtype=dtype, pin_memory=True)
        return b

    def __del__(self):
        try:
            if self.domain is not None:
                self.ctx.domain_release(self.domain)
            for h in self.fields:
                self.ctx.release_field(h)
            if self.own:
                self.ctx.close()
        except Exception:
            pass


_shared = None


def _context():
    """The program's context: one for the process."""
    global _shared
    if _shared is None:
        _shared = native.Context(0)
    return _shared


class _OnDevice:
    """A device buffer of the library's, as torch takes it."""

    def __init__(self, pointer, shape, typestr="<f4"):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (pointer, False), "version": 2}


def _upload(ctx, s, xyz, offset, size, spacing):
    h = ctx.upload_field_device(xyz.data_ptr(), tuple(xyz.shape[:3]), offset, size, spacing)
    s.fields.append(h)
    return h


def _camera(size):
    """In front of the domain, looking along +z (fovy 68 degrees)."""
    centre = size / 2.0
    return (float(centre[0]), float(centre[1]), float(-1.45 * max(size[0], size[1]))), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0)


def _stages(case):
    return native.STAGES_FROZEN if case["stages"] == "frozen" else native.STAGES_RESAMPLED


def prepare(case, seed):
    s = State(case)
    kind = case["kind"]
    if kind == "viewer":
        s.ctx, s.own = native.Context(0), True     # a viewer keeps its scene in a context of its own
    else:
        s.ctx = _context()
    ctx = s.ctx
    if kind in ("streamlines", "image", "viewer"):
        xyz, offset, size, spacing = _field(case["flow"], _shape(case), seed)
        s.field = _upload(ctx, s, xyz, offset, size, spacing)
        stride = (spacing * np.float32(case["stride"])).astype(np.float32)
        s.seeds = ctx.seed_generate(offset, size, stride, case["steps"] + 2)
        s.camera, s.radius = _camera(size), float(np.float32(0.1) * spacing[0])
        if kind == "streamlines":
            # room for every curve at its full length (seed, steps, termination vertex); what a pass does not fill stays 0
            n = len(s.seeds) * (case["steps"] + 2)
            s.vertices, s.colors = s.pinned("v", 4 * n, torch.float32).view(-1, 4), s.pinned("c", 4 * n, torch.float32).view(-1, 4)
            s.indices = s.pinned("i", n, torch.int32)
        if kind == "viewer":
            ctx.trace(s.field, s.seeds, native.RUNGE_KUTTA_4, native.STAGES_RESAMPLED, _step(case))
            ctx.curves_index()
            ctx.curves_color("hsv_constant_s", 0.75)
            ctx.ray_tracer_set_integral_curves(s.radius)
            if case["volume"]:
                speed = torch.linalg.vector_norm(xyz, dim=-1)
                s.volume = (speed / speed.max()).contiguous()
                torch.cuda.synchronize()
                ctx.ray_tracer_set_volume_device(s.volume.data_ptr(), _shape(case), offset, spacing)
            ctx.ray_tracer_set_image_size(case["width"], case["height"])
    elif kind == "domain":
        n = case["n"]
        xyz, spacing = workloads.beltrami_fourier_device(torch, n, seed=seed)
        s.domain = ctx.domain_create_device(xyz.data_ptr(), (n, n, n), spacing, case["ranks"])
        part = native.partition(case["ranks"], 0, (n, n, n))
        s.seeds, s.offsets = workloads.gaussian_mixture_seeds(case["seeds"], n, spacing, part, remaining=case["steps"] + 2, seed=seed)
        s.camera = _camera(_extent((n, n, n), spacing))
        s.radius = float(np.float32(0.1) * spacing[0])
    elif kind in ("ftle", "flow_map"):
        s.field = _upload(ctx, s, *_field(case["flow"], _shape(case), seed))
    elif kind == "insitu":
        s.xyz, s.offset, s.size, s.spacing = _field(case["flow"], _shape(case), seed)
        s.dims = np.array(_shape(case), np.int32)
        s.out = torch.empty(_shape(case), dtype=torch.float32, device="cuda")
        s.steps = torch.zeros(1, dtype=torch.int64, device="cuda")
    elif kind == "ftle_stage":
        s.flow_map = _upload(ctx, s, *_flow_map_input(case, seed))
    elif kind == "pathlines":
        s.jobs, s.ends, s.seeds = [], [], []
        for xyz, spacing, dt, seeds in _pathline_jobs(case, seed):
            n = xyz.shape[1:4]
            size = _extent(n, spacing)
            h = ctx.upload_unsteady_field_device(xyz.data_ptr(), n, xyz.shape[0], np.zeros(3, np.float32), size, spacing, 0.0, dt)
            s.fields.append(h)
            j = native.BatchJob()
            j.field, j.integrator, j.stage_mode = h, native.RUNGE_KUTTA_4, native.STAGES_RESAMPLED
            j.max_steps, j.step_size, j.time_begin = case["steps"], 0.01, 0.0
            end = torch.empty_like(seeds)
            j.seeds, j.seed_count, j.end_positions, j.end_steps = seeds.data_ptr(), len(seeds), end.data_ptr(), None
            s.jobs.append(j)
            s.ends.append(end)
            s.seeds.append(seeds)
    else:
        datasets, requests = _service_plan(case)
        s.service = native.Service(0, budget_bytes=8 << 30, lanes=2, max_batch=64)
        sizes = []
        for k, (flow, edge) in enumerate(datasets):
            xyz, offset, size, spacing = _field(flow, (edge,) * 3, seed * 16 + k)
            s.service.add_dataset_device(f"field{k}", xyz.data_ptr(), (edge,) * 3, offset, size, spacing)
            sizes.append((size, spacing, _step({"flow": flow})))
        s.messages = []
        for what, d, stride, steps in requests:
            size, spacing, step = sizes[d]
            m = {"mode": what, "dataset_filepath": f"field{d}", "seed_generation_stride": [stride] * 3,
                 "seed_generation_iterations": steps + (2 if what == "streamlines" else 1),
                 "particle_tracing_integrator": "runge_kutta_4", "particle_tracing_step_size": step,
                 "color_generation_mode": "hsv_constant_s", "color_generation_free_parameter": 0.75}
            if what == "streamlines":
                position, forward, up = _camera(size)
                m.update({"raytracing_camera_position": list(position), "raytracing_camera_forward": list(forward),
                          "raytracing_camera_up": list(up), "raytracing_image_size": [case["width"], case["height"]],
                          "raytracing_streamline_radius": float(np.float32(0.1) * spacing[0]), "raytracing_iterations": 1})
            s.messages.append(encode_settings(m))
    torch.cuda.synchronize()      # the inputs are there before the first call
    return s


# ---- one pass --------------------------------------------------------------------------
def _image(s, frames=1):
    """trace and serialize of the scene as set; the image in a pinned host buffer."""
    c = s.case
    s.ctx.ray_tracer_trace(frames)
    frame = s.pinned("frame", c["width"] * c["height"] * 4, torch.uint8)
    return s.ctx.ray_tracer_serialize(out=frame.numpy().reshape(c["height"], c["width"], 4))


def _render_curves(s):
    c, ctx = s.case, s.ctx
    ctx.curves_index()
    ctx.curves_color(c["color"], c["parameter"])
    ctx.ray_tracer_set_image_size(c["width"], c["height"])
    ctx.ray_tracer_set_camera(*s.camera)
    ctx.ray_tracer_clear_volume()
    ctx.ray_tracer_set_integral_curves(s.radius)
    return _image(s)


def run(s):
    c, ctx = s.case, s.ctx
    kind = c["kind"]
    if kind in ("streamlines", "image"):
        summary = ctx.trace(s.field, s.seeds, native.INTEGRATORS[c["integrator"]], _stages(c), _step(c))
        if kind == "image":
            return _render_curves(s)
        ctx.curves_index()
        ctx.curves_color(c["color"], c["parameter"])
        download, av, ai = native.library().pars_gpu_curves_download, 0, 0
        for b in range(summary["batches"]):
            nv, ni, _, _ = ctx.batch_info(b)
            status = download(ctx.handle, b, s.vertices.data_ptr() + 16 * av, s.colors.data_ptr() + 16 * av, s.indices.data_ptr() + 4 * ai)
            if status:
                raise native.ParsGpuError(status, "pars_gpu_curves_download")
            av, ai = av + nv, ai + ni
        return {"vertices": s.vertices, "colors": s.colors, "indices": s.indices}
    if kind == "domain":
        ctx.trace_domain(s.domain, s.seeds, s.offsets, native.RUNGE_KUTTA_4, _stages(c), 0.005)
        return _render_curves(s)
    if kind == "viewer":
        ctx.ray_tracer_set_camera(*s.camera)
        return _image(s, c["frames"])
    if kind == "ftle":
        fm, _ = ctx.flow_map_generate(s.field, c["steps"] + 1, c["scale"], native.INTEGRATORS[c["integrator"]], _stages(c), _step(c))
        shape = tuple(int(v) for v in ctx.field_info(fm)["shape"])
        ctx.ftle_generate(fm, c["steps"] * _step(c), _mode(c), download=False)
        ctx.release_field(fm)
        return torch.as_tensor(_OnDevice(ctx.ftle_device_pointer()[0], shape), device="cuda")
    if kind == "insitu":
        stream = torch.cuda.current_stream().cuda_stream
        status = native.library().pars_gpu_ftle_no_alloc(
            s.xyz.data_ptr(), s.dims.ctypes.data, s.offset.ctypes.data, s.size.ctypes.data, s.spacing.ctypes.data, c["steps"] + 1,
            native.INTEGRATORS[c["integrator"]], _stages(c), ctypes.c_float(_step(c)), ctypes.c_float(c["steps"] * _step(c)), _mode(c),
            s.out.data_ptr(), s.steps.data_ptr(), stream)
        if status:
            raise native.ParsGpuError(status, "pars_gpu_ftle_no_alloc")
        return {"ftle": s.out, "steps": s.steps}
    if kind == "flow_map":
        fm, steps = ctx.flow_map_generate(s.field, c["steps"] + 1, 1.0, native.INTEGRATORS[c["integrator"]], native.STAGES_RESAMPLED,
                                          _step(c))
        n = c["nx"] * c["ny"] * c["nz"]
        out = s.pinned("flow", 3 * n, torch.float32)
        status = native.library().pars_gpu_field_download(ctx.handle, fm, out.data_ptr())
        ctx.release_field(fm)
        if status:
            raise native.ParsGpuError(status, "pars_gpu_field_download")
        return {"flow_map": out.view(*_shape(c), 3), "steps": steps}
    if kind == "ftle_stage":
        ctx.ftle_generate(s.flow_map, 5.0, _mode(c), download=False)
        return torch.as_tensor(_OnDevice(ctx.ftle_device_pointer()[0], _shape(c)), device="cuda")
    if kind == "pathlines":
        steps = ctx.batch_advect(s.jobs)
        return {"positions": [e[:, :3] for e in s.ends], "steps": steps}     # w holds the coordinates' residual codes
    tickets = [s.service.submit(m) for m in s.messages]
    out, lib = [], native.library()
    for k, t in enumerate(tickets):
        s.service.wait(t)
        info = s.service.info(t)
        if info.kind == 0:
            n = info.image_size[0] * info.image_size[1] * 4
            b = s.pinned(f"r{k}", n, torch.uint8)
            s.service.image_into(t, b.data_ptr())
            out.append(b.view(info.image_size[1], info.image_size[0], 4))
        else:
            shape = tuple(info.ftle_shape)
            n = shape[0] * shape[1] * shape[2]
            b = s.pinned(f"r{k}", n, torch.float32)
            s.service.ftle_into(t, b.data_ptr())
            out.append(b.view(*shape))
        s.service.release(t)
    return out


def _mode(case):
    return native.FTLE_REGULAR if case["mode"] == "regular" else native.FTLE_FRACTIONAL_ANISOTROPY


# ---- work -------------------------------------------------------------------------------
def _steps_taken(case, seeds, step=None):
    """Particle-steps, estimated: in the ABC flow a particle is inside the box
    for about 1.3 time units on average (it leaves through a face); in the gyre
    it stays."""
    per = case["steps"] if case.get("flow") == "gyre" else min(case["steps"], 1.3 / (step or _step(case)))
    return seeds * per


def _step_flops(case):
    if case.get("stages") == "frozen":
        return FROZEN_STEP_FLOPS
    name = case.get("integrator", "runge_kutta_4")
    return RK4_STEP_FLOPS if name == "runge_kutta_4" else 80 * STAGES.get(name, 1) + 20


def work(case):
    kind = case["kind"]
    voxels = case["nx"] * case["ny"] * case["nz"] if "nx" in case else 0
    if kind in ("streamlines", "image"):
        seeds = voxels / case["stride"] ** 3
        steps = _steps_taken(case, seeds)
        out = 36 * steps if kind == "streamlines" else 4 * case["width"] * case["height"]
        return {"bytes": 12 * voxels + 48 * seeds + out, "flops": steps * (_step_flops(case) + (60 if kind == "image" else 20))}
    if kind == "domain":
        steps = _steps_taken(case, case["seeds"], 0.005)
        return {"bytes": 12 * case["n"] ** 3 + 48 * case["seeds"] + 4 * case["width"] * case["height"], "flops": steps * (_step_flops(case) + 60)}
    if kind == "viewer":
        segments = _steps_taken(case, voxels / case["stride"] ** 3)
        pixels = case["width"] * case["height"]
        samples = 2 * min(_shape(case)) if case["volume"] else 0      # two samples a cell, through the volume
        return {"bytes": 32 * segments + (4 * voxels if case["volume"] else 0) + 4 * pixels,
                "flops": case["frames"] * (60 * segments + pixels * (60 + 0.5 * samples * 40))}
    if kind in ("ftle", "insitu", "flow_map"):
        out = voxels * case.get("scale", 1.0) ** 3
        steps = _steps_taken(case, out)
        flops = steps * _step_flops({**case, "stages": case.get("stages", "resampled")})
        return {"bytes": 12 * voxels + out * (12 if kind == "flow_map" else 4), "flops": flops + (0 if kind == "flow_map" else 150 * out)}
    if kind == "ftle_stage":
        return {"bytes": 16 * voxels, "flops": 150 * voxels}
    if kind == "pathlines":
        rng, b, f = np.random.default_rng(case["layout"]), 0, 0
        for _ in range(case["fields"]):
            e = int(np.exp(rng.uniform(np.log(case["edge_lo"]), np.log(case["edge_hi"]))))
            m = int(np.exp(rng.uniform(np.log(case["seeds_lo"]), np.log(case["seeds_hi"]))))
            slices = max(2, int(case["slices"] * rng.uniform(0.7, 1.3)))
            b += 12 * e ** 3 * slices * min(1.0, case["steps"] * 0.01 / 10.0) + 32 * m
            f += m * case["steps"] * UNSTEADY_STEP_FLOPS
        return {"bytes": b, "flops": f}
    datasets, requests = _service_plan(case)
    b, f = sum(12 * e ** 3 for _, e in datasets), 0
    for what, d, stride, steps in requests:
        flow, edge = datasets[d]
        seeds = max(1, edge // stride) ** 3
        taken = _steps_taken({"flow": flow, "steps": steps}, seeds)
        f += taken * (RK4_STEP_FLOPS + (60 if what == "streamlines" else 0))
        b += 4 * case["width"] * case["height"] if what == "streamlines" else 4 * seeds
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits -------------------------------------------------------------------
# Explicit Runge-Kutta schemes as (stage rows, weights), and the two Adams
# schemes by name; the published coefficients.
_RK4 = ([[], [0.5], [0.0, 0.5], [0.0, 0.0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6])
_SCHEMES = {
    "euler": ([[]], [1.0]),
    "runge_kutta_4": _RK4,
    "modified_midpoint": ([[], [0.5], [0.0, 1.0]], [0.25, 0.5, 0.25]),
    "runge_kutta_cash_karp_54": ([[], [1 / 5], [3 / 40, 9 / 40], [3 / 10, -9 / 10, 6 / 5], [-11 / 54, 5 / 2, -70 / 27, 35 / 27],
                                  [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]],
                                 [37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771]),
    "runge_kutta_dormand_prince_5": ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
                                      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
                                      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656]],
                                     [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]),
}


def _cells(p, h, n):
    """Cell (floor) and inside test of positions p (m, 3) on the grid n at offset 0."""
    c = torch.floor(p / h)
    r = p - c * h
    c = c - (r < 0).double() + (r >= h).double()
    return c, ((c >= 0) & (c <= n - 2)).all(dim=1)


def _sample(data, n, c, h, p):
    """Trilinear velocity at p; points outside the grid take the nearest boundary cell, weight 0 or 1.  c: the cell of p."""
    low, high = c < 0, c > n - 2
    w = p / h - c
    w = torch.where(low, torch.zeros_like(w), torch.where(high, torch.ones_like(w), w))
    c = torch.minimum(torch.clamp(c, min=0), n - 2).long()
    ny, nz = int(n[1]), int(n[2])
    base = (c[:, 0] * ny + c[:, 1]) * nz + c[:, 2]
    wx, wy, wz = w[:, 0:1], w[:, 1:2], w[:, 2:3]
    out = 0.0
    for dx in (0, 1):
        for dy in (0, 1):
            k = base + (dx * ny + dy) * nz
            line = torch.lerp(data[k].double(), data[k + 1].double(), wz)
            out = out + (wx if dx else 1 - wx) * (wy if dy else 1 - wy) * line
    return out


def _advect64(slices, spacing, seeds, steps, h, scheme, dt=None, record=None):
    """End positions of seeds (m, 3) in FP64: at most `steps` steps of size h,
    ending where a particle is outside or its velocity is zero.  dt: the time
    between slices (unsteady).  record(k, alive, p) is called with the
    positions after step k."""
    n = torch.tensor(slices.shape[1:4], device="cuda", dtype=torch.float64)
    spacing = torch.from_numpy(spacing.astype(np.float64)).cuda()
    data = slices.reshape(slices.shape[0], -1, 3)
    h = float(np.float32(h))

    def velocity(p, t):
        c, inside = _cells(p, spacing, n)
        if dt is None:
            return _sample(data[0], n, c, spacing, p), inside
        k = min(max(math.floor(t / dt), 0), len(data) - 2)
        w = min(max(t / dt - k, 0.0), 1.0)
        return (1 - w) * _sample(data[k], n, c, spacing, p) + w * _sample(data[k + 1], n, c, spacing, p), inside

    end = seeds.clone()
    ids = torch.arange(len(seeds), device="cuda")
    p, previous = seeds.clone(), None
    rows, weights = _SCHEMES.get(scheme, _RK4)
    ck = (0.0, 0.5, 0.5, 1.0) if scheme == "runge_kutta_4" else (0.0,) * len(rows)
    for k in range(steps):
        k1, inside = velocity(p, k * h)
        live = inside & (k1.abs() > 1e-5).any(dim=1)
        if not bool(live.all()):
            end[ids[~live]] = p[~live]
            ids, p, k1 = ids[live], p[live], k1[live]
            previous = None if previous is None else previous[live]
            if len(ids) == 0:
                break
        if scheme.startswith("adams") and previous is not None:
            q = p + h * (1.5 * k1 - 0.5 * previous)
        else:
            stage = [k1]
            for row, c in zip(rows[1:], ck[1:]):
                stage.append(velocity(p + h * sum(a * s for a, s in zip(row, stage) if a), (k + c) * h)[0])
            q = p + h * sum(b * s for b, s in zip(weights, stage) if b)
        if scheme == "adams_bashforth_moulton_2":
            q = p + 0.5 * h * (k1 + velocity(q, 0.0)[0])
        p, previous = q, k1
        if record is not None:
            record(k, ids, p)
    end[ids] = p
    return end


def _lattice(n, spacing):
    """Seed positions offset + index * spacing in FP32 (what the kernels start from), as FP64."""
    axes = [(torch.arange(m, device="cuda", dtype=torch.float32) * float(np.float32(s))).double() for m, s in zip(n, spacing)]
    return torch.stack(torch.meshgrid(*axes, indexing="ij"), dim=-1).reshape(-1, 3)


def _ftle64(flow, spacing, time, mode):
    """FTLE (or fractional anisotropy) of a flow map (nx, ny, nz, 3) in FP64."""
    columns = []
    for axis in range(3):
        m = flow.shape[axis]
        lo = torch.arange(m, device="cuda").sub(1).clamp(min=0)
        hi = torch.arange(m, device="cuda").add(1).clamp(max=m - 1)
        width = ((hi - lo).double() * float(spacing[axis])).reshape([-1 if a == axis else 1 for a in range(4)])
        columns.append((flow.index_select(axis, hi).double() - flow.index_select(axis, lo).double()) / width)
    c = {(i, j): (columns[i] * columns[j]).sum(-1) for i in range(3) for j in range(i, 3)}
    del columns
    q = (c[0, 0] + c[1, 1] + c[2, 2]) / 3.0
    d = [c[i, i] - q for i in range(3)]
    off = c[0, 1] ** 2 + c[0, 2] ** 2 + c[1, 2] ** 2
    dev = d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + 2.0 * off
    if mode != "regular":
        return torch.sqrt(1.5 * dev / (dev + 3.0 * q * q))
    p = torch.sqrt(dev / 6.0)
    det = d[0] * (d[1] * d[2] - c[1, 2] ** 2) - c[0, 1] * (c[0, 1] * d[2] - c[1, 2] * c[0, 2]) + c[0, 2] * (c[0, 1] * c[1, 2] - d[1] * c[0, 2])
    r = torch.where(p > 0, det / (2.0 * p ** 3).clamp(min=1e-300), torch.zeros_like(p)).clamp(-1.0, 1.0)
    return 0.5 * torch.log(q + 2.0 * p * torch.cos(torch.acos(r) / 3.0)) / abs(time)


def exact(case, seed):
    """The outputs in 64 bits.  None for images (bytes), for the frozen scheme
    (defined by the reference's FP32 operations), for colours other than rgb,
    and for the largest flow map."""
    kind = case["kind"]
    if kind == "ftle_stage":
        p, _, _, spacing = _flow_map_input(case, seed)
        return _ftle64(p, spacing, 5.0, case["mode"]).float()
    if kind == "pathlines":
        ends = [_advect64(xyz, spacing, seeds[:, :3].double(), case["steps"], 0.01, "runge_kutta_4", dt=dt)
                for xyz, spacing, dt, seeds in _pathline_jobs(case, seed)]
        return {"positions": ends, "steps": None}
    if kind == "service":
        return _exact_service(case, seed)
    if kind not in ("ftle", "insitu", "flow_map", "streamlines") or case.get("stages") == "frozen":
        return None
    name = case["integrator"]
    if name not in _SCHEMES and not name.startswith("adams"):
        return None
    n, step = _shape(case), _step(case)
    xyz, _, _, spacing = _field(case["flow"], n, seed)
    if kind == "streamlines":
        return _exact_streamlines(case, xyz, spacing)
    scale = np.float32(case.get("scale", 1.0))
    m = [int(np.float32(v) * scale) for v in n]
    if m[0] * m[1] * m[2] * case["steps"] > 1.6e9:
        return None
    fine = (spacing / scale).astype(np.float32)
    flow = _advect64(xyz[None], spacing, _lattice(m, fine), case["steps"], step, name).reshape(*m, 3)
    if kind == "flow_map":
        return {"flow_map": flow, "steps": None}
    out = _ftle64(flow, fine, case["steps"] * step, case["mode"])
    return out if kind == "ftle" else {"ftle": out, "steps": None}


def _exact_streamlines(case, xyz, spacing):
    n = np.array(_shape(case))
    size = _extent(n, spacing)
    stride = (spacing * np.float32(case["stride"])).astype(np.float32)
    seeds = _lattice([int(size[i] / stride[i]) for i in range(3)], stride)
    m = len(seeds)
    path = torch.zeros((m, case["steps"] + 2, 4), device="cuda", dtype=torch.float64)
    length = torch.ones(m, device="cuda", dtype=torch.long)
    path[:, 0, :3] = seeds

    def record(k, ids, p):
        path[ids, k + 1, :3] = p
        length[ids] = k + 2

    _advect64(xyz[None], spacing, seeds, case["steps"], _step(case), case["integrator"], record=record)
    path[torch.arange(m, device="cuda"), length] = torch.tensor([-2.0, -2.0, -2.0, 0.0], device="cuda", dtype=torch.float64)
    kept = torch.arange(case["steps"] + 2, device="cuda")[None, :] <= length[:, None]
    vertices = torch.zeros((m * (case["steps"] + 2), 4), device="cuda", dtype=torch.float64)
    total = int(kept.sum())
    vertices[:total] = path[kept]
    if case["color"] != "rgb":
        return {"vertices": vertices, "colors": None, "indices": None}
    # |tangent| as (x, z, y), alpha 1; a curve's last vertex copies its colour, the termination vertices have none
    term = (vertices == torch.tensor([-2.0, -2.0, -2.0, 0.0], device="cuda", dtype=torch.float64)).all(dim=1)
    t = vertices[1:, :3] - vertices[:-1, :3]
    line = ~(term[1:] | term[:-1]) & (torch.arange(1, len(vertices), device="cuda") < total)
    t = (t / torch.linalg.vector_norm(t, dim=1, keepdim=True).clamp(min=1e-300)).abs()
    colors = torch.zeros_like(vertices)
    rgba = torch.cat([t[:, [0, 2, 1]], torch.ones_like(t[:, :1])], dim=1)
    colors[:-1][line] = rgba[line]
    at = torch.nonzero(line).flatten()
    last = at[:-1][at[1:] != at[:-1] + 1]
    colors[last + 1] = rgba[last]
    return {"vertices": vertices, "colors": colors, "indices": None}


def _exact_service(case, seed):
    datasets, requests = _service_plan(case)
    fields = [_field(flow, (edge,) * 3, seed * 16 + k) for k, (flow, edge) in enumerate(datasets)]
    out = []
    for what, d, stride, steps in requests:
        if what != "ftle":
            out.append(None)
            continue
        xyz, _, _, spacing = fields[d]
        scale = np.float32(1.0) / np.float32(stride)
        m = [int(np.float32(v) * scale) for v in xyz.shape[:3]]
        fine = (spacing / scale).astype(np.float32)
        step = np.float32(_step({"flow": datasets[d][0]}))
        flow = _advect64(xyz[None], spacing, _lattice(m, fine), steps, step, "runge_kutta_4").reshape(*m, 3)
        out.append(_ftle64(flow, fine, float(step * np.float32(steps + 1)), "regular"))
    return out
