"""The work this framework does for a program, as timed cases.

A case is a dict of plain values.  `prepare` builds what a program holds
before the call (a context with its inputs, device images, targets) from a
seed; `run` is one pass through the public entry points and returns its
outputs; `work` counts the bytes and operations the pass cannot do without;
`exact` gives the same outputs in 64 bits with plain torch (`_Exact` and the
functions after it).

Kinds of case:
  frame        one frame of the render loop: set the frame uniforms, march,
               composite over the backdrop.  `fused` 0 dispatches the
               subsystem's passes (march into the cloud RT, composite);
               1 calls the march with the composite in the same kernel
  flight       two consecutive frames of a moving camera after a cut, each
               with its sky-view and aerial-perspective bake, at half
               resolution with the temporal resolve
  first_frame  start-up: a new context, its noise and LUT bakes, one frame
  batch        two time steps of a batch of views of uneven size and scene
  grid         forward march of a voxel density grid
  adjoint      one gradient step of the grid fit: loss, d / d values,
               d / d density_scale
  range_grad   d loss / d (base, top) of the grid's layer
  layer_params d loss / d the six parameters of one procedural layer
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch
import torch.autograd.forward_ad as fwAD

from pedalsky_b200 import batch as B
from pedalsky_b200 import capi, scenes
from pedalsky_b200.capi import call
from pedalsky_b200.grid import GridProblem
from pedalsky_b200.layer_grad import layer_param_gradient
from pedalsky_b200.subsystem import PrepareContext, RenderContext, WeatherInputs, subsystem_for_scene

DEV = torch.device("cuda", 0)
STORAGE = {"u8": capi.STORAGE_U8, "f32": capi.STORAGE_F32, "f16": capi.STORAGE_F16, "bf16": capi.STORAGE_BF16}
FILTER = {"exact": capi.FILTER_EXACT, "hybrid": capi.FILTER_HYBRID}
SCHEDULE = {"plain": capi.SCHED_PLAIN, "fast": capi.SCHED_FAST}
PHASE = {"mie": capi.PHASE_APPROX_MIE, "hg": capi.PHASE_DUAL_LOBE_HG}

# type:base:top:coverage of each layer
ONE_LAYER = "0:1500:2300:0.5"
THREE_LAYERS = "0:1500:2300:0.5;4:4000:5000:0.7;5:8000:9000:0.3"
STORM = "7:600:12000:0.8"
GRID_LAYER = "0:1500:3500:0.5"


def _march(kind, name, width, height, layers, steps, light=6, octaves=4, phase="mie", storage="u8",
           filter="exact", schedule="plain", fused=0, coverage_map=0):
    return dict(name=name, kind=kind, width=width, height=height, layers=layers, steps=steps, light=light,
                octaves=octaves, phase=phase, storage=storage, filter=filter, schedule=schedule, fused=fused,
                coverage_map=coverage_map)


def _grid(kind, name, width, height, nx, ny, nz, steps, every=16):
    return dict(name=name, kind=kind, width=width, height=height, nx=nx, ny=ny, nz=nz, steps=steps, light=6,
                octaves=4, every=every)


def listed():
    fast = dict(storage="f16", filter="hybrid", schedule="fast")
    return [
        # a preview window: the smallest frame, default options, 3 octaves, dual-lobe phase
        _march("frame", "preview_320x180", 320, 180, ONE_LAYER, 64, octaves=3, phase="hg"),
        # the drop-in with default options on an ordinary three-layer sky
        _march("frame", "default_1080p", 1920, 1080, THREE_LAYERS, 128),
        # the same sky as a renderer that picked the production form runs it
        _march("frame", "production_1080p", 1920, 1080, THREE_LAYERS, 128, fused=1, **fast),
        # a window of odd size, exact filtering of 8-bit noise, two layers, the default 192 steps
        _march("frame", "exact_853x479", 853, 479, "2:900:1700:0.6;3:3200:3900:0.45", 192, storage="u8",
               schedule="fast"),
        # the largest frame: 4K under one deep storm layer with a 2048^2 coverage map
        _march("frame", "storm_2160p", 3840, 2160, STORM, 256, light=8, fused=1, coverage_map=2048, **fast),
        # a moving camera at the speed setting: half resolution, temporal resolve, per-frame LUT bakes
        _march("flight", "flight_1080p", 1920, 1080, THREE_LAYERS, 128, **fast),
        # program start to first picture
        _march("first_frame", "first_frame_640x360", 640, 360, ONE_LAYER, 96),
        # reflection-probe faces and side views of one world, rendered together
        dict(name="batch_12_views", kind="batch", views=12, scale=0.5, storage="f16", filter="hybrid"),
        # voxel clouds drawn without gradients
        _grid("grid", "grid_512", 512, 512, 256, 64, 256, 96),
        # one step of fitting the voxel grid to an image
        _grid("adjoint", "grid_fit_512", 512, 512, 256, 64, 256, 96),
        # the layer's altitude range in the same fit
        _grid("range_grad", "range_grad_512", 512, 512, 256, 64, 256, 96),
        # fitting a procedural layer's parameters to an image
        _march("layer_params", "layer_params_480x270", 480, 270, THREE_LAYERS, 128, storage="f32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_layers(rng, most):
    bands = sorted(rng.sample(range(3), rng.randint(1, most)))
    out = []
    for b in bands:
        lo, hi = ((700.0, 2600.0), (3000.0, 6000.0), (7000.0, 11000.0))[b]
        thick = rng.uniform(400.0, 1600.0)
        base = rng.uniform(lo, hi - thick)
        out.append("%d:%.0f:%.0f:%.2f" % (rng.randint(0, 6), base, base + thick, rng.uniform(0.3, 0.8)))
    return ";".join(out)


def draw(rng):
    kind = rng.choice(("plain", "plain", "fast", "fast", "storm", "flight", "first_frame", "batch", "grid",
                       "adjoint", "range_grad", "layer_params"))
    if kind in ("grid", "adjoint", "range_grad"):
        side = _log_int(rng, 64, 512)
        n = _log_int(rng, 32, 256)
        c = _grid(kind, "", side, max(1, int(side * rng.uniform(0.5, 1.0))), n, max(8, n // 4 + rng.randint(-3, 3)),
                  n + rng.randint(-9, 0), rng.randint(32, 96), every=rng.choice((8, 16, 16, 32)))
    elif kind == "batch":
        c = dict(kind="batch", views=rng.randint(2, 12), scale=round(rng.uniform(0.15, 0.5), 3), storage="f16",
                 filter="hybrid")
    else:
        w = _log_int(rng, 96, {"layer_params": 480, "first_frame": 960}.get(kind, 1920))
        h = max(1, int(w * rng.uniform(0.5, 0.62)))
        steps = rng.randint(48, 128)
        f = dict(storage="f16", filter="hybrid", schedule="fast")
        if kind == "plain":
            c = _march("frame", "", w, h, _draw_layers(rng, 3), steps, octaves=rng.randint(2, 4),
                       phase=rng.choice(("mie", "mie", "hg")), storage=rng.choice(("u8", "u8", "f32")))
        elif kind == "fast":
            f = rng.choice((f, f, dict(storage="f16", schedule="fast"), dict(storage="bf16", schedule="fast")))
            c = _march("frame", "", w, h, _draw_layers(rng, 3), rng.randint(64, 192), octaves=rng.randint(2, 4),
                       phase=rng.choice(("mie", "mie", "hg")), fused=rng.randint(0, 1), **f)
        elif kind == "storm":
            c = _march("frame", "", w, h, STORM, 2 * steps, light=rng.randint(6, 8), fused=1,
                       coverage_map=rng.choice((512, 1024, 2048)), **f)
        elif kind == "flight":
            c = _march("flight", "", w, h, _draw_layers(rng, 3), steps, **f)
        elif kind == "first_frame":
            c = _march("first_frame", "", w, h, _draw_layers(rng, 2), steps)
        else:
            c = _march("layer_params", "", w, h, _draw_layers(rng, 3), steps, storage=rng.choice(("f32", "u8")))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ scenes

def _layer_list(text):
    out = []
    for part in text.split(";"):
        t, base, top, cov = part.split(":")
        out.append((int(t), float(base), float(top), float(cov)))
    return out


def _pose(r):
    """Where a camera stands and the sun it sees."""
    return dict(cam_pos=(r.uniform(-8000.0, 8000.0), r.uniform(20.0, 300.0), r.uniform(-8000.0, 8000.0)),
                pitch_deg=r.uniform(5.0, 15.0), yaw_deg=r.uniform(0.0, 360.0), sun_alt_deg=r.uniform(20.0, 60.0),
                sun_az_deg=r.uniform(0.0, 360.0))


def _scene(width, height, layers, steps, light, octaves, opts, pose, r, coverage_map=0, fov=90.0, diurnal=0.0):
    """A scene assembled from `scenes`' parts; coverages move a little with the seed."""
    p = scenes.default_params()
    p.cloud_steps, p.light_steps, p.multi_scatter_octaves = steps, light, octaves
    p.diurnal_strength = diurnal
    descs = [(t, b, top, min(0.95, max(0.05, cov + r.uniform(-0.03, 0.03)))) for t, b, top, cov in layers]
    arr, n = scenes.synth_layers(descs)
    p.cloud_layer_count = n
    frame = scenes.frame_for(width, height, fov_deg=fov, **pose)
    if coverage_map:
        grid = scenes.mountain_wave_grid(size=coverage_map, seed=r.randrange(1 << 30))
        weather, wh, fmt = grid.reshape(-1), coverage_map, capi.WEATHER_R32F
    else:
        weather, wh, fmt = scenes.reference_weather(n), 128, capi.WEATHER_RGBA16F
    return scenes.Scene("case", width, height, p, arr, n, frame, scenes.world_default(), opts, weather, wh, wh,
                        fmt, scenes.wind_field())


def _options(case, composite=0):
    return scenes.options(phase=PHASE[case["phase"]], storage=STORAGE[case["storage"]],
                          filt=FILTER[case["filter"]], schedule=SCHEDULE[case["schedule"]], composite=composite)


def _prepare_context(s, frame=None):
    layers = [s.layers[i] for i in range(s.n_layers)]
    w = WeatherInputs(layers, s.weather, s.weather_w, s.weather_h, s.weather_format, s.wind, s.type_grid, revision=1)
    return PrepareContext(frame if frame is not None else s.frame, s.world, w)


class _State:
    """What a program holds between its calls; its context goes with it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        sub = self.__dict__.get("sub")
        if sub is not None:
            torch.cuda.synchronize()
            sub.close()


def _render_context(s, frame=None):
    f = frame if frame is not None else s.frame
    depth, bg = scenes.device_inputs(f, s.world, s.width, s.height, DEV)
    return depth, bg, torch.empty_like(bg)


def _frame_scene(case, seed):
    r = random.Random(seed)
    return _scene(case["width"], case["height"], _layer_list(case["layers"]), case["steps"], case["light"],
                  case["octaves"], _options(case, composite=case["fused"]), _pose(r), r,
                  coverage_map=case["coverage_map"], diurnal=1.0 if case["kind"] == "layer_params" else 0.0)


def _flight_scenes(case, seed):
    """The scene and its two frames: the camera turns 0.6 degrees and moves on between them."""
    r = random.Random(seed)
    pose = _pose(r)
    s = _scene(case["width"], case["height"], _layer_list(case["layers"]), case["steps"], case["light"],
               case["octaves"], _options(case), pose, r)
    x, y, z = pose["cam_pos"]
    moved = dict(pose, cam_pos=(x + 3.0, y + 0.5, z - 4.0), yaw_deg=pose["yaw_deg"] + 0.6)
    second = scenes.frame_for(s.width, s.height, fov_deg=90.0, **moved)
    C.memmove(second.prev_view_proj, s.frame.view_proj, C.sizeof(second.prev_view_proj))
    return s, [s.frame, second]


def _batch_scenes(case, seed):
    """Views of one world, half square faces and half 16:9 frames, at two time
    steps (the sun moves by half a degree): two lists of scenes."""
    r = random.Random(seed)
    opts = scenes.options(storage=STORAGE[case["storage"]], filt=FILTER[case["filter"]], schedule=capi.SCHED_FAST,
                          composite=1)
    now, then = [], []
    sizes = random.Random(case["views"])  # sizes and scenes belong to the case, poses to the seed
    for i in range(case["views"]):
        pose = _pose(r)
        if i % 2 == 0:
            w = h = sizes.choice(scenes.CUBE_SIZES)
            fov = 90.0
        else:
            w, h = sizes.choice(scenes.FRAME_SIZES)
            fov = 60.0
        w, h = max(8, int(w * case["scale"])), max(8, int(h * case["scale"]))
        layers = _layer_list(_draw_layers(sizes, 3))
        if i % 6 == 5:
            layers = [(7, 900.0, 9000.0, 0.7)]  # one view in six looks at a storm cell
        s = _scene(w, h, layers, sizes.randint(48, 160), 6, 4, opts, pose, r, fov=fov)
        now.append(s)
        later = scenes.frame_for(w, h, fov_deg=fov, **dict(pose, sun_az_deg=pose["sun_az_deg"] + 0.5))
        then.append(scenes.Scene("case", w, h, s.params, s.layers, s.n_layers, later, s.world, opts, s.weather,
                                 s.weather_w, s.weather_h, s.weather_format, s.wind))
    return now, then


def _worley(case, seed):
    """Flat-based blobs thresholded from the distance to seeded points, in [0, 0.05] 1/m, (ny, nz, nx)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator().manual_seed(seed)
    pts = torch.rand((48, 3), generator=g, dtype=torch.float64) * torch.tensor([20000.0, 2000.0, 20000.0],
                                                                             dtype=torch.float64)
    pts = pts.to(DEV)
    xs = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5) * (20000.0 / nx)
    ys = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * (2000.0 / ny)
    zs = (torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5) * (20000.0 / nz)
    best = torch.full((ny, nz, nx), 1e30, device=DEV, dtype=torch.float64)
    for p in pts:
        d = ((xs - p[0]) ** 2)[None, None, :] + ((2.5 * (ys - p[1])) ** 2)[:, None, None] + ((zs - p[2]) ** 2)[None, :, None]
        best = torch.minimum(best, d)
    return (0.05 * (1.0 - best.sqrt() / 1100.0).clamp(0.0, 1.0)).float()


def _grid_scene(case, seed):
    r = random.Random(seed)
    pose = dict(cam_pos=(r.uniform(-2000.0, 2000.0), 100.0, r.uniform(-2000.0, 2000.0)), pitch_deg=55.0,
                yaw_deg=r.uniform(0.0, 360.0), sun_alt_deg=r.uniform(25.0, 55.0), sun_az_deg=r.uniform(0.0, 360.0))
    s = _scene(case["width"], case["height"], _layer_list(GRID_LAYER), case["steps"], case["light"],
               case["octaves"], scenes.options(), pose, r, fov=60.0)
    s.background = scenes.sky_background(s.frame, s.width, s.height)
    s.extra["grid_spec"] = dict(min_x_m=-10000.0, min_z_m=-10000.0, size_x_m=20000.0, size_z_m=20000.0,
                                density_scale=1.0, exit_transmittance=0.01, checkpoint_every=case["every"])
    return s


def _grid_problem(case, seed):
    s = _grid_scene(case, seed)
    values = _worley(case, seed)
    return s, values, GridProblem(s, values.cpu().numpy(), device=DEV)


def _noisy(t, seed, rel):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (t * (1.0 + rel * torch.randn(t.shape, generator=g, device=DEV))).clamp_min(0.0)


# ----------------------------------------------------------- prepare / run

def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        s = _frame_scene(case, seed)
        depth, bg, color = _render_context(s)
        return _State(kind=kind, fused=case["fused"], s=s, sub=subsystem_for_scene(s), depth=depth, bg=bg,
                      color=color, ctx=_prepare_context(s))
    if kind == "flight":
        s, frames = _flight_scenes(case, seed)
        sub = subsystem_for_scene(s)
        opts = capi.MarchOptions.from_buffer_copy(sub.options)
        opts.half_res, opts.taa = 1, 1
        sub.set_options(opts)
        views = [(_prepare_context(s, f), _render_context(s, f)) for f in frames]
        return _State(kind=kind, s=s, sub=sub, views=views)
    if kind == "first_frame":
        s = _frame_scene(case, seed)
        depth, bg, color = _render_context(s)
        return _State(kind=kind, s=s, depth=depth, bg=bg, color=color)
    if kind == "batch":
        now, then = _batch_scenes(case, seed)
        sub = subsystem_for_scene(now[0])
        B.set_tuning(sub.handle, use_graph=1, form=capi.BATCH_PER_VIEW)
        return _State(kind=kind, sub=sub, steps=[B.Batch(now, DEV), B.Batch(then, DEV)])
    if kind == "layer_params":
        s = _frame_scene(case, seed)
        depth, bg, _ = _render_context(s)
        view = capi.View(s.width, s.height, depth.data_ptr(), None, None, None)
        target = _noisy(bg, seed, 0.05)
        return _State(kind=kind, s=s, sub=subsystem_for_scene(s), depth=depth, bg=bg, target=target, view=view,
                      layer=seed % s.n_layers, grad=torch.zeros(6, dtype=torch.float64, device=DEV),
                      loss=torch.zeros(1, dtype=torch.float64, device=DEV))
    s, values, p = _grid_problem(case, seed)
    st = _State(kind=kind, s=s, sub=subsystem_for_scene(s), p=p)
    if kind in ("adjoint", "range_grad"):
        p.set_target(_target(p.bg, seed))
        st.range = torch.zeros(2, dtype=torch.float64, device=DEV)
    return st


def _target(bg, seed):
    """A picture to fit: the backdrop under half-cover with 5 % pixel noise."""
    t = _noisy(bg, seed, 0.05)
    t[..., :3] *= 0.6
    return t


def _passes(sub, ctx, color, bg, depth):
    """One frame through the subsystem: the backdrop stands for the passes before the clouds."""
    color.copy_(bg)
    sub.prepare(ctx)
    rc = RenderContext(color=color, depth=depth)
    for p in sub.register_passes():
        sub.dispatch_pass(p.id, rc)


def run(st):
    if st.kind == "frame":
        if st.fused:
            st.color.copy_(st.bg)
            st.sub.prepare(st.ctx)
            v = capi.View(st.s.width, st.s.height, st.depth.data_ptr(), None, None, st.color.data_ptr())
            call("psc_render", st.sub.handle, C.byref(v), 1, C.c_void_p(torch.cuda.current_stream().cuda_stream))
            return {"color": st.color}
        _passes(st.sub, st.ctx, st.color, st.bg, st.depth)
        return {"color": st.color, "luminance": st.sub.cloud_rt[0], "transmittance": st.sub.cloud_rt[1]}
    if st.kind == "flight":
        st.sub.invalidate_taa_history()
        for ctx, (depth, bg, color) in st.views:
            st.sub.prepare(ctx)
            st.sub.set_atmosphere_luts()
            _passes(st.sub, ctx, color, bg, depth)
        return {"first": st.views[0][1][2], "second": st.views[1][1][2]}
    if st.kind == "first_frame":
        sub = subsystem_for_scene(st.s)
        _passes(sub, _prepare_context(st.s), st.color, st.bg, st.depth)
        out = {"color": st.color, "luminance": sub.cloud_rt[0], "transmittance": sub.cloud_rt[1]}
        sub.close()
        return out
    if st.kind == "batch":
        stream = torch.cuda.current_stream()
        for b in st.steps:
            b.reset_hdr()
            b.render(st.sub.handle, stream)
        return {"first": st.steps[0].hdr, "second": st.steps[1].hdr}
    if st.kind == "layer_params":
        st.grad.zero_()
        st.loss.zero_()
        layer_param_gradient(st.sub.handle, st.view, st.layer, st.bg, st.target, st.grad, st.loss)
        # the optimiser's step takes them in the parameters' type
        return {"grad": st.grad.float(), "loss": st.loss.float()}
    stream = torch.cuda.current_stream()
    if st.kind == "grid":
        lum, tr = st.p.render(st.sub.handle, stream=stream)
        return {"luminance": lum, "transmittance": tr}
    if st.kind == "adjoint":
        st.p.zero_grad()
        st.p.adjoint(st.sub.handle, stream=stream)
        acc = st.p.acc.float()  # loss and d / d density_scale in the parameters' type
        return {"luminance": st.p.L, "transmittance": st.p.T, "grad": st.p.grad, "acc": acc}
    st.range.zero_()
    st.p.layer_gradient(st.sub.handle, st.range, stream=stream)
    return {"range": st.range.float()}


# -------------------------------------------------------------------- work

NOISE_BYTES = 128 ** 3 * 4 + 32 ** 3 * 4 + 128 * 128 * 2 + 64 * 64
LUT_BYTES = 8 * (256 * 64 + 32 * 32 + 192 * 108 + 32 * 32 * 64)


def _march_flops(px, n_layers, steps, light):
    """Two thirds of the pixels are sky; every step there needs a position,
    height and density tap (100), a third of them the light taps (50 each) and
    the shading (250)."""
    return px * 0.67 * n_layers * steps * (100.0 + (50.0 * light + 250.0) / 3.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        now, _ = _batch_scenes(case, 0)
        b, f = 2.0 * (NOISE_BYTES + len(now) * LUT_BYTES), 0.0
        for s in now:
            px = s.width * s.height
            b += 2.0 * px * (4 + 16 + 16)
            f += 2.0 * _march_flops(px, s.n_layers, s.params.cloud_steps, s.params.light_steps)
        return {"bytes": b, "flops": f}
    px = case["width"] * case["height"]
    if kind in ("grid", "adjoint", "range_grad"):
        cells = case["nx"] * case["ny"] * case["nz"]
        samples = px * case["steps"]
        # every sample's grid tap (40), the seventh that is not empty its light taps and shading
        taps = samples * 60.0 + samples * 0.15 * (case["light"] * 60.0 + 300.0)
        if kind == "grid":
            return {"bytes": cells * 4.0 + px * 32.0, "flops": taps}
        # the gradient needs the light at every sample (a cell that is empty has one too)
        full = samples * (60.0 + case["light"] * 60.0 + 300.0)
        out = cells * 8.0 + px * 64.0 if kind == "adjoint" else px * 32.0 + cells * 4.0
        return {"bytes": out, "flops": full if kind == "adjoint" else 2.0 * taps}
    n_layers = len(_layer_list(case["layers"]))
    f = _march_flops(px, n_layers, case["steps"], case["light"])
    b = NOISE_BYTES + LUT_BYTES + case["coverage_map"] ** 2 * 4.0
    if kind == "flight":
        return {"bytes": 2.0 * (b + px * (4 + 16 + 16)), "flops": 2.0 * f / 4.0}
    if kind == "layer_params":
        return {"bytes": b + px * (4.0 + 16 + 16), "flops": 4.0 * f}
    if kind == "first_frame":  # the noise is written once: 8 cell-noise octaves of 27 cells each per texel
        return {"bytes": b + px * (4 + 16 + 16 + 32.0), "flops": f + 128 ** 3 * 8 * 27 * 10.0}
    return {"bytes": b + px * (4 + 16 + 16 + (0.0 if case["fused"] else 32.0)), "flops": f}


# ------------------------------------------------------------------- exact
# The march and the passes around it in 64 bits.  Every function works on
# flat arrays of samples; a layer's parameters may carry a forward-mode
# tangent, which the gradients read.

F64 = torch.float64
PI = math.pi


def _clamp01(x):
    return x.clamp(0.0, 1.0)


def _smooth(e0, e1, x):
    t = _clamp01((x - e0) / (e1 - e0))
    return t * t * (3.0 - 2.0 * t)


def _half(x):
    return x.half().to(F64)


def _sphere(oc, d, r):
    """Both distances to a sphere about the planet's centre; NaN where missed."""
    b = (oc * d).sum(-1)
    c = (oc * oc).sum(-1) - r * r
    q = b * b - c
    sq = torch.where(q >= 0, q.clamp_min(1e-30).sqrt(), torch.full_like(q, math.nan))
    return -b - sq, -b + sq


def _sample2(lut, u, v, wrap=False):
    """Bilinear (H, W, C) at texel centres u W - 1/2."""
    h, w = lut.shape[:2]
    x, y = u * w - 0.5, v * h - 0.5
    fx, fy = x.detach().floor(), y.detach().floor()
    wx, wy = (x - fx)[..., None], (y - fy)[..., None]
    ix, iy = fx.long(), fy.long()

    def at(i, j):
        if wrap:
            return lut[j % h, i % w]
        return lut[j.clamp(0, h - 1), i.clamp(0, w - 1)]

    a = at(ix, iy) * (1 - wx) + at(ix + 1, iy) * wx
    b = at(ix, iy + 1) * (1 - wx) + at(ix + 1, iy + 1) * wx
    return a * (1 - wy) + b * wy


def _sample3(vol, x, y, z, wrap):
    """Trilinear (D, H, W, C) at texel coordinates (already less 1/2)."""
    n = vol.shape[:3]
    f = [c.detach().floor() for c in (x, y, z)]
    wx, wy, wz = [(c - g)[..., None] for c, g in zip((x, y, z), f)]
    ix, iy, iz = [g.long() for g in f]

    def at(i, j, k):
        if wrap:
            return vol[k % n[0], j % n[1], i % n[2]]
        return vol[k.clamp(0, n[0] - 1), j.clamp(0, n[1] - 1), i.clamp(0, n[2] - 1)]

    out = 0.0
    for k, sz in ((iz, 1 - wz), (iz + 1, wz)):
        for j, sy in ((iy, 1 - wy), (iy + 1, wy)):
            out = out + (at(ix, j, k) * (1 - wx) + at(ix + 1, j, k) * wx) * (sy * sz)
    return out


def _density_h(w, h):
    """Rayleigh, Mie and ozone densities at height h."""
    oz = (1.0 - (h - w.ozone_center_m).abs() / max(w.ozone_thickness_m * 0.5, 1.0)).clamp_min(0.0)
    return torch.exp(-h / w.rayleigh_scale_height_m), torch.exp(-h / w.mie_scale_height_m), oz


def _vec(values):
    return torch.tensor([float(v) for v in values][:3], dtype=F64, device=DEV)


def _extinction(w, h):
    r, m, o = _density_h(w, h)
    return (_vec(w.rayleigh_scattering) * r[..., None] + (_vec(w.mie_scattering) + _vec(w.mie_absorption)) * m[..., None]
            + _vec(w.ozone_absorption) * o[..., None])


def _boundary(w, p, d):
    _, tt = _sphere(p, d, w.atmosphere_top_m)
    g, _ = _sphere(p, d, w.planet_radius_m)
    tt = torch.where(torch.isnan(tt), torch.zeros_like(tt), tt)
    return torch.where(g > 0, torch.minimum(tt, g), tt).clamp_min(0.0)


def _trans_uv(w, r, mu):
    R, top = w.planet_radius_m, w.atmosphere_top_m
    H = math.sqrt(top * top - R * R)
    rho = (r * r - R * R).clamp_min(0.0).sqrt()
    d = (-r * mu + (r * r * (mu * mu - 1.0) + top * top).clamp_min(0.0).sqrt()).clamp_min(0.0)
    d_min, d_max = top - r, rho + H
    return _clamp01((d - d_min) / (d_max - d_min).clamp_min(1.0)), rho / H


def _sun_visible(w, lut, p, sun):
    """Transmittance LUT toward the sun at p (planet-centred), 0 where the ground is in the way."""
    g, _ = _sphere(p, sun.expand_as(p), w.planet_radius_m)
    r = p.norm(dim=-1)
    mu = (p * sun).sum(-1) / r
    u, v = _trans_uv(w, r, mu)
    t = _sample2(lut, u, v)
    return torch.where((g > 0)[..., None], torch.zeros_like(t), t)


def _inscatter(w, luts, p, d, sun, dt, steps, illum, stop):
    """Single and multiple scattering along p + t d, `steps` mid-point steps of dt."""
    n = p.shape[0]
    lum, tr = torch.zeros(n, 3, dtype=F64, device=DEV), torch.ones(n, 3, dtype=F64, device=DEV)
    c = (d * sun).sum(-1)
    pr = (3.0 / (16.0 * PI)) * (1.0 + c * c)
    g = w.mie_g
    den = (1.0 + g * g - 2.0 * g * c).clamp_min(1e-4)
    pm = (1.0 - g * g) / (4.0 * PI * den ** 1.5)
    on = torch.ones(n, dtype=torch.bool, device=DEV)
    for s in range(steps):
        q = p + d * ((s + 0.5) * dt)[:, None]
        r = q.norm(dim=-1)
        h = r - w.planet_radius_m
        if stop:
            on = on & ~(h < 0)
        st = _extinction(w, h)
        trs = torch.exp(-st * dt[:, None])
        dr, dm, _ = _density_h(w, h)
        sr, sm = _vec(w.rayleigh_scattering) * dr[:, None], _vec(w.mie_scattering) * dm[:, None]
        vis = _sun_visible(w, luts["transmittance"], q, sun)
        hn = _clamp01(h / max(w.atmosphere_top_m - w.planet_radius_m, 1.0))
        sc = ((q * sun).sum(-1) / r.clamp_min(1.0)).clamp(-1.0, 1.0)
        ms = _sample2(luts["multiscatter"], sc * 0.5 + 0.5, hn)
        ins = ((sr * pr[:, None] + sm * pm[:, None]) * vis + (sr + sm) * ms) * illum
        add = tr * (ins - ins * trs) / st.clamp_min(1e-7)
        lum = torch.where(on[:, None], lum + add, lum)
        tr = torch.where(on[:, None], tr * trs, tr)
    return lum, tr


def _static_luts(w):
    """Transmittance and multiple-scattering LUTs, (H, W, 3), rounded to half as stored."""
    R, top = w.planet_radius_m, w.atmosphere_top_m
    H = math.sqrt(top * top - R * R)
    v, u = torch.meshgrid((torch.arange(64, device=DEV, dtype=F64) + 0.5) / 64,
                          (torch.arange(256, device=DEV, dtype=F64) + 0.5) / 256, indexing="ij")
    u, v = u.reshape(-1), v.reshape(-1)
    rho = v * H
    r = (rho * rho + R * R).sqrt()
    d_min, d_max = top - r, rho + H
    d = d_min + u * (d_max - d_min)
    mu = ((H * H - rho * rho - d * d) / (2.0 * r * d).clamp_min(1e-6)).clamp(-1.0, 1.0)
    zero = torch.zeros_like(r)
    p, q = torch.stack([zero, r, zero], -1), torch.stack([(1.0 - mu * mu).clamp_min(0.0).sqrt(), mu, zero], -1)
    dt = _boundary(w, p, q) / 40.0
    prev, od = _extinction(w, r - R), 0.0
    for i in range(1, 41):
        cur = _extinction(w, (p + q * (i * dt)[:, None]).norm(dim=-1) - R)
        od = od + (prev + cur) * (0.5 * dt)[:, None]
        prev = cur
    luts = {"transmittance": _half(torch.exp(-od)).reshape(64, 256, 3)}
    v, u = torch.meshgrid((torch.arange(32, device=DEV, dtype=F64) + 0.5) / 32,
                          (torch.arange(32, device=DEV, dtype=F64) + 0.5) / 32, indexing="ij")
    u, v = u.reshape(-1), v.reshape(-1)
    sc = u * 2.0 - 1.0
    sun = torch.stack([(1.0 - sc * sc).clamp_min(0.0).sqrt(), sc, torch.zeros_like(sc)], -1)
    r = R + v * (top - R)
    p = torch.stack([torch.zeros_like(r), r, torch.zeros_like(r)], -1)
    l2, fm = torch.zeros(1024, 3, dtype=F64, device=DEV), torch.zeros(1024, 3, dtype=F64, device=DEV)
    for i in range(64):
        z = 1.0 - 2.0 * (i + 0.5) / 64.0
        rr, phi = math.sqrt(max(1.0 - z * z, 0.0)), 2.0 * PI * math.fmod(i * 0.6180339887498949, 1.0)
        d = torch.tensor([rr * math.cos(phi), rr * math.sin(phi), z], dtype=F64, device=DEV).expand(1024, 3)
        dt = _boundary(w, p, d) / 20.0
        tr = torch.ones_like(l2)
        for s in range(20):
            q = p + d * ((s + 0.5) * dt)[:, None]
            h = q.norm(dim=-1) - R
            st = _extinction(w, h)
            dr, dm, _ = _density_h(w, h)
            both = _vec(w.rayleigh_scattering) * dr[:, None] + _vec(w.mie_scattering) * dm[:, None]
            trs = torch.exp(-st * dt[:, None])
            vis = _sun_visible(w, luts["transmittance"], q, sun)
            part = (1.0 - trs) / st.clamp_min(1e-7) * both * tr
            l2, fm, tr = l2 + part * vis, fm + part, tr * trs
    l2, fm = l2 / 64.0, fm / 64.0  # (4 pi / 64) / (4 pi)
    luts["multiscatter"] = _half(l2 / (1.0 - fm.clamp(0.0, 0.95))).reshape(32, 32, 3)
    return luts


def _frame_luts(w, f, statics):
    """The LUTs a frame reads: `statics` and the frame's sky view and aerial perspective."""
    luts = dict(statics)
    R = w.planet_radius_m
    cam, sun = _vec(f.camera_position_world), _vec(f.sun_direction)
    p = cam + torch.tensor([0.0, R, 0.0], dtype=F64, device=DEV)
    r = float(p.norm())
    pv = p * ((R + 1.0) / r) if r < R + 1.0 else p
    r = max(r, R + 1.0)
    v, u = torch.meshgrid((torch.arange(108, device=DEV, dtype=F64) + 0.5) / 108,
                          (torch.arange(192, device=DEV, dtype=F64) + 0.5) / 192, indexing="ij")
    u, v = u.reshape(-1), v.reshape(-1)
    zha = PI - math.asin(min(max(R / r, 0.0), 1.0))
    lo, hi = v * 2.0, (v - 0.5) * 2.0
    vza = torch.where(v < 0.5, lo * lo * zha, zha + hi * hi * (PI - zha))
    az = torch.atan2(sun[0], sun[2]) + u * 2.0 * PI
    d = torch.stack([vza.sin() * az.sin(), vza.cos(), vza.sin() * az.cos()], -1)
    pp = pv.expand_as(d)
    lum, tr = _inscatter(w, luts, pp, d, sun, _boundary(w, pp, d) / 32.0, 32, 1.0, False)
    g, _ = _sphere(pp, d, R)
    hit = g > 0
    pg = pp + d * torch.where(hit, g, torch.zeros_like(g))[:, None]
    ndl = ((pg / pg.norm(dim=-1, keepdim=True)) * sun).sum(-1).clamp_min(0.0)
    # on the ground itself the sun is hidden only below the horizon
    ground = tr * (_vec(w.ground_albedo) / PI) * ndl[:, None] * _ground_light(w, luts, pg, sun)
    luts["skyview"] = _half(torch.where(hit[:, None], lum + ground, lum)).reshape(108, 192, 3)
    z, y, x = torch.meshgrid((torch.arange(64, device=DEV, dtype=F64) + 0.5) / 64,
                             (torch.arange(32, device=DEV, dtype=F64) + 0.5) / 32,
                             (torch.arange(32, device=DEV, dtype=F64) + 0.5) / 32, indexing="ij")
    z, y, x = z.reshape(-1), y.reshape(-1), x.reshape(-1)
    d = _view_dirs(f, x * 2.0 - 1.0, -(y * 2.0 - 1.0))
    t = 50.0 * (100000.0 / 50.0) ** z
    lum, tr = _inscatter(w, luts, p.expand_as(d), d, sun, t / 16.0, 16, _vec(f.sun_illuminance), True)
    tl = tr @ torch.tensor([0.2126, 0.7152, 0.0722], dtype=F64, device=DEV)
    luts["aerial"] = _half(torch.cat([lum, tl[:, None]], -1)).reshape(64, 32, 32, 4)
    return luts


def _ground_light(w, luts, pg, sun):
    mu = (pg * sun).sum(-1) / pg.norm(dim=-1)
    u, v = _trans_uv(w, pg.norm(dim=-1), mu)
    t = _sample2(luts["transmittance"], u, v)
    return torch.where((mu > 0)[:, None], t, torch.zeros_like(t))


def _mat(m):
    return torch.tensor(np.array(m, np.float64), dtype=F64, device=DEV)  # [col][row]


def _unproject(f, nx, ny, dn):
    inv = _mat(f.inv_view_proj)
    h = inv[0] * nx[:, None] + inv[1] * ny[:, None] + inv[2] * dn[:, None] + inv[3]
    return h[:, :3] / h[:, 3:4] - _vec(f.camera_position_world)


def _view_dirs(f, nx, ny):
    d = _unproject(f, nx, ny, torch.ones_like(nx))
    return d / d.norm(dim=-1, keepdim=True)


class _Exact:
    """A scene's inputs in 64 bits."""

    def __init__(self, s, sub):
        self.s, self.w, self.p = s, s.world, s.params
        base = torch.from_numpy(sub.noise(capi.NOISE_BASE)).to(DEV).reshape(128, 128, 128, 4).to(F64) / 255.0
        det = torch.from_numpy(sub.noise(capi.NOISE_DETAIL)).to(DEV).reshape(32, 32, 32, 4).to(F64) / 255.0
        self.base = torch.stack([base[..., 0], 0.625 * base[..., 1] + 0.25 * base[..., 2] + 0.125 * base[..., 3]], -1)
        self.detail = (0.625 * det[..., 0] + 0.25 * det[..., 1] + 0.125 * det[..., 2])[..., None].contiguous()
        self.curl = torch.from_numpy(sub.noise(capi.NOISE_CURL)).to(DEV).reshape(128, 128, 2).to(F64) / 255.0
        self.blue = torch.from_numpy(sub.noise(capi.NOISE_BLUE)).to(DEV).reshape(64, 64).to(F64) / 255.0
        if s.weather_format == capi.WEATHER_R32F:
            wm = s.weather.reshape(s.weather_h, s.weather_w)
        else:
            wm = s.weather.view(np.float16).reshape(s.weather_h, s.weather_w, 4)[..., 0]
        self.weather = torch.from_numpy(np.ascontiguousarray(wm, np.float64)).to(DEV)[..., None]
        wind = s.wind.view(np.float16).reshape(32, 16, 32, 4).astype(np.float64)  # z, y, x
        col = wind[15:17, :, 15:17, :2].mean(axis=(0, 2))
        self.wind = torch.from_numpy(col).to(DEV)  # (16, 2), the centre column
        self.statics = _static_luts(s.world)

    def layers(self, frame):
        """The scene's layers as dicts of scalars."""
        sy = float(frame.sun_direction[1])
        t = min(max((sy + 0.1) / 0.5, 0.0), 1.0)
        bell = t * t * (3.0 - 2.0 * t)
        out = []
        for i in range(self.s.n_layers):
            L = self.s.layers[i]
            di = bell * self.p.diurnal_strength if L.cloud_type in (0, 2, 3, 7) else 0.0
            c = lambda v: torch.tensor(float(v), dtype=F64, device=DEV)  # noqa: E731
            out.append(dict(type=L.cloud_type, anvil=float(L.anvil_bias), droplet=float(L.droplet_diameter_um), di=di,
                            base=c(L.base_m), top=c(L.top_m), coverage=c(L.coverage), shape=c(L.shape_bias),
                            detail=c(L.detail_bias), scale=c(L.density_scale)))
        return out

    def sigma_t(self, L):
        t = min(max(1.0 - L["droplet"] / 20.0, 0.0), 1.0)
        s = 0.25 * t * t
        mod = torch.tensor([1.0 - 0.5 * s, 1.0, 1.0 + s], dtype=F64, device=DEV)
        return (_vec(self.p.sigma_s) + _vec(self.p.sigma_a)) * mod

    def skew(self, L):
        """Unit wind direction at the layer's middle times the skew length (drift is 0 at time 0)."""
        mid = 0.5 * (L["base"] + L["top"])
        y = (mid / 12000.0).clamp(0.0, 0.9999) * 16.0 - 0.5
        fl = y.detach().floor()
        i = int(fl)
        wv = self.wind[i % 16] * (1.0 - (y - fl)) + self.wind[(i + 1) % 16] * (y - fl)
        sp = (wv * wv).sum().sqrt()
        if float(sp.detach()) < 1e-3:
            return torch.zeros(2, dtype=F64, device=DEV)
        return wv / sp * (L["top"] - L["base"]).clamp_min(1.0) * self.p.wind_skew_strength

    def profile(self, L, h):
        t = L["type"]
        if t == 7:
            mid, mt = _smooth(0.95, 0.5, h), _smooth(0.65, 0.8, h)
            anvil = _smooth(0.7, 0.9, h) * 1.5 * min(max(L["anvil"], 0.0), 2.0)
            return _smooth(0.0, 0.05, h) * (mid * (1.0 - mt) + anvil * mt)
        a, e0, e1, falling = ((0.07, 1.0, 0.2, 0), (0.10, 0.6, 1.0, 1), (0.15, 1.0, 0.4, 0), (0.20, 1.0, 0.3, 0),
                              (0.30, 0.7, 1.0, 1), (0.40, 0.6, 1.0, 1), (0.50, 0.8, 1.0, 1))[t]
        g = _smooth(e0, e1, h)
        return _smooth(0.0, a, h) * (1.0 - g if falling else g)

    def density(self, L, skew, p, h, eff, light):
        sx, sz = skew[0] * h, skew[1] * h
        ax, ay, az = p[:, 0] - sx, p[:, 1], p[:, 2] - sz
        k = 128.0 / max(self.p.base_scale_m, 1.0)
        b = _sample3(self.base, ax * k - 0.5, ay * k - 0.5, az * k - 0.5, True)
        low = _clamp01(b[:, 1] + L["shape"] * L["di"] * 0.5)
        cloud = (b[:, 0] + (1.0 - low)) / (2.0 - low) * self.profile(L, h)
        cloud = (cloud - (1.0 - eff)) / eff.clamp_min(1e-5) * eff
        if not light:
            ds = max(self.p.detail_scale_m, 1.0)
            c = _sample2(self.curl, ax / ds, az / ds, wrap=True) * 2.0 - 1.0
            k = 32.0 / ds
            off = self.p.curl_strength * ds
            d = _sample3(self.detail, (ax + c[:, 0] * off) * k - 0.5, ay * k - 0.5, (az + c[:, 1] * off) * k - 0.5,
                         True)[:, 0]
            m = _clamp01(h * 10.0)
            lo = (d * (1.0 - m) + (1.0 - d) * m) * _clamp01(self.p.detail_strength + L["detail"] * L["di"])
            cloud = torch.where(cloud > 0, (cloud - lo) / (1.0 - lo).clamp_min(1e-5), cloud)
        ok = (h >= 0) & (h <= 1) & (eff >= 0.01)
        return torch.where(ok, _clamp01(cloud) * L["scale"], torch.zeros_like(cloud))

    def altitude(self, p):
        q = torch.stack([p[:, 0], p[:, 1] + self.w.planet_radius_m, p[:, 2]], -1)
        r = q.norm(dim=-1)
        return r - self.w.planet_radius_m, q / r[:, None]

    def phase(self, L, cos_t, g_scale, h):
        o = self.s.options
        hg = lambda g: (1.0 - g * g) / (4.0 * PI * (1.0 + g * g - 2.0 * g * cos_t).clamp_min(1e-4) ** 1.5)  # noqa: E731
        if o.phase_mode == capi.PHASE_DUAL_LOBE_HG:
            return hg(o.hg_g_forward * g_scale) * (1.0 - o.hg_blend) + hg(o.hg_g_backward * g_scale) * o.hg_blend
        d = torch.full_like(cos_t, L["droplet"])
        if L["type"] == 7:
            mt = _smooth(0.60, 0.85, h)
            d = d * (1.0 - mt) + 50.0 * mt
        d = (d * self.p.droplet_diameter_bias).clamp(5.0, 50.0)
        g1 = torch.exp(-0.0990567 / (d - 1.67154)) * g_scale
        g2 = (torch.exp(-2.20679 / (d + 3.91029)) - 0.428934) * g_scale
        al = torch.exp(3.62489 - 8.29288 / (d + 5.52825))
        wd = torch.exp(-0.599085 / (d - 0.641583) - 0.665888)
        q = g2 * g2
        den = (1.0 + q - 2.0 * g2 * cos_t).clamp_min(1e-4) ** 1.5
        dr = (1.0 - q) * (1.0 + al * cos_t * cos_t) / (4.0 * (1.0 + al * (1.0 + 2.0 * q) / 3.0) * PI * den).clamp_min(1e-6)
        ph = (1.0 - wd) * hg(g1) + wd * dr
        ice = _smooth(35.0, 50.0, d)
        width = (0.5 * PI / 180.0) / max(g_scale, 0.1)

        def halo(peak):
            return torch.exp(-0.5 * ((cos_t - peak) / max(width * math.sqrt(1.0 - peak * peak), 1e-4)) ** 2)

        return ph + ice * (0.08 * halo(0.92718) + 0.03 * halo(0.69466))

    def lighting(self, luts, frame, alt, up):
        """Sun transmittance and sky ambient (times the illuminance) at points of altitude `alt`."""
        R = self.w.planet_radius_m
        sun, ill = _vec(frame.sun_direction), _vec(frame.sun_illuminance)
        r = (R + alt).clamp_min(R + 1.0)
        mu = (up * sun).sum(-1).clamp(-1.0, 1.0)
        u, v = _trans_uv(self.w, r, mu)
        ts = _sample2(luts["transmittance"], u, v)
        dark = mu <= -(1.0 - (R / r) ** 2).clamp_min(0.0).sqrt()
        ts = torch.where(dark[:, None], torch.zeros_like(ts), ts)
        flat = (up[:, 0] ** 2 + up[:, 2] ** 2).clamp_min(1e-30).sqrt()
        vza = torch.atan2(flat, up[:, 1])
        zha = PI - torch.asin((R / (R + alt)).clamp(max=1.0 - 1e-15))
        vv = torch.where(vza < zha, _clamp01(vza / zha).clamp_min(1e-30).sqrt() * 0.5,
                         0.5 + _clamp01((vza - zha) / (PI - zha)).clamp_min(1e-30).sqrt() * 0.5)
        du = (torch.atan2(up[:, 0], up[:, 2]) - math.atan2(float(sun[0]), float(sun[2]))) / (2.0 * PI)
        du = du - du.detach().floor()
        return ts * ill, _sample2(luts["skyview"], du, vv) * ill

    def rays(self, frame, width, height, depth, rows):
        """Directions, clip distances, image coordinates and jitter of a band of rows."""
        y, x = torch.meshgrid(torch.arange(rows[0], rows[1], device=DEV), torch.arange(width, device=DEV), indexing="ij")
        x, y = x.reshape(-1), y.reshape(-1)
        u, v = (x.to(F64) + 0.5) / width, (y.to(F64) + 0.5) / height
        nx, ny = u * 2.0 - 1.0, 1.0 - v * 2.0
        d = _view_dirs(frame, nx, ny)
        clip = torch.full_like(u, 1e30)
        if depth is not None:
            dn = depth[rows[0]:rows[1]].reshape(-1).to(F64)
            t = _unproject(frame, nx, ny, dn).norm(dim=-1)
            clip = torch.where(dn > 0, t, clip)
        return d, clip, u, v, self.blue[y % 64, x % 64]

    def segment(self, L, oc, d, clip):
        rb, rt = self.w.planet_radius_m + L["base"], self.w.planet_radius_m + L["top"]
        b0, b1 = _sphere(oc, d, rb)
        t0, t1 = _sphere(oc, d, rt)
        r0 = float(oc.norm())
        if r0 < float(rb.detach()):
            lo, hi, ok = b1.clamp_min(0.0), t1.clamp_min(0.0), ~torch.isnan(b1) & ~torch.isnan(t1)
        else:
            first = torch.where(b0 > 0, b0, t1)
            lo, hi, ok = t0.clamp_min(0.0), torch.minimum(first, t1).clamp_min(0.0), ~torch.isnan(t1)
        hi = torch.minimum(hi, clip)
        return lo, hi, ok & (hi > lo)

    def march(self, frame, luts, width, height, depth, rows, layers):
        """(L, T) of a band of rows, (n, 3) each, with aerial perspective.  The
        camera stands below every layer, so layers are crossed bottom up."""
        d, clip, u, v, jit = self.rays(frame, width, height, depth, rows)
        n = d.shape[0]
        cam, sun = _vec(frame.camera_position_world), _vec(frame.sun_direction)
        oc = cam + torch.tensor([0.0, self.w.planet_radius_m, 0.0], dtype=F64, device=DEV)
        z = lambda *k: torch.zeros(*k, dtype=F64, device=DEV)  # noqa: E731
        Lum, T, tw, tn = z(n, 3), torch.ones(n, 3, dtype=F64, device=DEV), z(n), z(n)
        weights = torch.tensor([0.2126, 0.7152, 0.0722], dtype=F64, device=DEV)
        ss = _vec(self.p.sigma_s)
        for L in layers:
            lo, hi, hit = self.segment(L, oc, d, clip)
            st, skew = self.sigma_t(L), self.skew(L)
            ids = torch.nonzero(hit & (T.detach().amax(-1) >= 0.01))[:, 0]
            step = (hi - lo) / self.p.cloud_steps
            thick = (L["top"] - L["base"]).clamp_min(1.0)
            for k in range(self.p.cloud_steps):
                ids = ids[T.detach()[ids].amax(-1) >= 0.01]
                if ids.numel() == 0:
                    break
                t = lo[ids] + (k + jit[ids]) * step[ids]
                p = cam + d[ids] * t[:, None]
                alt, up = self.altitude(p)
                wr = _sample2(self.weather, p[:, 0] / self.p.weather_scale_m + 0.5, p[:, 2] / self.p.weather_scale_m + 0.5,
                              wrap=True)[:, 0]
                eff = _clamp01(wr * L["coverage"])
                den = self.density(L, skew, p, (alt - L["base"]) / thick, eff, False)
                sel = torch.nonzero(den.detach() > 1e-3)[:, 0]
                if sel.numel() == 0:
                    continue
                i, den, p, alt, up, eff, t = ids[sel], den[sel], p[sel], alt[sel], up[sel], eff[sel], t[sel]
                dist = ((L["top"] - alt) / max(float(sun[1]), 0.05)).clamp_min(1.0)
                ls, od = dist / self.p.light_steps, 0.0
                for j in range(self.p.light_steps):
                    q = p + sun * ((j + 0.5) * ls)[:, None]
                    qa, _ = self.altitude(q)
                    od = od + self.density(L, skew, q, (qa - L["base"]) / thick, eff, True) * ls
                hn = _clamp01((alt - L["base"]) / thick)
                sl, sky = self.lighting(luts, frame, alt, up)
                cos_t = (d[i] * sun).sum(-1)
                x = od[:, None] * st
                S, a, b, c = 0.0, 1.0, 1.0, 1.0
                for _ in range(self.p.multi_scatter_octaves):
                    S = S + (a * self.phase(L, cos_t, c, hn))[:, None] * torch.exp(-x * b)
                    a, b, c = a * self.p.multi_scatter_a, b * self.p.multi_scatter_b, c * self.p.multi_scatter_c
                beer = torch.exp(-x)
                pw = self.p.powder_strength
                energy = beer * (1.0 - pw) + beer * (1.0 - torch.exp(-2.0 * x)) * 2.0 * pw
                amb = sky * ((0.3 + 0.7 * hn) * self.p.ambient_strength)[:, None]
                ins = den[:, None] * ss * (S * sl * energy + amb)
                ext = (den[:, None] * st).clamp_min(1e-6)
                tr = torch.exp(-ext * step[i][:, None])
                add = T[i] * ins * (1.0 - tr) / ext
                w = add @ weights
                Lum, T = Lum.index_add(0, i, add), T.index_copy(0, i, T[i] * tr)
                tw, tn = tw.index_add(0, i, w * t), tn.index_add(0, i, w)
        op = 1.0 - T @ weights
        az = _clamp01(torch.log((tw / tn.clamp_min(1e-6)).clamp_min(50.0) / 50.0) / math.log(100000.0 / 50.0))
        ap = _sample3(luts["aerial"], u * 32.0 - 0.5, v * 32.0 - 0.5, az * 64.0 - 0.5, False)
        out = Lum * ap[:, 3:4] + ap[:, :3] * op[:, None]
        return torch.where((op > 1e-4)[:, None], out, Lum), T

    def image(self, frame, luts, width, height, depth):
        """The cloud RT: L and T of shape (height, width, 4), in bands of about half a million rays."""
        band = max(1, (1 << 19) // width)
        parts = [self.march(frame, luts, width, height, depth, (y, min(height, y + band)), self.layers(frame))
                 for y in range(0, height, band)]
        one = torch.ones(height, width, 1, dtype=F64, device=DEV)
        return [torch.cat([torch.cat(k).reshape(height, width, 3), one], -1) for k in zip(*parts)]


def _composite(l, t, bg):
    return l + bg.to(F64) * t


def _catmull_rom(img, width, height):
    """An RT reconstructed at every pixel of a larger image, 4x4 taps on clamped texels."""
    for axis, n in ((0, height), (1, width)):
        m = img.shape[axis]
        sp = (torch.arange(n, device=DEV, dtype=F64) + 0.5) / n * m
        b = (sp - 0.5).floor()
        f = sp - (b + 0.5)
        w = [f * (-0.5 + f * (1.0 - 0.5 * f)), 1.0 + f * f * (-2.5 + 1.5 * f), f * (0.5 + f * (2.0 - 1.5 * f)),
             f * f * (-0.5 + 0.5 * f)]
        out = 0.0
        for k in range(4):
            i = (b.long() - 1 + k).clamp(0, m - 1)
            out = out + img.index_select(axis, i) * (w[k][:, None, None] if axis == 0 else w[k][None, :, None])
        img = out
    return img


def _resolve(f, l, t, hist_l, hist_t):
    """The temporal resolve of one frame against the last one's."""
    h, w = l.shape[:2]
    y, x = torch.meshgrid((torch.arange(h, device=DEV, dtype=F64) + 0.5) / h,
                          (torch.arange(w, device=DEV, dtype=F64) + 0.5) / w, indexing="ij")
    d = _view_dirs(f, x.reshape(-1) * 2.0 - 1.0, 1.0 - y.reshape(-1) * 2.0)
    m = _mat(f.prev_view_proj)
    pc = m[0] * d[:, 0:1] + m[1] * d[:, 1:2] + m[2] * d[:, 2:3]
    pu, pv = pc[:, 0] / pc[:, 3] * 0.5 + 0.5, 1.0 - (pc[:, 1] / pc[:, 3] * 0.5 + 0.5)
    ok = (pc[:, 3] > 1e-4) & (pu >= 0) & (pu <= 1) & (pv >= 0) & (pv <= 1)
    k = torch.where(ok, torch.full_like(pu, 0.125), torch.ones_like(pu)).reshape(h, w, 1)
    out = []
    for cur, hist in ((l, hist_l), (t, hist_t)):
        old = _sample2(hist, pu, pv).reshape(h, w, 4)
        pad = torch.nn.functional.pad(cur.permute(2, 0, 1)[None], (1, 1, 1, 1), mode="replicate")[0]
        near = torch.stack([pad[:, i:i + h, j:j + w] for i in range(3) for j in range(3)])
        old = torch.minimum(torch.maximum(old, near.amin(0).permute(1, 2, 0)), near.amax(0).permute(1, 2, 0))
        out.append(old * (1.0 - k) + cur * k)
    return out[0].clamp_min(0.0), out[1].clamp(0.0, 1.0)


def _exact_frame(s, sub):
    e = _Exact(s, sub)
    depth, bg, _ = _render_context(s)
    l, t = e.image(s.frame, _frame_luts(s.world, s.frame, e.statics), s.width, s.height, depth)
    return l, t, _composite(l, t, bg)


def _exact_flight(s, frames, sub):
    e = _Exact(s, sub)
    rw, rh = max(1, s.width // 2), max(1, s.height // 2)
    xs = (torch.arange(rw, device=DEV, dtype=F64) * (s.width / rw)).long().clamp(max=s.width - 1)
    ys = (torch.arange(rh, device=DEV, dtype=F64) * (s.height / rh)).long().clamp(max=s.height - 1)
    hist, out = None, []
    for f in frames:
        depth, bg, _ = _render_context(s, f)
        l, t = e.image(f, _frame_luts(s.world, f, e.statics), rw, rh, depth[ys][:, xs])
        hist = (l, t) if hist is None else _resolve(f, l, t, *hist)
        big_l, big_t = [_catmull_rom(k, s.width, s.height) for k in hist]
        out.append(_composite(big_l.clamp_min(0.0), big_t.clamp(0.0, 1.0), bg))
    return out


def _exact_batch(lists, sub):
    out = []
    for scs in lists:
        imgs = []
        for s in scs:
            imgs.append(_exact_frame(s, sub)[2])
        out.append(imgs)
    return out


PARAMS = ("coverage", "shape", "detail", "scale", "base", "top")  # in the gradient's order


def _exact_layer_params(s, sub, layer, target):
    """The loss and its derivative along each parameter in turn."""
    e = _Exact(s, sub)
    depth, bg, _ = _render_context(s)
    luts = _frame_luts(s.world, s.frame, e.statics)
    inv = 1.0 / (3.0 * s.width * s.height)
    bg3, tg3 = bg[..., :3].to(F64).reshape(-1, 3), target[..., :3].to(F64).reshape(-1, 3)
    grad, loss = [], 0.0
    for name in PARAMS:
        with fwAD.dual_level():
            layers = e.layers(s.frame)
            layers[layer][name] = fwAD.make_dual(layers[layer][name], torch.ones((), dtype=F64, device=DEV))
            l, t = e.march(s.frame, luts, s.width, s.height, depth, (0, s.height), layers)
            dual = fwAD.unpack_dual((((l + bg3 * t) - tg3) ** 2).sum() * inv)
            loss = dual.primal
            grad.append(dual.tangent if dual.tangent is not None else torch.zeros_like(loss))
    return torch.stack(grad), loss.reshape(1)


class _ExactGrid:
    """The voxel form: density from a grid, every step contributing."""

    def __init__(self, s, sub, values):
        self.e, self.s, self.spec = _Exact(s, sub), s, s.extra["grid_spec"]
        ny, nz, nx = self.n = values.shape
        self.pad = torch.zeros(ny + 2, nz + 2, nx + 2, dtype=F64, device=DEV)
        self.pad[1:-1, 1:-1, 1:-1] = values.to(F64)
        self.luts = _frame_luts(s.world, s.frame, self.e.statics)

    def coords(self, L, x, alt, z):
        ny, nz, nx = self.n
        sp = self.spec
        c = [(alt - L["base"]) * (ny / (L["top"] - L["base"]).clamp_min(1.0)) - 0.5,
             (z - sp["min_z_m"]) * (nz / sp["size_z_m"]) - 0.5, (x - sp["min_x_m"]) * (nx / sp["size_x_m"]) - 0.5]
        f = [k.detach().floor() for k in c]
        return [g.long() for g in f], [k - g for k, g in zip(c, f)]

    def corners(self, i, w):
        """(flat padded index, weight) of the eight corners."""
        ny, nz, nx = self.n
        for a in range(2):
            for b in range(2):
                for c in range(2):
                    y, z, x = [(k + o + 1).clamp(0, m + 1) for k, o, m in zip(i, (a, b, c), (ny, nz, nx))]
                    wt = (w[0] if a else 1 - w[0]) * (w[1] if b else 1 - w[1]) * (w[2] if c else 1 - w[2])
                    yield (y * (nz + 2) + z) * (nx + 2) + x, wt

    def fetch(self, i, w):
        flat = self.pad.reshape(-1)
        return sum(flat[k] * wt for k, wt in self.corners(i, w))

    def rows(self, rows, L, taps=None):
        """The samples of a band of rows: grid value and light sum, (n, steps)
        each, and what the step integral needs.  `taps` receives the grid
        coordinates of each sum's fetches."""
        e, s = self.e, self.s
        d, clip, _, _, jit = e.rays(s.frame, s.width, s.height, None, rows)
        cam, sun = _vec(s.frame.camera_position_world), _vec(s.frame.sun_direction)
        oc = cam + torch.tensor([0.0, s.world.planet_radius_m, 0.0], dtype=F64, device=DEV)
        lo, hi, hit = e.segment(L, oc, d, clip)
        lo, hi = torch.where(hit, lo, torch.zeros_like(lo)), torch.where(hit, hi, torch.zeros_like(hi))
        n, S = d.shape[0], s.params.cloud_steps
        step = (hi - lo) / S
        t = (lo[:, None] + (torch.arange(S, device=DEV, dtype=F64) + jit[:, None]) * step[:, None]).reshape(-1)
        p = cam + d.repeat_interleave(S, 0) * t[:, None]
        alt, up = e.altitude(p)
        i, w = self.coords(L, p[:, 0], alt, p[:, 2])
        gv = self.fetch(i, w)
        if taps is not None:
            taps.append((i, w, None))
        ls = ((L["top"] - alt) / max(float(sun[1]), 0.05)).clamp_min(1.0) / s.params.light_steps
        gl = 0.0
        for j in range(s.params.light_steps):
            q = p + sun * ((j + 0.5) * ls)[:, None]
            qa, _ = e.altitude(q)
            i, w = self.coords(L, q[:, 0], qa, q[:, 2])
            gl = gl + self.fetch(i, w)
            if taps is not None:
                taps.append((i, w, ls))
        sl, sky = e.lighting(self.luts, s.frame, alt, up)
        hn = _clamp01((alt - L["base"]) / (L["top"] - L["base"]).clamp_min(1.0))
        amb = sky * ((0.3 + 0.7 * hn) * s.params.ambient_strength)[:, None]
        shape = lambda k: k.reshape((n, S) + k.shape[1:])  # noqa: E731
        return dict(gv=shape(gv), gl=shape(gl * ls), sl=shape(sl), amb=shape(amb), step=step, hit=hit,
                    cos=(d * sun).sum(-1))

    def scale(self, L):
        return 3.0 / float(self.e.sigma_t(L).sum())

    def shade(self, L, r, gv, gl, k):
        """(L, T) of the band's rays, (n, 3), from grid values and light sums times k."""
        p, st = self.s.params, self.e.sigma_t(L)
        x = (k * gl)[..., None] * st
        S, a, b, c = 0.0, 1.0, 1.0, 1.0
        for _ in range(p.multi_scatter_octaves):
            ph = self.e.phase(L, r["cos"], c, torch.zeros_like(r["cos"]))
            S = S + (a * ph)[:, None, None] * torch.exp(-x * b)
            a, b, c = a * p.multi_scatter_a, b * p.multi_scatter_b, c * p.multi_scatter_c
        beer = torch.exp(-x)
        energy = beer + p.powder_strength * (2.0 * beer * (1.0 - beer * beer) - beer)
        X = S * r["sl"] * energy + r["amb"]
        tau = (k * gv * r["step"][:, None])[..., None] * st
        before = tau.cumsum(1) - tau
        on = (torch.exp(-before.detach()).amax(-1) >= self.spec["exit_transmittance"]) & r["hit"][:, None]
        tau = torch.where(on[..., None], tau, torch.zeros_like(tau))
        Tb = torch.exp(-(tau.cumsum(1) - tau))
        lum = (Tb * X * (-torch.expm1(-tau)) * (_vec(p.sigma_s) / st)).sum(1)
        return lum, torch.exp(-tau.sum(1))

    def bands(self):
        band = max(1, 16384 // self.s.width)
        return [(y, min(self.s.height, y + band)) for y in range(0, self.s.height, band)]

    def render(self):
        L = self.e.layers(self.s.frame)[0]
        k = self.scale(L) * self.spec["density_scale"]
        out = []
        for rows in self.bands():
            r = self.rows(rows, L)
            out.append(self.shade(L, r, r["gv"], r["gl"], k))
        return [self.whole(torch.cat(v)) for v in zip(*out)]

    def whole(self, rgb):
        h, w = self.s.height, self.s.width
        return torch.cat([rgb.reshape(h, w, 3), torch.ones(h, w, 1, dtype=F64, device=DEV)], -1)

    def adjoint(self, bg, target):
        L = self.e.layers(self.s.frame)[0]
        w, h = self.s.width, self.s.height
        ks = self.scale(L)
        grad = torch.zeros(self.pad.numel(), dtype=F64, device=DEV)
        loss, dscale, out = 0.0, 0.0, []
        for rows in self.bands():
            taps = []
            r = self.rows(rows, L, taps)
            gv, gl = r["gv"].requires_grad_(), r["gl"].requires_grad_()
            ds = torch.tensor(self.spec["density_scale"], dtype=F64, device=DEV, requires_grad=True)
            lum, tr = self.shade(L, r, gv, gl, ks * ds)
            b, t = [k[rows[0]:rows[1], :, :3].to(F64).reshape(-1, 3) for k in (bg, target)]
            part = ((lum + b * tr - t) ** 2).sum() / (3.0 * w * h)
            dv, dl, dd = torch.autograd.grad(part, (gv, gl, ds))
            out.append((lum.detach(), tr.detach()))
            loss, dscale = loss + part.detach(), dscale + dd
            for i, wt, ls in taps:
                g = dv.reshape(-1) if ls is None else dl.reshape(-1) * ls
                for idx, c in self.corners(i, wt):
                    grad.index_add_(0, idx, g * c)
        ny, nz, nx = self.n
        grad = grad.reshape(ny + 2, nz + 2, nx + 2)[1:-1, 1:-1, 1:-1].contiguous()
        lum, tr = [self.whole(torch.cat(v)) for v in zip(*out)]
        return {"luminance": lum, "transmittance": tr, "grad": grad, "acc": torch.stack([loss, dscale])}

    def range_gradient(self, bg, target):
        w, h = self.s.width, self.s.height
        out = []
        for name in ("base", "top"):
            total = 0.0
            for rows in self.bands():
                with fwAD.dual_level():
                    L = self.e.layers(self.s.frame)[0]
                    k = self.scale(L) * self.spec["density_scale"]
                    L[name] = fwAD.make_dual(L[name], torch.ones((), dtype=F64, device=DEV))
                    r = self.rows(rows, L)
                    lum, tr = self.shade(L, r, r["gv"], r["gl"], k)
                    b, t = [c[rows[0]:rows[1], :, :3].to(F64).reshape(-1, 3) for c in (bg, target)]
                    total = total + fwAD.unpack_dual(((lum + b * tr - t) ** 2).sum() / (3.0 * w * h)).tangent
            out.append(total)
        return torch.stack(out)


def exact(case, seed):
    """What `run` returns, in 64 bits.  The context made here supplies the
    noise volumes (bytes, an input of the march) and nothing else."""
    kind = case["kind"]
    if kind == "batch":
        now, then = _batch_scenes(case, seed)
        st = _State(sub=subsystem_for_scene(now[0]))
        a, b = _exact_batch((now, then), st.sub)
        return {"first": a, "second": b}
    if kind == "flight":
        s, frames = _flight_scenes(case, seed)
        st = _State(sub=subsystem_for_scene(s))
        a, b = _exact_flight(s, frames, st.sub)
        return {"first": a, "second": b}
    if kind in ("frame", "first_frame"):
        s = _frame_scene(case, seed)
        st = _State(sub=subsystem_for_scene(s))
        l, t, c = _exact_frame(s, st.sub)
        return {"color": c} if case["fused"] else {"color": c, "luminance": l, "transmittance": t}
    if kind == "layer_params":
        s = _frame_scene(case, seed)
        st = _State(sub=subsystem_for_scene(s))
        _, bg, _ = _render_context(s)
        grad, loss = _exact_layer_params(s, st.sub, seed % s.n_layers, _noisy(bg, seed, 0.05))
        return {"grad": grad, "loss": loss}
    s = _grid_scene(case, seed)
    st = _State(sub=subsystem_for_scene(s))
    g = _ExactGrid(s, st.sub, _worley(case, seed))
    if kind == "grid":
        l, t = g.render()
        return {"luminance": l, "transmittance": t}
    bg = torch.from_numpy(np.ascontiguousarray(s.background, np.float32)).to(DEV)
    if kind == "adjoint":
        return g.adjoint(bg, _target(bg, seed))
    return {"range": g.range_gradient(bg, _target(bg, seed))}
