"""The work that is measured: what programs built on this library have it do, through its public entry
points, from a thumbnail to a 1080p frame of four rays a pixel, in every precision, and around the trace
the renderer's frame, its disc inputs, batches of views and the gradients of an image loss.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` makes what a program holds
before a call, `run` makes the call and returns its outputs, `work` says what it cannot do without, and
`exact` evaluates the same images, losses and gradients in 64 bits with plain torch operations.

A case's "kind" is the entry point:
  trace    artfCudaHoleTrace: one frame into device memory
  render   artfCudaHoleRender: one frame, host map and fluid in, host frame out
  batch    artfCudaBatchGraphLaunch / artfCudaHoleBatch: many uneven views in one launch
  adjoint  fit.HoleLoss, forward and backward: a loss and its gradient in the five scene parameters
  frame    the renderer backend's table: a gas step, the trace, bloom, tone map, the pixels read back
  gas      artfCudaFluidAdvance: the disc's gas moved on
  disc     artfCudaPaintDisc and artfCudaFluidNew: the inputs of a new disc or spin
"""
from __future__ import annotations

import ctypes as C
import math
from types import SimpleNamespace

import numpy as np
import torch

from artful_gb300 import capi, fit, scenes

PRECISION = {"exact": capi.EXACT, "fp32": capi.FP32, "fp64": capi.FP64, "mixed": capi.MIXED}
STEPS = 26  # a ray's steps on the benchmark views, on average (25.3 to 27)


# ---- the cases ---------------------------------------------------------------------------------------

def _trace(name, precision, width, height, **more):
    case = {"name": name, "kind": "trace", "precision": precision, "width": width, "height": height, "jitter": 0,
            "samples": 1, "spin": 0.9, "inclination": 80.0, "distance": 30.0, "moving": False, "ends": False}
    return {**case, **more}


def listed():
    return [
        # the first picture a user makes: the plain method's small frame, in the reference's own bits
        _trace("first_look_320x180", "exact", 320, 180),
        # a thumbnail of an odd size from a moving eye, with each ray's end record: latency counts
        _trace("thumbnail_101x67", "mixed", 101, 67, spin=0.6, inclination=70.0, distance=26.0, moving=True, ends=True),
        # a preview in fast FP32, 2 x 2 stratified rays a pixel
        _trace("preview_1280x720", "fp32", 1280, 720, samples=2, spin=0.6, inclination=60.0),
        # the plain FP64 trace that other precisions are checked against, a quarter of a 1080p frame
        _trace("fp64_960x540", "fp64", 960, 540, spin=0.998, inclination=85.0, distance=50.0),
        # the headline frame: 1080p, four jittered rays a pixel, mixed precision
        _trace("headline_1080p_x4", "mixed", 1920, 1080, jitter=4, spin=0.998, inclination=85.0, distance=50.0),
        # a program without CUDA memory of its own: host buffers in, a host frame out
        {"name": "render_1080p_host", "kind": "render", "precision": "mixed", "width": 1920, "height": 1080, "jitter": 0,
         "samples": 1, "spin": 0.9, "inclination": 75.0, "distance": 40.0, "moving": False, "pinned": False},
        # a training set's worth of uneven views in one captured launch
        {"name": "batch_64_views", "kind": "batch", "views": 64, "most": 1280, "graph": True, "jitter": 0},
        # one gradient of a full-size view with a checkpoint every 32 steps
        {"name": "adjoint_512x288", "kind": "adjoint", "views": 1, "width": 512, "height": 288, "checkpoint": 32},
        # one optimiser step of 32 independent fits, every state kept
        {"name": "fit_step_32x256x144", "kind": "adjoint", "views": 32, "width": 256, "height": 144, "checkpoint": 1},
        # an application's frame: the gas a step on, trace, bloom, tone map, BGRA in a host array
        {"name": "frame_1080p", "kind": "frame", "precision": "exact", "width": 1920, "height": 1080, "samples": 1,
         "spin": 0.9, "inclination": 80.0, "distance": 30.0, "outer": 12.0, "bloom": 4.5},
        # an animation's clock jumping ahead: the gas caught up
        {"name": "gas_24_steps", "kind": "gas", "steps": 24, "spin": 0.9, "outer": 12.0},
        # the disc or the spin changed: its map painted, its gas started
        {"name": "new_disc", "kind": "disc", "spin": 0.6, "outer": 34.0},
    ]


def draw(rng):
    def size(least, most):
        w = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
        return w, max(1, int(round(w * rng.choice((9 / 16, 9 / 16, 3 / 4, 0.41)))))

    def view():
        return {"spin": round(rng.uniform(-0.5, 0.998), 3), "inclination": round(rng.uniform(5.0, 89.0), 1),
                "distance": round(rng.uniform(20.0, 80.0), 1)}

    kind = rng.choice(("trace", "trace", "trace", "trace", "render", "batch", "adjoint", "adjoint", "frame", "gas", "disc"))
    if kind in ("trace", "render"):
        precision = rng.choice(("exact", "fp32", "mixed", "mixed", "fp64" if kind == "trace" else "mixed"))
        w, h = size(60, 960 if precision == "fp64" else 1920)
        jitter, samples = rng.choice(((0, 1), (0, 1), (0, 2), (4, 1), (3, 1)))
        if precision == "fp64" or w * h * max(jitter, samples * samples) > 8300000:
            jitter, samples = 0, 1
        case = {"kind": kind, "precision": precision, "width": w, "height": h, "jitter": jitter, "samples": samples,
                "moving": rng.random() < 0.25, **view()}
        return {**case, **({"ends": rng.random() < 0.25} if kind == "trace" else {"pinned": rng.random() < 0.5})}
    if kind == "batch":
        most = rng.choice((320, 640, 1280))
        return {"kind": kind, "views": rng.randint(2, 64), "most": most, "graph": rng.random() < 0.5,
                "jitter": rng.choice((0, 0, 0, 2 if most < 1280 else 0))}
    if kind == "adjoint":
        w, h = size(64, 512)
        return {"kind": kind, "views": rng.randint(1, max(1, min(32, 1100000 // (w * h)))), "width": w, "height": h,
                "checkpoint": rng.choice((1, 1, 8, 20, 32, 64))}
    if kind == "frame":
        w, h = size(100, 1920)
        return {"kind": kind, "precision": rng.choice(("exact", "exact", "mixed", "fp32")), "width": w, "height": h,
                "samples": rng.choice((1, 1, 2)), "outer": rng.choice((12.0, 34.0)), "bloom": rng.choice((0.0, 4.5)),
                **view()}
    if kind == "gas":
        return {"kind": kind, "steps": rng.randint(1, 48), "spin": round(rng.uniform(-0.5, 0.99), 3),
                "outer": round(rng.uniform(12.0, 40.0), 1)}
    return {"kind": kind, "spin": round(rng.uniform(-0.5, 0.99), 3), "outer": round(rng.uniform(12.0, 40.0), 1)}


# ---- what a program holds ------------------------------------------------------------------------------

_shared = {}


def _context():
    """The one context a program makes, and keeps."""
    if "ctx" not in _shared:
        torch.zeros(1, device="cuda")
        ctx = C.c_void_p()
        capi.check(capi.load().artfCudaCreate(0, C.byref(ctx)))
        _shared["ctx"] = ctx
    return _shared["ctx"]


class _Held:
    """A state; `free` lets go of the library objects it owns."""

    def __init__(self, **items):
        self.free = None
        self.__dict__.update(items)

    def __del__(self):
        if self.free:
            self.free()


def _scene(case, rng, width, height):
    """The case's view, moved a little by the seed."""
    desc = scenes.hole_desc(case["spin"], samples=case["samples"], doppler=1.0,
                            shutter=2.0 if case["moving"] else 0.0, time=float(rng.uniform(0.0, 9.0)),
                            velocity=(0.2, 0.0, 0.1) if case["moving"] else (0.0, 0.0, 0.0))
    camera = scenes.camera(case["inclination"] + float(rng.uniform(-0.5, 0.5)), case["distance"])
    return scenes.Scene("case", desc, camera, width, height, seed=int(rng.integers(1, 1 << 30)),
                        emissivity=float(rng.uniform(2.5, 3.2)), jitter=case["jitter"], jitter_seed=int(rng.integers(1, 1 << 30)))


def _fluid(rng):
    """A gas of smooth clumps around 1."""
    x = np.arange(capi.FLUID_WIDTH) * (2 * np.pi / capi.FLUID_WIDTH)
    y = np.arange(capi.FLUID_HEIGHT)[:, None] / 40.0
    p, q = rng.uniform(0, 6, 2)
    return (1.0 + 0.4 * np.sin(3 * x + y + p) + 0.3 * np.cos(7 * x - 2 * y + q)).astype(np.float32).ravel()


def prepare(case, seed):
    lib, kind, rng = capi.load(), case["kind"], np.random.default_rng(seed)
    if kind in ("trace", "render"):
        scene = _scene(case, rng, case["width"], case["height"])
        frame, frame64, clamped = scenes.frame(scene)
        s = _Held(kind=kind, ctx=_context(), lib=lib, frame=frame, frame64=frame64)
        s.map = torch.from_numpy(scenes.synth_map(lib, clamped, scene.seed, scene.emissivity))
        s.fluid = torch.from_numpy(_fluid(rng))
        s.opts = capi.TraceOptions(PRECISION[case["precision"]], scene.jitter, scene.jitter_seed, 1.0, 0.0, 0, 0, 1)
        shape = (case["height"], case["width"], 4)
        if kind == "trace":
            s.map, s.fluid = s.map.cuda(), s.fluid.cuda()
            s.hdr = torch.empty(shape, dtype=torch.float32, device="cuda")
            rays = scene.jitter or case["samples"] ** 2
            s.ends = torch.empty((case["height"] * case["width"] * rays, 8), dtype=torch.float32, device="cuda") if case["ends"] else None
        else:
            s.hdr = torch.empty(shape, dtype=torch.float32, pin_memory=case["pinned"])
            s.version = seed * 4096 + int(rng.integers(1, 4096))  # (the map of this scene: copied when another was drawn)
        return s
    if kind == "batch":
        return _prepare_batch(case, rng, lib)
    if kind == "adjoint":
        return _prepare_adjoint(case, rng, lib, seed)
    if kind == "frame":
        opts = capi.RendererOptions(capi.BACKEND)
        opts.width, opts.height = case["width"], case["height"]
        r = lib.artfCudaNew(C.byref(opts))
        if not r:
            raise RuntimeError(lib.artfCudaLastError())
        lib.artfCudaRendererSetDeviceInputs(r, True)
        lib.artfCudaRendererSetPrecision(r, PRECISION[case["precision"]])
        scene = lib.artfCudaSceneNew()
        camera = scenes.camera(case["inclination"] + float(rng.uniform(-0.5, 0.5)), case["distance"])
        lib.artfCudaSceneSetCamera(scene, C.byref(camera))
        desc = scenes.hole_desc(case["spin"], outer=case["outer"], samples=case["samples"], time=float(rng.uniform(0.0, 50.0)))
        desc.bloom = case["bloom"]
        vt = C.cast(r, C.POINTER(capi.RendererHead)).contents.vt.contents
        s = _Held(kind=kind, lib=lib, r=r, scene=scene, vt=vt, desc=desc,
                  bgra=np.zeros((case["height"], case["width"]), np.uint32))
        s.free = lambda: (vt.destroy(r), lib.artfCudaSceneFree(scene))
        return s
    if kind == "gas":
        ctx = _context()
        clamped = scenes.clamp(scenes.hole_desc(case["spin"] + float(rng.uniform(-0.002, 0.002)), outer=case["outer"]))
        gas = _Gas(lib, ctx, (clamped.discInner, clamped.discOuter, clamped.spin))
        return _Held(kind=kind, lib=lib, gas=gas, time=0.0, by=0.2 * case["steps"], field=torch.as_tensor(gas, device="cuda"))
    clamped = scenes.clamp(scenes.hole_desc(case["spin"] + float(rng.uniform(-0.002, 0.002)), outer=case["outer"]))
    return _Held(kind=kind, lib=lib, ctx=_context(), disc=(clamped.discInner, clamped.discOuter, clamped.spin),
                 map=torch.empty(capi.MAP_FLOATS, dtype=torch.float32, device="cuda"), gas=None)


class _Gas:
    """A gas of the library's; as a tensor, its field in device memory, which keeps the gas."""

    def __init__(self, lib, ctx, disc):
        self.lib, self.handle = lib, C.c_void_p()
        capi.check(lib.artfCudaFluidNew(ctx, *disc, 0.0, C.byref(self.handle)))
        self.__cuda_array_interface__ = {"data": (lib.artfCudaFluidField(self.handle), False), "typestr": "<f4", "version": 2,
                                         "shape": (capi.FLUID_HEIGHT, capi.FLUID_WIDTH), "strides": None}

    def __del__(self):
        self.lib.artfCudaFluidFree(self.handle)


def _prepare_batch(case, rng, lib):
    """Views of uneven size, spin, inclination and distance, each with its own map: the painted part
    shared, the rings its own."""
    views, keep, frames, host = [], [], [], None
    widths = np.random.default_rng(case["views"]).integers(case["most"] // 10, case["most"] + 1, case["views"])
    for w in (int(w) for w in widths):
        desc, camera = scenes.hole_desc(float(rng.uniform(0.0, 0.998))), scenes.camera(float(rng.uniform(5.0, 89.0)), float(rng.uniform(20.0, 80.0)))
        scene = scenes.Scene("view", desc, camera, w, max(1, w * 9 // 16), seed=int(rng.integers(1, 1 << 30)) if host is None else scene.seed)
        frame, frame64, clamped = scenes.frame(scene)
        if host is None:
            host = scenes.synth_map(lib, clamped, scene.seed, 3.0)
            base, fluid = torch.from_numpy(host).cuda(), torch.from_numpy(_fluid(rng)).cuda()
        rings = capi.SynthDesc(scene.seed, clamped.discInner, clamped.discOuter, clamped.spin, 3.0, 2000)
        lib.artfCudaSynthRings(C.byref(rings), host.ctypes.data)
        m = base.clone()
        m[capi.ROWS_AT:capi.COLORS_AT] = torch.from_numpy(host[capi.ROWS_AT:capi.COLORS_AT]).cuda()
        m[capi.GLOW_AT:capi.DUST_AT] = torch.from_numpy(host[capi.GLOW_AT:capi.DUST_AT]).cuda()
        hdr = torch.empty((scene.height, scene.width, 4), dtype=torch.float32, device="cuda")
        views.append(capi.View(frame, frame64, m.data_ptr(), fluid.data_ptr(), hdr.data_ptr(), None))
        keep.append((m, fluid, hdr))
        frames.append((frame, frame64))
    s = _Held(kind="batch", lib=lib, ctx=_context(), keep=keep, frames=frames, graph=None)
    s.table = (capi.View * len(views))(*views)
    s.opts = capi.TraceOptions(capi.MIXED, case["jitter"], int(rng.integers(1, 1 << 30)), 1.0, 0.0, 0, 0, 1)
    # (the images as the batch leaves them, in a list of at most 64 views)
    s.hdr = [k[2] for k in keep]
    if case["graph"]:
        graph = C.c_void_p()
        torch.cuda.synchronize()
        capi.check(lib.artfCudaBatchGraphCreate(s.ctx, s.table, len(views), C.byref(s.opts), C.byref(graph)))
        s.graph = graph
        s.free = lambda: lib.artfCudaBatchGraphDestroy(graph)
    return s


def _prepare_adjoint(case, rng, lib, seed):
    """Fits of spin, inclination and inner radius: target images (the exact trace's) and starts off by 15 %."""
    w, h, n, ctx = case["width"], case["height"], case["views"], _context()
    fits = fit.config5_fits(n, seed=seed % (1 << 30))
    fluid = torch.from_numpy(_fluid(rng)).cuda()
    targets = torch.empty((n, h, w, 4), dtype=torch.float32, device="cuda")
    opts = capi.TraceOptions(capi.EXACT, 0, 0, 1.0, 0.0, 0, 0, 1)
    base = torch.from_numpy(fit.param_map(fits[0][0])).cuda()
    for k, (target, _) in enumerate(fits):
        frame = fit.frames(target, w, h)[0]
        m = base if k == 0 else torch.from_numpy(fit.param_map(target)).cuda()
        torch.cuda.synchronize()
        capi.check(lib.artfCudaHoleTrace(ctx, C.byref(frame), None, m.data_ptr(), fluid.data_ptr(), C.byref(opts),
                                         targets[k].data_ptr(), None, None))
        torch.cuda.synchronize()
    starts = [start for _, start in fits]
    adjoint = fit.Adjoint(lib, ctx, w, h, base.data_ptr(), fluid.data_ptr(), checkpoint=case["checkpoint"])
    # the parameters as a training script holds them: a host tensor of torch's default type
    theta = torch.tensor(np.stack([fit.theta_of(p) for p in starts]), dtype=torch.float32, requires_grad=True)
    return _Held(kind="adjoint", adjoint=adjoint, loss=fit.hole_loss(), theta=theta, starts=starts, targets=targets,
                 map=base, fluid=fluid)


# ---- one pass ------------------------------------------------------------------------------------------

def run(s):
    if s.kind == "trace":
        capi.check(s.lib.artfCudaHoleTrace(s.ctx, C.byref(s.frame), C.byref(s.frame64), s.map.data_ptr(), s.fluid.data_ptr(),
                                           C.byref(s.opts), s.hdr.data_ptr(), s.ends.data_ptr() if s.ends is not None else None, None))
        out = _image(s.hdr)
        if s.ends is not None:
            out["hit"], out["escape"], out["mino"] = s.ends[:, 0:2], s.ends[:, 2:5], s.ends[:, 5]
            out["counts"] = s.ends.view(torch.int16)[:, 12:15]  # steps, crossings and kind, wide steps
        return out
    if s.kind == "render":
        stats = capi.TraceStats()
        capi.check(s.lib.artfCudaHoleRender(s.ctx, C.byref(s.frame), C.byref(s.frame64), s.map.data_ptr(), s.version, s.fluid.data_ptr(),
                                            s.version, C.byref(s.opts), s.hdr.data_ptr(), C.byref(stats)))
        return _image(s.hdr)
    if s.kind == "batch":
        if s.graph is not None:
            capi.check(s.lib.artfCudaBatchGraphLaunch(s.graph, None))
        else:
            capi.check(s.lib.artfCudaHoleBatch(s.ctx, s.table, len(s.table), C.byref(s.opts), None))
        return s.hdr
    if s.kind == "adjoint":
        s.theta.grad = None
        loss = s.loss.apply(s.theta, s.adjoint, s.starts, s.targets)
        loss.sum().backward()
        return {"loss": loss.detach(), "grad": s.theta.grad}
    if s.kind == "frame":
        s.desc.time += 0.2  # (one gas step a frame)
        s.lib.artfCudaSceneSetBlackHole(s.scene, C.byref(s.desc))
        if not s.vt.draw(s.r, s.scene) or not s.vt.readPixels(s.r, s.bgra.ctypes.data):
            raise RuntimeError(s.lib.artfCudaLastError())
        return s.bgra
    if s.kind == "gas":
        s.time += s.by
        capi.check(s.lib.artfCudaFluidAdvance(s.gas.handle, s.time + 0.05, None))
        return s.field
    capi.check(s.lib.artfCudaPaintDisc(s.ctx, s.map.data_ptr(), *s.disc))
    s.gas = _Gas(s.lib, s.ctx, s.disc)  # (the gas of the last disc goes with its last reader)
    return {"map": s.map, "gas": torch.as_tensor(s.gas, device="cuda")}


def _image(hdr):
    """A frame's light, and its pixels' classes."""
    return {"light": hdr[..., :3], "classes": hdr[..., 3]}


# ---- what a pass cannot do without ---------------------------------------------------------------------

def work(case):
    """Bytes: the map and gas read once, the frame and records written once.  Operations: 4,030 a ray (100 a
    ray, 149 a step, a crossing's 375 for half the rays), three times that with its gradient; a gas step's 130
    a cell and a painted texel's 30 lattice points of 40."""
    kind, inputs = case["kind"], 4.0 * (capi.MAP_FLOATS + capi.FLUID_FLOATS)
    ray = 100 + 149 * STEPS + 60
    if kind in ("trace", "render"):
        pixels = case["width"] * case["height"]
        rays = pixels * (case["jitter"] or case["samples"] ** 2)
        return {"bytes": inputs + 16 * pixels + (32 * rays if case.get("ends") else 0), "flops": rays * ray}
    if kind == "batch":
        w = 0.55 * case["most"]
        pixels = case["views"] * 1.16 * w * w * 9 / 16
        return {"bytes": case["views"] * 4.0 * capi.MAP_FLOATS + 4.0 * capi.FLUID_FLOATS + 16 * pixels,
                "flops": pixels * max(1, case["jitter"]) * ray}
    if kind == "adjoint":
        pixels = case["views"] * case["width"] * case["height"]
        return {"bytes": inputs + 16 * pixels, "flops": 3 * pixels * ray}
    if kind == "frame":
        pixels = case["width"] * case["height"]
        return {"bytes": inputs + 8 * pixels + 2 * 7 * 4.0 * capi.FLUID_FLOATS,
                "flops": pixels * (case["samples"] ** 2 * ray + 200) + 130 * capi.FLUID_FLOATS}
    if kind == "gas":
        return {"bytes": 7 * 4.0 * capi.FLUID_FLOATS, "flops": case["steps"] * 130.0 * capi.FLUID_FLOATS}
    texels = capi.MAP_FLOATS
    return {"bytes": 4.0 * (texels + 7 * capi.FLUID_FLOATS), "flops": 1200.0 * texels + 60 * 130.0 * capi.FLUID_FLOATS}


# ---- the same in 64 bits, with torch alone --------------------------------------------------------------

def exact(case, seed):
    """The images, ray ends, losses and gradients of the same inputs from the equations in double.  Pixels of
    the renderer are bytes, and the gas and the painted map are held to the reference's own float bytes: they
    have no other value."""
    if case["kind"] not in ("trace", "render", "batch", "adjoint"):
        return None
    s = prepare(case, seed)
    torch.cuda.synchronize()
    if case["kind"] in ("trace", "render"):
        wide = case["precision"] in ("fp64", "mixed")
        f = _frame_of(s.frame64 if wide else s.frame)
        image, ends = _image64(s.frame, f, s.map.cuda(), s.fluid.cuda(), s.opts.jitter, s.opts.seed, case.get("ends"))
        out = _image(image)
        if ends is not None:
            out["hit"], out["escape"], out["mino"] = ends[:, 0:2], ends[:, 2:5], ends[:, 5]
            out["counts"] = None
        return out
    if case["kind"] == "batch":
        return [_image64(frame, _frame_of(frame64), m, fluid, s.opts.jitter, s.opts.seed, False)[0]
                for (frame, frame64), (m, fluid, _) in zip(s.frames, s.keep)]
    w, h = case["width"], case["height"]
    losses, grads = [], []
    for k, (start, values) in enumerate(zip(s.starts, s.theta.detach().numpy())):
        p = fit.with_theta(start, values)
        frame, _, jac = fit.frames(p, w, h)
        f = _frame_of(frame)
        f.q = float(np.float32(p.emissivity))
        fields = None
        if len(s.starts) == 1:
            fields = torch.tensor(_fields(f) + [f.q], dtype=torch.float64, device="cuda", requires_grad=True)
            _set_fields(f, fields)
        nx, ny, t = _positions(frame, 0, 0)
        rgb = _trace64(f, s.map, s.fluid, nx[0], ny[0], t[0])[0]
        loss = (rgb - s.targets[k].reshape(-1, 4)[:, :3].double()).square().sum() / (3 * w * h)
        losses.append(float(loss.detach()))
        if fields is not None:
            loss.backward()
            g = fields.grad.cpu().numpy()
            total = g[:28] @ jac
            total[3] += g[28]
            grads.append(total)
    return {"loss": torch.tensor(losses, dtype=torch.float64), "grad": torch.tensor(np.array(grads)) if grads else None}


def _k(x):
    """A constant as the equations hold it: a float's value."""
    return float(np.float32(x))


def _frame_of(f):
    g = SimpleNamespace(**{n: [float(v) for v in getattr(f, n)] for n in capi.FRAME_FIELDS})
    g.a, g.horizon, g.height, g.inner, g.outer, g.thickness = g.spin[0], g.spin[1], g.spin[2], g.disc[0], g.disc[1], g.disc[3]
    g.gain, g.doppler, g.stars = g.look[0], g.look[1], g.look[2]
    g.q = None
    return g


def _fields(f):
    """The 28 fields the gradient goes through, in their order."""
    return (f.forward[:3] + f.right[:3] + f.up[:3] + f.metric + f.place + f.er[:3] + f.etheta[:3] + f.ephi[:3] + [f.a, f.inner])


def _set_fields(f, t):
    f.forward, f.right, f.up, f.metric, f.place = t[0:3], t[3:6], t[6:9], t[9:13], t[13:17]
    f.er, f.etheta, f.ephi, f.a, f.inner, f.q = t[17:20], t[20:23], t[23:26], t[26], t[27], t[28]


def _mix32(x):
    m = 0xFFFFFFFF
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & m
    x = x ^ (x >> 15)
    x = (x * 0x846CA68B) & m
    return x ^ (x >> 16)


def _positions(frame, jitter, seed):
    """Each ray's image position and moment, in the floats they are given in: (rays, pixels)."""
    w, h, side = int(frame.size[0]), int(frame.size[1]), int(frame.size[2])
    f32 = torch.float32
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    x, y = x.reshape(-1), y.reshape(-1)
    px, py = torch.tensor(frame.image[1], dtype=f32, device="cuda"), torch.tensor(frame.image[2], dtype=f32, device="cuda")
    nx, ny, t = [], [], []
    for k in range(jitter or side * side):
        if jitter:
            base = _mix32(torch.tensor((seed ^ 0xA511E9B3) & 0xFFFFFFFF, device="cuda"))
            base = _mix32(base ^ (y * w + x))
            dx = (_mix32((base + 2 * k) & 0xFFFFFFFF) >> 8).to(f32) * (1.0 / 16777216.0)
            dy = (_mix32((base + 2 * k + 1) & 0xFFFFFFFF) >> 8).to(f32) * (1.0 / 16777216.0)
            nx.append((x.to(f32) + dx) * px - 1.0)
            moment = np.float32(np.float32(k * 5 % jitter) + np.float32(0.5)) / np.float32(jitter) - np.float32(0.5)
        else:
            sy, sx = divmod(k, side)
            dx = np.float32(np.float32(sx) + np.float32(0.5)) / np.float32(side)
            dy = float(np.float32(np.float32(sy) + np.float32(0.5)) / np.float32(side))
            nx.append(((x & 7).to(f32) + ((x & ~7).to(f32) + float(dx))) * px - 1.0)
            moment = np.float32(k * 5 % (side * side) + 0.5) * np.float32(frame.image[3]) - np.float32(0.5)
        ny.append(1.0 - (y.to(f32) + dy) * py)
        t.append(frame.disc[2] + frame.spin[3] * float(moment))
    return torch.stack(nx).double(), torch.stack(ny).double(), t


def _image64(frame, f, m, fluid, jitter, seed, want_ends):
    w, h = int(frame.size[0]), int(frame.size[1])
    nx, ny, t = _positions(frame, jitter, seed)
    total, bits, ends = 0.0, torch.zeros(w * h, dtype=torch.int64, device="cuda"), []
    with torch.no_grad():
        for k in range(len(t)):
            rgb, lit, sky, end = _trace64(f, m, fluid, nx[k], ny[k], t[k])
            total = total + rgb
            bits = bits | lit.long() | (sky.long() * 2) | ((~lit & ~sky).long() * 4)
            ends.append(end)
        image = torch.cat([total / len(t), bits[:, None].double()], 1).reshape(h, w, 4)
    return image, torch.stack(ends, 1).reshape(-1, 6) if want_ends else None


def _turns(y, x):
    ax, ay = x.abs(), y.abs()
    q = torch.minimum(ax, ay) / torch.maximum(ax, ay).clamp(min=_k(1e-20))
    s = q * q
    r = ((_k(-.0464964749) * s + _k(.15931422)) * s - _k(.327622764)) * s * q + q
    r = torch.where(ay > ax, _k(1.57079633) - r, r)
    r = torch.where(x < 0, _k(3.14159265) - r, r)
    return torch.where(y < 0, -r, r) * _k(.15915494)


def _sine(turns):
    t = turns - torch.floor(turns + 0.5)
    t = torch.where(t > 0.25, 0.5 - t, t)
    t = torch.where(t < -0.25, -0.5 - t, t)
    x = t * _k(6.2831853)
    x2 = x * x
    p = x2 * _k(2.7557319e-6) + _k(-1.9841270e-4)
    p = (p * x2 + _k(8.3333333e-3)) * x2 + _k(-.16666667)
    return p * x2 * x + x


def _row(table, at, width, row, turn):
    pos = (turn - torch.floor(turn)) * width
    column = torch.floor(pos.detach())
    c0 = column.long() & (width - 1)
    base = at + row * width
    lo, hi = table[base + c0].double(), table[base + ((c0 + 1) & (width - 1))].double()
    return lo + (hi - lo) * (pos - column)


def _star(d, cells, density, size, gain):
    p = d * cells
    c = torch.floor(p.detach())
    i = c.long() & 0xFFFFFFFF
    m = 0xFFFFFFFF
    h = (i[:, 0] * 73856093 & m) ^ (i[:, 1] * 19349663 & m) ^ (i[:, 2] * 83492791 & m)
    h = ((h ^ (h >> 15)) * 0x2C1B3C6D) & m
    h = ((h ^ (h >> 12)) * 0x297A2D39) & m
    h = h ^ (h >> 15)
    inv = _k(np.float32(1) / np.float32(255))
    at = torch.stack([(h >> 8) & 255, (h >> 16) & 255, (h >> 24) & 255], 1).double() * inv
    e = p - c - at
    light = (1.0 - e.square().sum(1) * _k(np.float32(1) / (np.float32(size) * np.float32(size)))).clamp(min=0.0)
    light = torch.where((h & 255) < density, light * light * _k(gain), torch.zeros_like(light))
    warm = ((h >> 3) & 255).double() * inv
    return torch.stack([light * (0.75 + warm * 0.25), light * _k(.82), light * (1.0 - warm * _k(.45))], 1)


def _trace64(f, m, fluid, nx, ny, time):
    """Rays of image positions (nx, ny) at one moment: their light, whether the disc lit them and they reached
    the sky, and their ends.  The stepper, its step, its ends and the shading are the documented ones."""
    n, dev = nx.numel(), nx.device
    a, inner = f.a, f.inner
    spinning = float(a) != 0.0
    a2 = a * a
    d = [f.forward[k] + nx * f.right[k] + ny * f.up[k] for k in range(3)]
    inv = 1.0 / torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    d = [x * inv for x in d]
    moved = torch.ones_like(nx)
    g = float(f.boost[3])
    if g > 1.0:
        cosine = -(d[0] * f.boost[0] + d[1] * f.boost[1] + d[2] * f.boost[2])
        push, moved = g * (1.0 + g / (g + 1.0) * cosine), 1.0 / (g * (1.0 + cosine))
        d = [(d[k] - f.boost[k] * push) * moved for k in range(3)]
    rho, root_delta, u0, mu0 = f.place[0], f.place[1], f.place[2], f.place[3]
    ie = 1.0 / (f.metric[0] - f.metric[1] * d[2])
    xi, axis, across = -f.metric[2] * d[2] * ie, f.metric[3] * d[2] * ie, rho * d[1] * ie
    eta = across * across + mu0 * mu0 * (axis * axis - a2)
    big = eta + xi * xi
    c = {"ie": ie * moved, "xi": xi, "big": big, "h": _k(.13089969) / torch.sqrt(big.clamp(min=4.0)), "uA": a2 - big,
         "uB": 3.0 * (eta + (xi - a) ** 2), "uC": -2.0 * a2 * eta, "xiA": xi * a}
    one = torch.ones_like(nx)
    s = {"u": u0 * one, "w": -u0 * u0 * root_delta * rho * d[0] * ie, "psi": 0.0 * one, "through": one,
         "n0": f.er[0] * one, "n1": f.er[1] * one, "n2": f.er[2] * one}
    for k in range(3):
        s["v%d" % k] = across * f.etheta[k] + axis * f.ephi[k]

    def drag(x, k):
        return -a * x * (2.0 - k["xiA"] * x) / (1.0 - 2.0 * x + a2 * x * x).clamp(min=_k(1e-3)) if spinning else 0.0 * x

    def bend(x, k):
        return x * (k["uA"] + x * (k["uB"] + x * k["uC"]))

    s["drag"] = drag(s["u"], c)
    at = torch.arange(n, device=dev)
    rgb = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    lit = torch.zeros(n, dtype=torch.bool, device=dev)
    sky = torch.zeros(n, dtype=torch.bool, device=dev)
    end = torch.zeros((n, 6), dtype=torch.float64, device=dev)
    end[:, 0:2] = math.nan
    rho_scale = 1.0 / (1.0 - inner / f.outer)
    third = _k(np.float32(1) / np.float32(6))
    for i in range(192):
        h, h2 = c["h"], c["h"] * c["h"]
        k1 = bend(s["u"], c)
        mid = s["u"] + 0.5 * h * s["w"] + 0.125 * h2 * k1
        k2 = bend(mid, c)
        k3 = bend(s["u"] + h * s["w"] + 0.5 * h2 * k2, c)
        e = {"u": s["u"] + h * s["w"] + third * h2 * (k1 + 2.0 * k2), "w": s["w"] + third * h * (k1 + k3 + 4.0 * k2)}
        e["drag"] = drag(e["u"], c)
        e["psi"] = s["psi"] + third * h * (s["drag"] + e["drag"] + 4.0 * drag(mid, c))
        z = s["n2"]
        c1 = c["big"] + 2.0 * a2 * z * z
        a1 = [-c1 * s["n0"], -c1 * s["n1"], (a2 - c1) * z]
        p = [s["n%d" % k] + 0.5 * h * s["v%d" % k] + 0.125 * h2 * a1[k] for k in range(3)]
        c2 = c["big"] + 2.0 * a2 * p[2] * p[2]
        b2 = [-c2 * p[0], -c2 * p[1], (a2 - c2) * p[2]]
        p = [s["n%d" % k] + h * s["v%d" % k] + 0.5 * h2 * b2[k] for k in range(3)]
        c3 = c["big"] + 2.0 * a2 * p[2] * p[2]
        b3 = [-c3 * p[0], -c3 * p[1], (a2 - c3) * p[2]]
        for k in range(3):
            e["n%d" % k] = s["n%d" % k] + h * s["v%d" % k] + third * h2 * (a1[k] + 2.0 * b2[k])
            e["v%d" % k] = s["v%d" % k] + third * h * (a1[k] + b3[k] + 4.0 * b2[k])
        through = s["through"]
        hit = torch.nonzero(z * e["n2"] < 0).reshape(-1)
        if hit.numel():
            q = {k: x[hit] for k, x in s.items()}
            r = {k: x[hit] for k, x in e.items()}
            o = {k: x[hit] for k, x in c.items()}
            part = q["n2"] / (q["n2"] - r["n2"])
            hu = part * o["h"]
            hh = 0.5 * hu * hu
            uc = q["u"] + hu * q["w"] + hh * k1[hit]
            center = (1.0 - inner * uc) * rho_scale
            ok = torch.nonzero((center > _k(-.03)) & (center < _k(1.02))).reshape(-1)
            if ok.numel():
                sub = hit[ok]
                q, r, o = ({k: x[ok] for k, x in y.items()} for y in (q, r, o))
                b = [x[sub] for x in a1]
                light, clear, turn, uc = _crossing(f, m, fluid, time, rho_scale, q, r, o, part[ok], hu[ok], hh[ok], uc[ok],
                                                   k1[sub], b)
                rgb = torch.index_add(rgb, 0, at[sub], light)
                through = through.index_put((sub,), clear)
                with torch.no_grad():
                    first = (light.sum(1) > 0) & ~lit[at[sub]]
                    who = at[sub][first]
                    lit[who] = True
                    end[who, 0] = 1.0 / uc[first]
                    end[who, 1] = (turn - torch.floor(turn))[first]
        away = e["u"] < 0
        gone = torch.nonzero(away).reshape(-1)
        if gone.numel():
            q = {k: x[gone] for k, x in s.items()}
            r = {k: x[gone] for k, x in e.items()}
            part = q["u"] / (q["u"] - r["u"])
            v = [q["n%d" % k] + part * (r["n%d" % k] - q["n%d" % k]) for k in range(3)]
            inv = 1.0 / torch.sqrt((v[0] * v[0] + v[1] * v[1] + v[2] * v[2]).clamp(min=_k(1e-12)))
            turn = (q["psi"] + part * (r["psi"] - q["psi"])) * _k(.15915494)
            sine, cosine = _sine(turn), _sine(turn + 0.25)
            v = [x * inv for x in v]
            way = torch.stack([v[0] * cosine - v[1] * sine, v[0] * sine + v[1] * cosine, v[2]], 1)
            sky[at[gone]] = True
            with torch.no_grad():
                end[at[gone], 2:5] = way
                end[at[gone], 5] = (i + part) * c["h"][gone]
            if f.stars > 0:
                light = _sky(f, m, way, c["ie"][gone], through[gone])
                rgb = torch.index_add(rgb, 0, at[gone], light)
        over = (e["u"] > f.horizon) | ~(through > _k(.004))
        with torch.no_grad():
            done = torch.nonzero(over & ~away).reshape(-1)
            end[at[done], 5] = (i + 1) * c["h"][done]
        e["through"] = through
        s = e
        if bool((away | over).any()):
            keep = torch.nonzero(~(away | over)).reshape(-1)
            at = at[keep]
            s, c = {k: x[keep] for k, x in s.items()}, {k: x[keep] for k, x in c.items()}
            if not at.numel():
                break
    if at.numel():
        with torch.no_grad():
            end[at, 5] = 192 * c["h"]
    return rgb, lit, sky, end


def _crossing(f, m, fluid, time, rho_scale, q, r, o, part, hu, hh, uc, k1, a1):
    a, inner = f.a, f.inner
    wc = q["w"] + hu * k1
    cx, cy = q["n0"] + hu * q["v0"] + hh * a1[0], q["n1"] + hu * q["v1"] + hh * a1[1]
    vx, vy, vz = q["v0"] + hu * a1[0], q["v1"] + hu * a1[1], q["v2"] + hu * a1[2]
    psi, dragged = q["psi"] + part * (r["psi"] - q["psi"]), q["drag"] + part * (r["drag"] - q["drag"])
    turn = _turns(cy, cx) + psi * _k(.15915494)
    rate = ((cx * vy - cy * vx) / (cx * cx + cy * cy).clamp(min=_k(1e-6)) + dragged) * _k(.15915494)
    slope = wc / uc
    mu = (vz.abs() / torch.sqrt(vx * vx + vy * vy + vz * vz + slope * slope)).clamp(min=_k(.02))
    slant = f.thickness / 3.0 / mu
    reach = torch.minimum(f.height / vz.abs().clamp(min=_k(1e-5)), o["h"] * 1.5)
    top = capi.MAP_HEIGHT - 1

    def speed(row):
        if f.q is None:
            return m[capi.ROWS_AT + 2 * row].double()
        rad = inner / (1.0 - row.double() / top * (1.0 - inner / f.outer))
        return 1.0 / (_k(6.2831853) * (rad * torch.sqrt(rad) + a))

    glow, clear = 0.0, q["through"]
    for k in range(3):
        t = float(np.float32(np.float32(np.float32(k) + np.float32(.5)) * np.float32(np.float32(2) / np.float32(3))) - np.float32(1))
        ds = reach * t
        rho = (1.0 - inner * (uc + wc * ds)) * rho_scale
        inside = (rho > 0) & (rho < 1)
        rho = torch.where(inside, rho, torch.zeros_like(rho))
        pos = rho * top
        row = torch.floor(pos.detach()).clamp(max=top - 1)
        r0 = row.long()
        s0, s1 = speed(r0), speed(r0 + 1)
        tk = turn + torch.where(inside, rate * ds, torch.zeros_like(ds))
        d0, d1 = _row(m, 0, capi.MAP_WIDTH, r0, tk - s0 * time), _row(m, 0, capi.MAP_WIDTH, r0 + 1, tk - s1 * time)
        density = d0 + (d1 - d0) * (pos - row)
        fpos = rho * (capi.FLUID_HEIGHT - 1)
        frow = torch.floor(fpos.detach()).clamp(max=capi.FLUID_HEIGHT - 2)
        ft = tk - s0 * (time - f.flow[0])
        g0, g1 = _row(fluid, 0, capi.FLUID_WIDTH, frow.long(), ft), _row(fluid, 0, capi.FLUID_WIDTH, frow.long() + 1, ft)
        density = density * (_k(np.float32(1) - np.float32(.1)) + _k(.1) * (g0 + (g1 - g0) * (fpos - frow)))
        drow = torch.floor((rho * (capi.DUST_HEIGHT - 1)).detach()).clamp(max=capi.DUST_HEIGHT - 1).long()
        dusty = _row(m, capi.DUST_AT, capi.DUST_WIDTH, drow, tk - s0 * time)
        height = t * (reach / f.height)
        level = (1.0 - vz * vz * (height * height)).clamp(min=0.0)
        density = torch.where(inside, density * level, torch.zeros_like(density))
        depth = slant * density * (1.0 + 25.0 * dusty)
        alpha = depth / (1.0 + depth)
        glow = glow + clear * alpha * (density * (1.0 - _k(.97) * dusty))
        clear = clear * (1.0 - alpha)
    center = ((1.0 - inner * uc) * rho_scale).detach().clamp(min=0.0, max=1.0)
    ring = (center * top).long()
    heat = m[capi.ROWS_AT + 2 * ring + 1].double()
    if f.q is None:
        gives = m[capi.GLOW_AT + ring].double()
    else:
        gives = torch.exp(f.q * torch.log(1.0 - ring.double() / top * (1.0 - inner / f.outer)))
    light = f.gain * glow * gives
    if f.doppler != 0:
        safe = uc.clamp(min=_k(1e-4))
        root = safe * torch.sqrt(safe)
        lift = 1.0 + a * root
        beneath = (1.0 - 3.0 * safe + 2.0 * a * root).clamp(min=_k(1e-4))
        shift = torch.sqrt(beneath) * o["ie"] / (lift * (1.0 - root / lift * o["xi"]))
        shift = 1.0 + f.doppler * (shift - 1.0)
        light = light * shift ** 4
        heat = heat * shift
    color = (heat.detach() * (capi.COLORS // 2)).clamp(max=capi.COLORS - 1).long()
    rgb = torch.stack([m[capi.COLORS_AT + 3 * color + j].double() for j in range(3)], 1)
    return light[:, None] * rgb, clear, turn.detach(), uc.detach()


def _sky(f, m, way, ie, through):
    rgb = _star(way, 90.0, 26, .1, 1.6) + _star(way, 240.0, 70, .17, .22)
    turn = _turns(way[:, 1], way[:, 0])
    pos = (way[:, 2] * 0.5 + 0.5) * (capi.SKY_HEIGHT - 1)
    row = torch.floor(pos.detach()).clamp(max=capi.SKY_HEIGHT - 2)
    s0, s1 = (_row(m, capi.SKY_AT, capi.SKY_WIDTH, row.long() + k, turn) for k in (0, 1))
    dust = s0 + (s1 - s0) * (pos - row)
    rgb = rgb + dust[:, None] * torch.tensor([_k(.92), _k(.86), 1.0], dtype=torch.float64, device=way.device)
    shown = through * f.stars
    if f.doppler != 0:
        shown = shown * (1.0 + f.doppler * (ie - 1.0)) ** 4
    return rgb * shown[:, None]
