"""Performance cases: the renders that a user of this framework asks for, over the sizes they are asked for at.

A case is a dict of plain values; ``prepare`` makes its scene from a seed with the generators of
``forgedthoughts_gb300.workloads``, ``run`` is one call of the public entry points, ``work`` the bytes and operations
that it cannot do without, and ``exact`` the same result from a plain 64-bit torch restatement of the march.

Kinds:

* ``preview``: ``ft.render_depth`` with host outputs, spheres on a ground: what an editor asks for on each change.
* ``depth``:   ``ft_render_depth`` with device outputs, a union_round field: a full-size depth frame, plain or through
  the FP16 brick cache.
* ``trace``:   a Whitted frame of a union_round field, device outputs (``device``) or host ones.
* ``path``:    ``ft.render_pathtrace``: the progressive path tracer.
* ``shells``:  depth of spheres that carry ``domain`` and ``distance_post`` hooks, interpreted or compiled (``jit``).
* ``batch``:   many scenes of uneven size in one ``ft.Batch`` launch, each read back.
* ``fit``:     one step of inverse shape fitting: new parameters, depth and silhouette of all views, the loss and
  its gradient.
* ``open``:    a scene's source to its preview: parse, lower, build, upload, render (``ftc depth``).
"""
from __future__ import annotations

import ctypes
import dataclasses
import math
import re

import numpy as np
import torch

import forgedthoughts_gb300 as ft
from forgedthoughts_gb300 import _native, workloads

TAU = 0.05


def listed():
    return [
        # the smallest preview: a thumbnail, where the call itself counts
        {"name": "preview_thumb", "kind": "preview", "n": 8, "width": 64, "height": 64, "aa": 1},
        # the plain depth preview of the benchmark configurations: 256 x 256, 8 spheres
        {"name": "preview_256", "kind": "preview", "n": 8, "width": 256, "height": 256, "aa": 1},
        # a scene of many hard-unioned objects at an odd size
        {"name": "preview_objects", "kind": "preview", "n": 700, "width": 613, "height": 347, "aa": 4},
        # a full-size depth frame of the 512-primitive blended field, 2 x 2 samples
        {"name": "depth_field", "kind": "depth", "n": 512, "width": 1920, "height": 1080, "aa": 4, "bricks": False},
        # the precision form of a depth frame: marching through the FP16 brick cache
        {"name": "depth_bricks", "kind": "depth", "n": 512, "width": 1280, "height": 720, "aa": 1, "bricks": True},
        # the headline frame: Whitted trace of the field, depth 6
        {"name": "trace_field", "kind": "trace", "n": 512, "width": 1920, "height": 1080, "aa": 4, "depth": 6,
         "jitter": False, "device": True},
        # a small jittered trace into host memory: a preview while editing
        {"name": "trace_small", "kind": "trace", "n": 96, "width": 353, "height": 199, "aa": 1, "depth": 3,
         "jitter": True, "device": False},
        # the path tracer at its default settings
        {"name": "path_16spp", "kind": "path", "n": 96, "width": 320, "height": 180, "spp": 16, "bounces": 4},
        # hooked objects with the scene compiled at run time
        {"name": "shells_jit", "kind": "shells", "n": 512, "width": 640, "height": 360, "jit": True},
        # many scenes in one launch: half depth previews, half Whitted
        {"name": "batch_20", "kind": "batch", "n": 20, "most": 2048},
        # an optimisation step: 64 primitives, 449 parameters, a ring of views
        {"name": "fit_step", "kind": "fit", "n": 64, "views": 32, "size": 256},
        # opening a scene: source text to its preview
        {"name": "open_scene", "kind": "open", "n": 512, "width": 800, "height": 600},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["preview", "preview", "depth", "depth", "trace", "trace", "path", "shells", "batch", "fit",
                       "open"])
    if kind == "preview":
        return {"kind": kind, "n": _log_int(rng, 1, 1024), "width": _log_int(rng, 33, 1024),
                "height": _log_int(rng, 33, 768), "aa": rng.choice([1, 1, 4])}
    if kind == "depth":
        return {"kind": kind, "n": _log_int(rng, 8, 768), "width": _log_int(rng, 160, 1920),
                "height": _log_int(rng, 90, 1080), "aa": rng.choice([1, 4]), "bricks": rng.random() < 0.3}
    if kind == "trace":
        return {"kind": kind, "n": _log_int(rng, 8, 512), "width": _log_int(rng, 100, 1280),
                "height": _log_int(rng, 90, 720), "aa": rng.choice([1, 2, 4]), "depth": rng.randint(1, 6),
                "jitter": rng.random() < 0.5, "device": rng.random() < 0.5}
    if kind == "path":
        return {"kind": kind, "n": _log_int(rng, 8, 256), "width": _log_int(rng, 64, 320),
                "height": _log_int(rng, 64, 240), "spp": rng.choice([8, 16, 24]), "bounces": rng.choice([3, 4, 5])}
    if kind == "shells":
        return {"kind": kind, "n": _log_int(rng, 8, 512), "width": _log_int(rng, 100, 480),
                "height": _log_int(rng, 80, 300), "jit": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "n": rng.randint(3, 20), "most": _log_int(rng, 64, 2048)}
    if kind == "fit":
        return {"kind": kind, "n": _log_int(rng, 8, 96), "views": rng.randint(1, 40), "size": _log_int(rng, 40, 256)}
    return {"kind": "open", "n": _log_int(rng, 8, 600), "width": _log_int(rng, 100, 1024),
            "height": _log_int(rng, 90, 768)}


# ---------------------------------------------------------------- inputs
def _workload(case, seed):
    kind = case["kind"]
    if kind == "preview":
        return workloads.spheres_on_ground(case["n"], seed, case["width"], case["height"])
    if kind in ("depth", "trace", "path", "open"):
        return workloads.union_round_field(case["n"], seed, case["width"], case["height"], case.get("aa", 1))
    if kind == "shells":
        return workloads.twisted_shells(case["n"], seed, case["width"], case["height"])
    raise ValueError(kind)


def _batch_workloads(case, seed):
    """Scenes drawn as ``workloads.batch_scenes`` draws them, of at most ``most`` spheres; their sizes and modes (depth
    preview or Whitted of depth 2) take turns, so that each seed asks for the same images of other scenes."""
    out, first = [], 1000 * (seed % 100000)
    while len(out) < case["n"]:
        w = workloads.batch_scenes(1, first)[0]
        first += 1
        if w.source.count("Sphere") <= case["most"]:
            size = (64, 128, 256, 512)[len(out) % 4]
            out.append(dataclasses.replace(w, options=dataclasses.replace(w.options, width=size, height=size),
                                           max_depth=2 * (len(out) // 4 % 2)))
    return out


def _fit_inputs(case, seed):
    theta_rng = np.random.default_rng(seed + 1)
    src = workloads.shape_fit(case["n"], seed)
    return src, workloads.shape_fit_options(case["size"]), ft.ring_views(case["views"]), theta_rng


class _Fit:
    """Shape fitting against target images, all on the device."""

    def __init__(self, case, seed):
        src, self.opts, self.views, rng = _fit_inputs(case, seed)
        self.scene = ft.ParamScene(src)
        self.theta = self.scene.get_params()
        shape = (case["views"], case["size"], case["size"])
        new = lambda dt: torch.empty(shape, dtype=dt, device="cuda")  # noqa: E731
        self.t, self.mask, self.sil = new(torch.float32), new(torch.uint8), new(torch.float32)
        self.grad = torch.zeros(self.theta.size, dtype=torch.float64, device="cuda")
        self.cviews, self.copts = ft.views_c(self.views), self.opts.to_c()
        target = (self.theta + rng.normal(0.0, 0.05, self.theta.shape)).astype(np.float32)
        self.scene.set_params(target)
        self.render()
        self.t0, self.mask0, self.sil0 = self.t.clone(), self.mask.clone(), self.sil.clone()

    def render(self):
        s = torch.cuda.current_stream().cuda_stream
        _ok(_native.lib().ft_render_views(self.scene.state.gpu().handle, self.cviews, len(self.views),
                                          ctypes.byref(self.copts), TAU, _p(self.t), _p(self.mask), _p(self.sil),
                                          _native.FT_FLAG_DEVICE_POINTERS, ctypes.c_void_p(s)))

    def step(self):
        self.scene.set_params(self.theta)
        self.render()
        both = (self.mask != 0) & (self.mask0 != 0)
        dt = torch.where(both, self.t - self.t0, torch.zeros_like(self.t))
        ds = self.sil - self.sil0
        loss = dt.square().sum(dtype=torch.float64) + ds.square().sum(dtype=torch.float64)
        gt, gs = 2.0 * dt, 2.0 * ds
        s = torch.cuda.current_stream().cuda_stream
        _ok(_native.lib().ft_render_backward(self.scene.state.gpu().handle, self.cviews, len(self.views),
                                             ctypes.byref(self.copts), TAU, self.scene.layout, self.scene.n_params,
                                             _p(gt), _p(gs), _p(self.grad), _native.FT_FLAG_DEVICE_POINTERS,
                                             ctypes.c_void_p(s)))
        return {"t": self.t, "mask": self.mask, "sil": self.sil, "loss": loss.float(), "grad": self.grad.float()}


def _p(x):
    return ctypes.c_void_p(x.data_ptr())


def _ok(rc):
    if rc != 0:
        raise RuntimeError(_native.last_error())


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": dict(case)}
    if kind == "open":
        state["workload"] = _workload(case, seed)
        return state
    if kind == "batch":
        ws = _batch_workloads(case, seed)
        state["depths"] = [w.max_depth for w in ws]
        state["batch"] = ft.Batch([(ft.parse_and_eval(w.source), w.options, w.aa, w.max_depth) for w in ws])
        return state
    if kind == "fit":
        state["fit"] = _Fit(case, seed)
        return state
    w = _workload(case, seed)
    scene = ft.parse_and_eval(w.source)
    scene.gpu()
    state.update(workload=w, scene=scene, seed=seed & 0xFFFF)
    if case.get("jit"):
        scene.gpu().jit()
    if case.get("bricks"):
        scene.gpu().build_bricks()
    if kind == "depth" or case.get("device"):
        px = case["width"] * case["height"]
        items = px * case["aa"]
        new = lambda n, dt: torch.empty(n, dtype=dt, device="cuda")  # noqa: E731
        if kind == "depth":
            state["out"] = {"t": new(items, torch.float32), "mask": new(items, torch.uint8),
                            "material": new(items, torch.int32), "normal": new(items * 3, torch.float32),
                            "rgb8": new(px * 3, torch.uint8)}
        else:
            state["out"] = {"rgb": new(px * 3, torch.float32), "rgb8": new(px * 3, torch.uint8)}
        state["options"] = w.options.to_c()
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "open":
        w = state["workload"]
        scene = ft.parse_and_eval(w.source)
        img = ft.render_depth(scene, w.options, w.accel, 1, want_t=False, want_mask=False)
        scene.close()
        return {"rgb8": img.rgb8}
    if kind == "batch":
        b = state["batch"]
        b.launch(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        got = [b.read(i) for i in range(case["n"])]
        return [[r["t"], r["mask"], r["rgb8"]] if d == 0 else [r["rgb"], r["rgb8"]]
                for r, d in zip(got, state["depths"])]
    if kind == "fit":
        return state["fit"].step()
    w, scene = state["workload"], state["scene"]
    if kind in ("preview", "shells"):
        img = ft.render_depth(scene, w.options, w.accel, case.get("aa", 1), want_material=True, want_normal=True)
        return {"t": img.t, "mask": img.mask, "material": img.material, "normal": img.normal, "rgb8": img.rgb8}
    if kind == "path":
        rgb, rgb8, count = ft.render_pathtrace(scene, w.options, w.accel,
                                               ft.PathtraceSettings(spp=case["spp"], max_bounces=case["bounces"]))
        return {"rgb": rgb, "rgb8": rgb8, "count": count}
    if kind == "trace" and not case["device"]:
        rgb, rgb8 = ft.render_trace(scene, w.options, w.accel, case["aa"], case["depth"],
                                    jitter_seed=state["seed"] if case["jitter"] else None)
        return {"rgb": rgb, "rgb8": rgb8}
    lib, out = _native.lib(), state["out"]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    flags = _native.FT_FLAG_DEVICE_POINTERS
    if kind == "trace":
        flags |= ft.jitter_flags(state["seed"] if case["jitter"] else None)
        _ok(lib.ft_render_trace(scene.gpu().handle, ctypes.byref(state["options"]), int(w.accel), case["aa"],
                                case["depth"], _p(out["rgb"]), _p(out["rgb8"]), flags, stream))
        return out
    if case["bricks"]:
        flags |= _native.FT_FLAG_FP16_BRICKS
    _ok(lib.ft_render_depth(scene.gpu().handle, ctypes.byref(state["options"]), int(w.accel), case["aa"],
                            _p(out["t"]), _p(out["mask"]), _p(out["material"]), _p(out["normal"]), _p(out["rgb8"]),
                            flags, stream))
    return out


# ---------------------------------------------------------------- the work of a pass
# One distance evaluation needs at least the nearest primitive and the ground: about 24 operations each (the point in
# the primitive's frame, its distance, the minimum).  A ray that hits marches some 25 samples, bisects 10 times, takes
# 6 normal taps and looks its material up; a shadow ray marches some 10.
_EVAL = 48.0
_HIT = 25 + 10 + 6 + 1
_SHADOW = 10


def work(case):
    kind = case["kind"]
    if kind == "batch":
        px = float(sum((64, 128, 256, 512)[i % 4] ** 2 for i in range(case["n"])))
        return {"bytes": px * 15, "flops": px * 1.5 * _HIT * _EVAL}
    if kind == "fit":
        # the forward march, a 40-step minimum search for the rays that miss, the march again for the adjoint
        rays = case["views"] * case["size"] ** 2
        return {"bytes": rays * 17.0, "flops": rays * 2 * _HIT * _EVAL}
    px = float(case["width"] * case["height"])
    if kind == "open":
        return {"bytes": px * 3 + 200.0 * case["n"], "flops": px * (_HIT - 6) * _EVAL}
    if kind == "path":
        # each sample: a path of about two bounces, a shadow ray at each
        return {"bytes": px * 19, "flops": px * case["spp"] * 2 * (_HIT + _SHADOW) * _EVAL}
    items = px * case.get("aa", 1)
    if kind == "trace":
        # half of the samples reflect or refract once more at each level
        levels = sum(0.5 ** k for k in range(case["depth"]))
        return {"bytes": px * 15, "flops": items * levels * (_HIT + _SHADOW) * _EVAL}
    per = 21 * items + 3 * px
    return {"bytes": per, "flops": items * _HIT * _EVAL * (2 if kind == "shells" else 1)}


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    kind = case["kind"]
    if kind == "preview" and case["width"] * case["height"] * case["aa"] * case["n"] < 1 << 30:
        m = _March(_parse(_workload(case, seed).source), case["width"], case["height"], case["aa"])
        t, mask, normal = m.depth()
        shape = (case["height"], case["width"], case["aa"])
        return {"t": t.reshape(shape), "mask": None, "material": None, "normal": normal.reshape(*shape, 3),
                "rgb8": None}
    if kind == "depth" and case["width"] * case["height"] * case["aa"] * case["n"] < 1 << 28:
        m = _March(_parse(_workload(case, seed).source), case["width"], case["height"], case["aa"])
        t, mask, normal = m.depth()
        return {"t": t.reshape(-1), "mask": None, "material": None, "normal": normal.reshape(-1), "rgb8": None}
    if kind == "batch" and case["n"] * case["most"] < 1 << 11:
        out = []
        for w in _batch_workloads(case, seed):
            if w.max_depth:
                out.append([None, None])
                continue
            o = w.options
            t, _, _ = _March(_parse(w.source), o.width, o.height, 1).depth(normals=False)
            out.append([t.reshape(o.height, o.width, 1), None, None])
        return out
    if kind == "fit" and case["views"] * case["size"] ** 2 * case["n"] < 1 << 28:
        return _exact_fit(case, seed)
    return None  # whole integrators, hook programs, and frames that take too long in 64 bits


_NUM = r"(-?[0-9.]+)"
_VEC = r"vec3\(" + _NUM + ", " + _NUM + ", " + _NUM + r"\)"


def _parse(src):
    """Primitives (and how they combine) of a generated scene's source."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    c, rot, size, box = [], [], [], []
    for line in src.splitlines():
        m = re.match(r"let \w+ = (Sphere|Box) \{ (?:radius: " + _NUM + "|size: " + _VEC + "), pos: " + _VEC +
                     r"(?:, rot: " + _VEC + ")?", line)
        if not m:
            continue
        g = [float(np.float32(x)) if x is not None and k else x for k, x in enumerate(m.groups())]
        box.append(g[0] == "Box")
        size.append([0.5 * g[2], 0.5 * g[3], 0.5 * g[4]] if g[0] == "Box" else [g[1]] * 3)
        c.append(g[5:8])
        rot.append(g[9] if g[9] is not None else 0.0)
    cam = re.search(r"Camera \{ origin: " + _VEC + ", target: " + _VEC + ", fov_y: " + _NUM, src)
    k = re.search(r"union_round\(\w+, " + _NUM, src)
    f64 = lambda x: torch.tensor(x, dtype=torch.float64, device=dev)  # noqa: E731
    return {"c": f64(c).reshape(-1, 3), "rot": f64(rot), "size": f64(size).reshape(-1, 3),
            "box": torch.tensor(box, device=dev), "ground": "var ground" in src,
            "r": f64(float(np.float32(k.group(1)))) if k else None,
            "camera": [float(np.float32(x)) for x in cam.groups()] if cam else None, "dev": dev}


def _field(s, p):
    """Distances of points (N, 3) in 64 bits."""
    out = torch.empty(p.shape[0], dtype=torch.float64, device=p.device)
    if not p.shape[0]:
        return out
    n = max(1, s["c"].shape[0])
    if p.requires_grad or s["c"].requires_grad:
        return _field_part(s, p)
    for i in range(0, p.shape[0], max(1, (1 << 25) // n)):
        out[i:i + max(1, (1 << 25) // n)] = _field_part(s, p[i:i + max(1, (1 << 25) // n)])
    return out


def _field_part(s, p):
    d = None
    if s["c"].shape[0]:
        q = p[:, None, :] - s["c"]
        a = torch.deg2rad(-s["rot"])
        ca, sa = torch.cos(a), torch.sin(a)
        x, y, z = ca * q[..., 0] + sa * q[..., 2], q[..., 1], -sa * q[..., 0] + ca * q[..., 2]
        e = torch.stack([x.abs(), y.abs(), z.abs()], -1) - s["size"]
        outside = e.clamp(min=0.0).square().sum(-1)
        outside = torch.where(outside > 0, outside, torch.ones_like(outside)).sqrt() * (outside > 0)
        boxd = outside + e.amax(-1).clamp(max=0.0)
        v = torch.where(s["box"], boxd, (x * x + y * y + z * z).sqrt() - s["size"][:, 0])
        if s["r"] is None:
            d = v.amin(1)
        else:  # the balanced pairwise tree of the generators
            r = s["r"]
            while v.shape[1] > 1:
                m = v.shape[1] // 2 * 2
                u, w = v[:, 0:m:2], v[:, 1:m:2]
                l2 = (r - u).clamp(min=0.0).square() + (r - w).clamp(min=0.0).square()
                l = torch.where(l2 > 0, l2, torch.ones_like(l2)).sqrt() * (l2 > 0)
                v = torch.cat([torch.maximum(r.expand_as(u), torch.minimum(u, w)) - l, v[:, m:]], 1)
            d = v[:, 0]
    if s["ground"]:
        e = (p - p.new_tensor([0.0, -0.5, 0.0])).abs() - p.new_tensor([110.0, 0.5, 110.0])
        g = e.clamp(min=0.0).square().sum(1).sqrt() + e.amax(1).clamp(max=0.0)
        d = g if d is None else torch.minimum(d, g)
    return d


class _March:
    """raymarch_hit with the options of the generated workloads (256 steps, epsilon 1e-4, distance 100, scale 0.7)."""

    eps, scale, far, steps = float(np.float32(1e-4)), float(np.float32(0.7)), 100.0, 256

    def __init__(self, s, width, height, aa, camera=None):
        self.s = s
        v = lambda x: torch.tensor(x, dtype=torch.float64, device=s["dev"])  # noqa: E731
        cam = camera or s["camera"]
        o, tgt, fov = v(cam[0:3]), v(cam[3:6]), cam[6]
        fwd = torch.nn.functional.normalize(tgt - o, dim=0)
        right = torch.nn.functional.normalize(torch.linalg.cross(fwd, v([0.0, 1.0, 0.0])), dim=0)
        up = torch.linalg.cross(right, fwd)
        grid = int(math.ceil(math.sqrt(aa)))
        sub = torch.arange(aa, device=s["dev"])
        sx, sy = ((sub % grid) + 0.5) / grid, ((sub // grid) + 0.5) / grid
        px, py = torch.arange(width, device=s["dev"]).double(), torch.arange(height, device=s["dev"]).double()
        nx = ((px[None, :, None] + sx) / width * 2.0 - 1.0) * (width / height)
        ny = 1.0 - (py[:, None, None] + sy) / height * 2.0
        nx, ny = torch.broadcast_tensors(nx, ny)
        k = math.tan(math.radians(fov) * 0.5)
        d = fwd + right * (nx.reshape(-1, 1) * k) + up * (ny.reshape(-1, 1) * k)
        self.d = d / d.norm(dim=1, keepdim=True)
        self.o = o
        half = torch.where(s["box"][:, None], s["size"].norm(dim=1, keepdim=True).expand(-1, 3), s["size"])
        mn, mx = (s["c"] - half), (s["c"] + half)
        if s["ground"]:
            h = v([110.0, 0.5, 110.0]).norm()
            g = v([0.0, -0.5, 0.0])
            mn, mx = torch.cat([mn, (g - h)[None]]), torch.cat([mx, (g + h)[None]])
        t0, t1 = (mn.amin(0) - o) / self.d, (mx.amax(0) - o) / self.d
        lo, hi = torch.minimum(t0, t1).amax(1), torch.maximum(t0, t1).amin(1)
        self.inside = hi >= lo
        self.start = lo.clamp(min=0.0)
        self.max_t = hi.clamp(max=self.far)

    def f(self, at, t):
        return _field(self.s, self.o + self.d[at] * t[:, None])

    def step_of(self, f):
        return (f.abs() * self.scale).clamp(min=max(0.5 * self.eps, 1e-5))

    def march(self):
        """hit, bracket (lo, hi), and the smallest sample with its neighbours."""
        n, dev = self.d.shape[0], self.d.device
        hit = torch.zeros(n, dtype=torch.bool, device=dev)
        t, prev = self.start.clone(), self.start.clone()
        best = torch.full((n,), math.inf, dtype=torch.float64, device=dev)
        tp, tb, tn = t.clone(), t.clone(), t.clone()
        need = torch.zeros_like(hit)
        live = torch.nonzero(self.inside).flatten()
        for _ in range(self.steps):
            live = live[t[live] <= self.max_t[live]]
            if not live.numel():
                break
            f = self.f(live, t[live])
            later = live[need[live]]
            tn[later] = t[later]
            need[live] = False
            low = f < best[live]
            at = live[low]
            best[at], tp[at], tb[at], tn[at], need[at] = f[low], prev[at], t[at], t[at], True
            done = f.abs() < self.eps
            hit[live[done]] = True
            live, f = live[~done], f[~done]
            prev[live] = t[live]
            t[live] += self.step_of(f)
        lo, hi = prev.clone(), t.clone()
        at = torch.nonzero(hit).flatten()
        for _ in range(10):
            mid = 0.5 * (lo[at] + hi[at])
            under = self.f(at, mid).abs() < self.eps
            hi[at] = torch.where(under, mid, hi[at])
            lo[at] = torch.where(under, lo[at], mid)
        return hit, lo, hi, best, tp, tb, tn, need

    def depth(self, normals=True):
        hit, _, hi = self.march()[:3]
        t = torch.where(hit, hi, torch.zeros_like(hi))
        normal = torch.zeros_like(self.d)
        if normals:
            at = torch.nonzero(hit).flatten()
            pos, e = self.o + self.d[at] * hi[at][:, None], 4.0 * self.eps
            g = torch.stack([_field(self.s, pos + e * a) - _field(self.s, pos - e * a)
                             for a in torch.eye(3, dtype=torch.float64, device=pos.device)], 1)
            normal[at] = torch.nn.functional.normalize(g, dim=1)
        return t, hit, normal

    def view(self):
        """Depth (the zero of f), silhouette, and the points that carry the gradient: the hit or the ray's minimum."""
        hit, lo, hi, best, tp, tb, tn, need = self.march()
        at = torch.nonzero(hit).flatten()
        a, b = lo[at], hi[at]
        fa, fb = self.f(at, a), self.f(at, b)
        for _ in range(3):
            same = fa == fb
            new = torch.where(same, b, b - fb * (b - a) / torch.where(same, torch.ones_like(fa), fb - fa))
            a, fa, b = torch.where(same, a, b), torch.where(same, fa, fb), new
            fb = self.f(at, b)
        where = torch.where(hit, hi, torch.zeros_like(hi))
        where[at] = b
        value = torch.full_like(where, math.inf)
        at = torch.nonzero(~hit & torch.isfinite(best)).flatten()
        a, x, fx = tp[at], tb[at], best[at]
        b = torch.where(need[at], x + self.step_of(fx), tn[at])
        fb = self.f(at, b)
        for _ in range(64):
            go = (fb < fx) & (b < self.far)
            if not go.any():
                break
            a, x, fx = torch.where(go, x, a), torch.where(go, b, x), torch.where(go, fb, fx)
            b = torch.where(go, x + self.step_of(fx), b)
            fb = self.f(at, b)
        a = torch.where(a < x, a, (x - self.step_of(fx)).clamp(min=0.0))
        fa = self.f(at, a)
        for _ in range(64):
            go = (fa < fx) & (a > 0.0)
            if not go.any():
                break
            b, x, fx = torch.where(go, x, b), torch.where(go, a, x), torch.where(go, fa, fx)
            a = torch.where(go, (x - self.step_of(fx)).clamp(min=0.0), a)
            fa = self.f(at, a)
        for _ in range(60):
            right = b - x > x - a
            u = torch.where(right, x + 0.3819660112501051 * (b - x), x - 0.3819660112501051 * (x - a))
            fu = self.f(at, u)
            low = fu < fx
            a = torch.where(low & (u > x), x, torch.where(~low & ~(u > x), u, a))
            b = torch.where(low & ~(u > x), x, torch.where(~low & (u > x), u, b))
            x, fx = torch.where(low, u, x), torch.where(low, fu, fx)
        where[at], value[at] = x, fx
        sil = torch.exp(-value.clamp(min=0.0) / TAU)
        sil[hit] = 1.0
        return hit, where, sil, value


def _exact_fit(case, seed):
    src, opts, views, rng = _fit_inputs(case, seed)
    s = _parse(src)
    n = s["c"].shape[0]
    # the parameters: per primitive its centre, turn about y and three sizes (a sphere: its radius in the first), then
    # the blend radius
    theta = torch.cat([s["c"], s["rot"][:, None], s["size"]], 1)
    flat = torch.cat([torch.where(s["box"][:, None] | (torch.arange(7, device=theta.device) < 5), theta, 0.0 * theta)
                      .reshape(-1), s["r"].reshape(1)])
    target = (flat.cpu().numpy().astype(np.float32) + rng.normal(0.0, 0.05, flat.numel())).astype(np.float32)

    def scene(v):
        q = v[:-1].reshape(n, 7)
        return dict(s, c=q[:, 0:3], rot=q[:, 3], size=q[:, 4:7], r=v[-1])

    def sphere_sizes(q):  # the bounds of a sphere are its radius on every axis
        return dict(q, size=torch.where(q["box"][:, None], q["size"], q["size"][:, 0:1]))

    a = sphere_sizes(scene(flat))
    b = sphere_sizes(scene(torch.tensor(target, dtype=torch.float64, device=flat.device)))
    out_t, out_s, loss, grad = [], [], 0.0, torch.zeros_like(flat)
    for o, tgt, fov in views:
        cam = [float(np.float32(x)) for x in (*o, *tgt, fov)]
        m = _March(a, opts.width, opts.height, 1, cam)
        hit, at, sil, value = m.view()
        hit0, at0, sil0, _ = _March(b, opts.width, opts.height, 1, cam).view()
        dt = torch.where(hit & hit0, at - at0, torch.zeros_like(at))
        ds = sil - sil0
        loss += float(dt.square().sum() + ds.square().sum())
        out_t.append(torch.where(hit, at, torch.zeros_like(at)))
        out_s.append(sil)
        p = m.o + m.d * at[:, None]
        for rays in (torch.nonzero(hit & (dt != 0)).flatten(),
                     torch.nonzero(~hit & (ds != 0) & (value > 0) & torch.isfinite(value)).flatten()):
            for i in range(0, rays.numel(), 1 << 14):
                k = rays[i:i + (1 << 14)]
                q, v = p[k].clone().requires_grad_(True), flat.clone().requires_grad_(True)
                f = _field_part(scene(v), q)
                slope = (torch.autograd.grad(f.sum(), q, retain_graph=True)[0] * m.d[k]).sum(1)
                w = torch.where(hit[k], -2.0 * dt[k] / torch.where(hit[k], slope, torch.ones_like(slope)),
                                -2.0 * ds[k] * sil[k] / TAU)
                grad += torch.autograd.grad((f * w).sum(), v)[0]
    shape = (case["views"], case["size"], case["size"])
    return {"t": torch.stack(out_t).reshape(shape).cpu(), "mask": None, "sil": torch.stack(out_s).reshape(shape).cpu(),
            "loss": loss, "grad": grad.cpu()}
