"""The work that a user of this library has it do, as cases that can be timed.

Every case goes through the public Python entry points (``Renderer``, ``UploadedScene``,
``Batch``, ``dvg.torch_ops``).  Scenes come from ``dvg.synth``, the seeded generator of the
benchmark and the tests, at the benchmark's sizes and at odd ones between them:

* a *render* is one frame of an uploaded scene into a device image;
* a *step* is one optimisation step's device work: render, L2 loss against a target and
  the gradients of every scene parameter (the target is the render of another scene);
* a *batch* is the same step for many scenes in one CUDA-graph replay;
* a *host* pass is the crate-shaped pair ``render`` / ``render_backward`` on host arrays;
* an *sdf* pass is the signed-distance image;
* an *autograd* pass is forward and backward of the torch function.

``exact`` gives images, losses and distances in 64-bit floating point from the definitions
(polynomial curves, winding numbers, closest points, filter-weighted averages), without this
library's code.  Gradients have no such value here: their geometry part is an estimate over
sampled edge points, or the crate's own (documented) adjoint formulas.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "diffvg-rs_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from dvg import BackwardOptions, Batch, DeviceGrads, Renderer, RenderOptions, device_view, pack_scene, synth  # noqa: E402
from dvg import torch_ops  # noqa: E402
from dvg.scene import (Circle, Color, Ellipse, FillRule, FilterType, GradientStop, LinearGradient, Mat3,  # noqa: E402
                       PathGeometry, RadialGradient)


def _case(kind, scene, width, height, count, spp_x, spp_y, prefilter=False, boundary=0, scenes=1):
    """count: paths of a plain / large / styled scene, or the shapes of a mixed one; boundary: edge
    samples of a gradient pass (0: the crate's width*height*spp); scenes: scenes of a batch."""
    return {"kind": kind, "scene": scene, "width": width, "height": height, "count": count, "spp_x": spp_x,
            "spp_y": spp_y, "prefilter": prefilter, "boundary": boundary, "scenes": scenes}


def listed():
    def named(name, *a, **k):
        return {"name": name, **_case(*a, **k)}

    return [
        # one small icon drawn on its own: launch latency counts as much as the pixels
        named("icon_render", "render", "plain", 64, 64, 10, 2, 2),
        # a frame with more shapes on a canvas that fills neither tiles nor warps evenly, 3x3 samples
        named("mixed_render_odd", "render", "mixed", 613, 347, 208, 3, 3),
        # a large illustration: 4096 paths of 16 segments, a quarter of them stroked
        named("large_render", "render", "large", 1024, 1024, 4096, 4, 4),
        # the crate's default rendering mode (analytic coverage), on an odd canvas
        named("prefiltered_render_odd", "render", "mixed", 333, 251, 82, 2, 2, prefilter=True),
        # fitting steps: the plain scene, a small crossing one, and the benchmark's mixed scene
        named("plain_step", "step", "plain", 256, 256, 16, 2, 2),
        named("adjoint_step", "step", "adjoint", 128, 128, 8, 4, 4),
        named("mixed_step", "step", "mixed", 512, 512, 256, 4, 4, boundary=512 * 512),
        # the same in the crate's default mode
        named("prefiltered_step", "step", "mixed", 512, 512, 256, 2, 2, prefilter=True),
        # fitting a large illustration, with the crate's own number of edge samples
        named("large_step", "step", "large", 1024, 1024, 4096, 4, 4),
        # many small scenes at once (a data set of icons): one graph replay
        named("batch_step", "batch", "plain", 64, 64, 10, 4, 4, scenes=64),
        # a program that keeps its scene on the host and calls the crate's two functions
        named("mixed_host", "host", "mixed", 512, 512, 256, 4, 4, boundary=512 * 512),
        # a signed-distance image of glyph-like outlines
        named("outline_sdf", "sdf", "plain", 256, 256, 48, 2, 2),
    ]


def draw(rng):
    """One more case of the same ranges (sizes log-uniform, odd ones among them)."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["render", "render", "step", "step", "step", "batch", "host", "sdf", "autograd"])
    spp_x, spp_y = rng.choice([(1, 1), (2, 2), (2, 2), (3, 3), (4, 4), (4, 4), (2, 3), (4, 2)])
    if kind == "batch":
        return _case(kind, "plain", 64, 64, rng.randint(4, 16), spp_x, spp_y, scenes=size(4, 96))
    if kind == "autograd":
        w, h = size(64, 384), size(64, 384)
        return _case(kind, rng.choice(["plain", "styled"]), w, h, size(4, 32), spp_x, spp_y)
    if kind == "sdf":
        w, h = size(64, 384), size(64, 384)
        return _case(kind, "plain", w, h, size(8, 64), min(spp_x, 2), min(spp_y, 2))
    scene = rng.choice(["plain", "mixed", "mixed", "styled", "large"])
    if scene == "large":
        w, h = size(200, 900), size(200, 900)
        count, boundary = max(8, w * h // 256), rng.choice([0, w * h])
    elif scene == "mixed":
        w, h = size(48, 800), size(48, 800)
        count, boundary = max(4, w * h // 1024), rng.choice([0, w * h])
    else:
        w, h = size(48, 512), size(48, 512)
        count, boundary = size(4, 24), rng.choice([0, w * h])
    prefilter = scene != "large" and rng.random() < 0.4
    return _case(kind, scene, w, h, count, spp_x, spp_y, prefilter=prefilter, boundary=boundary)


# ------------------------------------------------------------------ scenes
def _base_scene(case):
    """The case's structure (segment, stop and shape counts): the generator's scene of one fixed seed."""
    w, h, n = case["width"], case["height"], case["count"]
    if case["scene"] == "plain":
        # above 16 paths each path keeps to a part of the canvas, as in the batch workload
        return synth.plain_scene(0, w, h, n, min(1.0, math.sqrt(16.0 / n)))
    if case["scene"] == "adjoint":
        return synth.adjoint_scene(0, w, h)
    if case["scene"] == "mixed":
        return synth.mixed_scene(0, w, h, scale=n / 256.0)
    if case["scene"] == "styled":
        return synth.styled_stroke_scene(0, w, h, n)
    return synth.large_scene(0, w, h, n)


def _vary(scene, seed):
    """Draws the values of a scene again (points, places, rotations, colours, stops, widths) from
    `seed`, within each shape's own extent, and keeps its structure."""
    rng = np.random.default_rng(seed)

    def f32(v):
        return float(np.float32(v))

    def colour():
        r, g, b = rng.uniform(0.0, 1.0, 3)
        return Color(f32(r), f32(g), f32(b), f32(rng.uniform(0.3, 1.0)))

    for s in scene.shapes:
        if isinstance(s.geometry, PathGeometry):
            pts = np.asarray(s.geometry.path.points)
            pts = rng.uniform(pts.min(0), pts.max(0), pts.shape).astype(np.float32)
            s.geometry.path.points = [tuple(map(float, p)) for p in pts]
        s.stroke_width = f32(s.stroke_width * rng.uniform(0.8, 1.25))
    for g in scene.groups:
        m = g.shape_to_canvas
        move = (0.0, 0.0)
        if abs(float(m.flat()[2])) + abs(float(m.flat()[5])) > 0.0:  # a placed group: another place and turn
            x, y = m.transform_point((0.0, 0.0))
            nx, ny = float(rng.uniform(0.0, scene.width)), float(rng.uniform(0.0, scene.height))
            turn = Mat3.rotate(float(rng.uniform(0.0, 2.0 * math.pi)))
            g.set_shape_to_canvas(Mat3.translate(nx, ny).mul(turn).mul(Mat3.translate(-x, -y)).mul(m))
            move = (nx - x, ny - y)
        for which in ("fill", "stroke"):
            p = getattr(g, which)
            if isinstance(p, Color):
                setattr(g, which, colour())
            elif p is not None:
                offs = np.sort(rng.uniform(0.0, 1.0, len(p.stops))).astype(np.float32)
                p.stops = [GradientStop(float(o), colour()) for o in offs]
                for name in ("start", "end", "center"):
                    if hasattr(p, name):
                        v = getattr(p, name)
                        setattr(p, name, (v[0] + move[0], v[1] + move[1]))
    return scene


def _scene(case, seed):
    return _vary(_base_scene(case), seed)


def _batch_scene(case, seed, i):
    n = 4 + (case["count"] + 5 * i) % 13
    return _vary(synth.plain_scene(i, case["width"], case["height"], n), seed * 1000 + i)


def _options(case, seed):
    return RenderOptions(samples_x=case["spp_x"], samples_y=case["spp_y"], seed=seed & 0xffff, jitter=True,
                         use_prefiltering=case["prefilter"])


_RENDERER = []


def _renderer():
    """The process's renderer (a program keeps one for all its scenes)."""
    if not _RENDERER:
        _RENDERER.append(Renderer(0))
    return _RENDERER[0]


def _target(r, scene, opts, out):
    """Renders another scene of the case's kind into the device image `out`."""
    up = r.upload(scene)
    up.render_device(opts, out.data_ptr())
    torch.cuda.synchronize()
    up.close()


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    r = _renderer()
    h, w = case["height"], case["width"]
    opts = _options(case, seed)
    st = {"case": case, "opts": opts, "renderer": r}
    if case["kind"] == "batch":
        n = case["scenes"]
        scenes = [_batch_scene(case, seed, i) for i in range(n)]
        st["ups"] = [r.upload(s) for s in scenes]
        b = Batch(r, st["ups"], opts, BackwardOptions(boundary_samples=case["boundary"]))
        st["batch"] = b
        tmp = torch.empty((h, w, 4), dtype=torch.float32, device=dev)
        lo, hi, glo, ghi = [], [], [], []
        for i in range(n):
            img, tgt, g = b.buffers(i)
            _target(r, _batch_scene(case, seed + 500, i), opts, tmp)
            tgt.copy_(tmp.reshape(-1))
            lo.append(img.data_ptr())
            hi.append(img.data_ptr() + 4 * img.numel())
            glo.append(_address(g.d_shape_params))
            ghi.append(_address(g.d_background) + 16)
        torch.cuda.synchronize()
        st["images"] = device_view(min(lo), (max(hi) - min(lo)) // 4)
        st["grads"] = device_view(min(glo), (max(ghi) - min(glo)) // 4)
        st["images"].owner = st["grads"].owner = b  # the views alias the batch's memory: they keep it
        return st
    scene = _scene(case, seed)
    if case["kind"] == "render":
        st["up"] = r.upload(scene)
        st["image"] = torch.empty((h, w, 4), dtype=torch.float32, device=dev)
    elif case["kind"] == "sdf":
        st["up"] = r.upload(scene)
        st["sdf"] = torch.empty((h, w), dtype=torch.float32, device=dev)
    elif case["kind"] == "step":
        st["up"] = r.upload(scene)
        st["image"] = torch.empty((h, w, 4), dtype=torch.float32, device=dev)
        st["target"] = torch.empty((h, w, 4), dtype=torch.float32, device=dev)
        st["loss"] = torch.zeros(1, dtype=torch.float32, device=dev)
        _target(r, _scene(case, seed + 500), opts, st["target"])
        st["grads"] = DeviceGrads(st["up"].packed, dev)
        st["bopts"] = BackwardOptions(boundary_samples=case["boundary"])
    elif case["kind"] == "host":
        st["scene"] = scene
        st["target"] = r.render(_scene(case, seed + 500), opts).pixels.copy()
        st["d_image"] = torch.empty((h, w, 4), dtype=torch.float32, pin_memory=True).numpy()
        st["bopts"] = BackwardOptions(boundary_samples=case["boundary"])
    else:  # autograd
        st["scene"] = scene
        pts, paints = torch_ops.scene_tensors(scene, dev)
        st["points"], st["paints"] = pts.requires_grad_(True), paints.requires_grad_(True)
        st["target"] = torch.empty((h, w, 4), dtype=torch.float32, device=dev)
        _target(r, _scene(case, seed + 500), opts, st["target"])
        st["bopts"] = BackwardOptions(boundary_samples=case["boundary"])
    torch.cuda.synchronize()
    return st


def _address(p):
    """Address held by a ctypes float pointer."""
    import ctypes

    return ctypes.cast(p, ctypes.c_void_p).value


def run(state):
    case = state["case"]
    if case["kind"] == "render":
        state["up"].render_device(state["opts"], state["image"].data_ptr())
        return {"image": state["image"]}
    if case["kind"] == "sdf":
        state["up"].render_sdf_device(state["opts"], state["sdf"].data_ptr())
        return {"sdf": state["sdf"]}
    if case["kind"] == "step":
        state["up"].fwd_bwd_l2_device(state["opts"], state["bopts"], state["target"].data_ptr(),
                                      state["image"].data_ptr(), state["loss"].data_ptr(), state["grads"])
        return {"image": state["image"], "loss": state["loss"], **state["grads"].tensors}
    if case["kind"] == "batch":
        state["batch"].step()
        return {"images": state["images"], "grads": state["grads"]}
    r, scene, opts = state["renderer"], state["scene"], state["opts"]
    if case["kind"] == "host":
        packed = pack_scene(scene)
        image = r.render(scene, opts, packed=packed).pixels
        np.subtract(image, state["target"], out=state["d_image"])
        np.multiply(state["d_image"], 2.0, out=state["d_image"])
        g = r.render_backward(scene, opts, state["bopts"], state["d_image"], packed=packed)
        return {"image": image, **{k: v for k, v in g.buffers.arrays.items() if v is not None}}
    pts, paints = state["points"], state["paints"]
    image = torch_ops.render(pts, paints, r, scene, opts, state["bopts"])
    loss = ((image - state["target"]) ** 2).sum()
    d_pts, d_paints = torch.autograd.grad(loss, (pts, paints))
    return {"image": image, "loss": loss, "d_points": d_pts, "d_paints": d_paints}


# ------------------------------------------------------------------ unavoidable work
def work(case):
    """Bytes: scene, target and image once, gradients once.  Flops: per sample its position, one
    filter weight and four colour sums per pixel that the filter reaches, and (a gradient pass)
    the same again twice; per edge sample two colours and one gathered gradient."""
    w, h, n = case["width"], case["height"], case["count"]
    spp = case["spp_x"] * case["spp_y"]
    samples = w * h * spp * case["scenes"]
    floats = {"plain": 2 * 18 + 30, "adjoint": 2 * 12 + 30, "mixed": 2 * 18 + 60, "styled": 2 * 8 + 30,
              "large": 2 * 48 + 60}[case["scene"]] * n * case["scenes"]
    image = 16 * w * h * case["scenes"]
    reach = 9 if case["scene"] == "mixed" else 1
    flops = samples * (20 + 15 * reach)
    if case["kind"] == "sdf":
        return {"bytes": 4 * floats + image // 4, "flops": samples * 50}
    if case["kind"] == "render":
        return {"bytes": 4 * floats + image, "flops": flops}
    edge = 0 if case["prefilter"] else (case["boundary"] or w * h * spp) * case["scenes"]
    return {"bytes": 8 * floats + 2 * image, "flops": 3 * flops + edge * (100 + 20 * reach)}


# ------------------------------------------------------------------ 64-bit values
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_F = torch.float64


def exact(case, seed):
    """Images, losses and distances in 64 bits (see the module's docstring)."""
    samples = case["width"] * case["height"] * case["spp_x"] * case["spp_y"] * case["scenes"]
    if case["scene"] in ("large", "styled") or samples * case["count"] > 1.2e9:
        # large: minutes of root finding; styled: its joins and caps are defined by this library alone
        return None
    opts = _options(case, seed)
    if case["kind"] == "batch":
        w, h, n = case["width"], case["height"], case["scenes"]
        if n * w * h * case["spp_x"] * case["spp_y"] > 5e6:
            return None
        im = [_image(_batch_scene(case, seed, i), opts).reshape(-1) for i in range(n)]
        return {"images": torch.cat(im) if w * h % 16 == 0 else None, "grads": None}
    scene = _scene(case, seed)
    if case["kind"] == "sdf":
        return {"sdf": _sdf(scene, opts)}
    image = _image(scene, opts)
    if case["kind"] == "render":
        return {"image": image}
    out = {"image": image}
    if case["kind"] in ("step", "autograd"):
        loss = ((image - _image(_scene(case, seed + 500), opts)) ** 2).sum()
        out["loss"] = loss.reshape(1) if case["kind"] == "step" else loss
    return out


def _sample_points(w, h, opts, jitter, sdf=False):
    """Sample positions [h, w, syn, sxn]: stratified, moved by the crate's PCG32 stream.  They
    are inputs of the path, in 32 bits by definition."""
    sxn, syn = opts.samples_x, opts.samples_y
    shape = (h, w, syn, sxn)
    idx = np.arange(h * w * syn * sxn, dtype=np.uint64)
    rx = ry = np.full(idx.shape, 0.5, np.float32)
    if jitter:
        with np.errstate(over="ignore"):
            mul, inc = np.uint64(6364136223846793005), ((idx + np.uint64(1)) << np.uint64(1)) | np.uint64(1)

            def step(s):
                return s * mul + inc

            def unit(s):
                x = (((s >> np.uint64(18)) ^ s) >> np.uint64(27)).astype(np.uint32)
                rot = (s >> np.uint64(59)).astype(np.uint32)
                u = (x >> rot) | (x << ((np.uint32(32) - rot) & np.uint32(31)))
                return ((u >> np.uint32(9)) | np.uint32(0x3f800000)).view(np.float32) - np.float32(1)

            s = step(np.zeros_like(idx)) + np.uint64(0x853c49e6748fea9b) + np.uint64(opts.seed)
            s = step(s)
            rx = unit(s)
            ry = unit(step(s))
    y, x, sy, sx = np.meshgrid(np.arange(h, dtype=np.float32), np.arange(w, dtype=np.float32),
                               np.arange(syn, dtype=np.float32), np.arange(sxn, dtype=np.float32), indexing="ij")
    rx, ry = rx.reshape(shape), ry.reshape(shape)
    if sdf:
        px, py = x + (sx + rx) * (np.float32(1) / np.float32(sxn)), y + (sy + ry) * (np.float32(1) / np.float32(syn))
    else:
        px, py = x + (sx + rx) / np.float32(sxn), y + (sy + ry) / np.float32(syn)
    return (torch.from_numpy(px.astype(np.float64)).to(_DEV).reshape(h, w, -1),
            torch.from_numpy(py.astype(np.float64)).to(_DEV).reshape(h, w, -1))


def _affine(m):
    return np.asarray(m.flat(), np.float64).reshape(3, 3)


class _Group:
    """One shape group of one shape, in 64 bits."""

    def __init__(self, scene, g):
        assert len(g.shape_indices) == 1
        self.g, self.shape = g, scene.shapes[g.shape_indices[0]]
        self.to_canvas = _affine(g.shape_to_canvas) @ _affine(self.shape.transform)
        self.to_shape = np.linalg.inv(_affine(self.shape.transform)) @ _affine(g.canvas_to_shape)
        geo = self.shape.geometry
        self.path = geo.path if isinstance(geo, PathGeometry) else None
        if self.path is not None:
            pts = np.asarray(self.path.points, np.float64)
            self.segs, k = [], 0  # control points of each segment
            for nc in self.path.num_control_points:
                ids = [k + j for j in range(nc + 2)]
                if self.path.is_closed:
                    ids[-1] %= len(pts)
                self.segs.append(pts[ids])
                k += nc + 1
            box = pts
        else:
            c = np.asarray(geo.center, np.float64)
            r = np.abs([geo.radius, geo.radius] if isinstance(geo, Circle) else geo.radius).astype(np.float64)
            box = np.array([c + r * s for s in ((-1, -1), (1, -1), (-1, 1), (1, 1))])
        lo, hi = box.min(0) - self.shape.stroke_width, box.max(0) + self.shape.stroke_width
        q = np.array([[lo[0], lo[1], 1], [hi[0], lo[1], 1], [lo[0], hi[1], 1], [hi[0], hi[1], 1]]) @ self.to_canvas.T
        self.lo, self.hi = q[:, :2].min(0), q[:, :2].max(0)

    def local(self, px, py):
        m = self.to_shape
        return m[0, 0] * px + m[0, 1] * py + m[0, 2], m[1, 0] * px + m[1, 1] * py + m[1, 2]

    def winding(self, x, y):
        geo = self.shape.geometry
        if self.path is None:
            rx, ry = (geo.radius, geo.radius) if isinstance(geo, Circle) else geo.radius
            return ((((x - geo.center[0]) / rx) ** 2 + ((y - geo.center[1]) / ry) ** 2) < 1.0).to(torch.int32)
        rows = []  # monotone pieces: x and y coefficients, parameter range, y at both ends
        for s in self.segs:
            cx, cy = _poly(s[:, 0]), _poly(s[:, 1])
            roots = np.roots(np.trim_zeros([3 * cy[3], 2 * cy[2], cy[1]], "f")) if cy[1:].any() else np.array([])
            ts = [0.0] + sorted(float(r.real) for r in roots if abs(r.imag) < 1e-14 and 0 < r.real < 1) + [1.0]
            ys = [s[0, 1]] + [float(np.polyval(cy[::-1], t)) for t in ts[1:-1]] + [s[-1, 1]]
            for k in range(len(ts) - 1):
                if ys[k] != ys[k + 1]:
                    rows.append([*cx, *cy, ts[k], ts[k + 1], ys[k], ys[k + 1]])
        out = torch.zeros(x.shape, dtype=torch.int32, device=x.device)
        if not rows:
            return out
        tab = torch.tensor(rows, dtype=_F, device=x.device)
        fx, fy, fo = x.reshape(-1), y.reshape(-1), out.reshape(-1)
        step = max(1, int(1.5e7) // len(rows))
        for a in range(0, fx.numel(), step):
            sx, sy = fx[a:a + step], fy[a:a + step]
            c = [tab[:, k:k + 1] for k in range(12)]
            up = c[11] > c[10]
            on = (sy >= torch.minimum(c[10], c[11])) & (sy < torch.maximum(c[10], c[11]))
            p, q = on.nonzero(as_tuple=True)
            k = [v[p, 0] for v in c]
            ty, u = sy[q], up[p, 0]
            lo, hi = k[8].clone(), k[9].clone()
            for _ in range(48):
                t = 0.5 * (lo + hi)
                below = (((k[7] * t + k[6]) * t + k[5]) * t + k[4] < ty) == u
                lo, hi = torch.where(below, t, lo), torch.where(below, hi, t)
            t = 0.5 * (lo + hi)
            right = ((k[3] * t + k[2]) * t + k[1]) * t + k[0] > sx[q]
            fo[a:a + step].index_add_(0, q, torch.where(right, torch.where(u, 1, -1), 0).to(torch.int32))
        return out

    def distance(self, x, y):
        """Distance to the outline in shape space."""
        geo = self.shape.geometry
        if isinstance(geo, Circle):
            return (torch.sqrt((x - geo.center[0]) ** 2 + (y - geo.center[1]) ** 2) - geo.radius).abs()
        if isinstance(geo, Ellipse):
            rx, ry = geo.radius
            dx, dy = (x - geo.center[0]).abs(), (y - geo.center[1]).abs()
            lo, hi = torch.zeros_like(dx), torch.full_like(dx, math.pi / 2)
            for _ in range(54):
                t = 0.5 * (lo + hi)
                s, c = torch.sin(t), torch.cos(t)
                neg = rx * dx * s - ry * dy * c + (ry * ry - rx * rx) * s * c < 0
                lo, hi = torch.where(neg, t, lo), torch.where(neg, hi, t)
            return torch.sqrt((dx - rx * torch.cos(lo)) ** 2 + (dy - ry * torch.sin(lo)) ** 2)
        best = torch.full_like(x, math.inf)
        for s in self.segs:
            cx, cy = _poly(s[:, 0]), _poly(s[:, 1])
            n = 1 if len(s) == 2 else 48

            def at(t):
                return (((cx[3] * t + cx[2]) * t + cx[1]) * t + cx[0] - x,
                        ((cy[3] * t + cy[2]) * t + cy[1]) * t + cy[0] - y)

            bd, bt = torch.full_like(x, math.inf), torch.zeros_like(x)
            for k in range(n + 1):
                ux, uy = at(k / n)
                d = ux * ux + uy * uy
                near = d < bd
                bd, bt = torch.where(near, d, bd), torch.where(near, torch.full_like(x, k / n), bt)
            lo, hi = (bt - 1.0 / n).clamp(min=0.0), (bt + 1.0 / n).clamp(max=1.0)
            for _ in range(50):
                t = 0.5 * (lo + hi)
                ux, uy = at(t)
                neg = (ux * ((3 * cx[3] * t + 2 * cx[2]) * t + cx[1]) + uy * ((3 * cy[3] * t + 2 * cy[2]) * t + cy[1])) < 0
                lo, hi = torch.where(neg, t, lo), torch.where(neg, hi, t)
            ux, uy = at(lo)
            best = torch.minimum(best, torch.minimum(bd, ux * ux + uy * uy))
        return torch.sqrt(best)

    def inside(self, x, y):
        w = self.winding(x, y)
        return (w.abs() % 2 == 1) if self.g.fill_rule == FillRule.EVEN_ODD else w != 0


def _poly(p):
    """Power coefficients (ascending, four of them) of a Bezier coordinate."""
    if len(p) == 2:
        return np.array([p[0], p[1] - p[0], 0.0, 0.0])
    if len(p) == 3:
        return np.array([p[0], 2 * (p[1] - p[0]), p[0] - 2 * p[1] + p[2], 0.0])
    return np.array([p[0], 3 * (p[1] - p[0]), 3 * (p[0] - 2 * p[1] + p[2]), p[3] - 3 * p[2] + 3 * p[1] - p[0]])


def _paint(paint, px, py):
    """Colour [..., 4] of a paint at canvas points."""
    if not isinstance(paint, (LinearGradient, RadialGradient)):
        return torch.tensor(paint.to_tuple(), dtype=_F, device=px.device).expand(*px.shape, 4)
    if isinstance(paint, LinearGradient):
        ex, ey = paint.end[0] - paint.start[0], paint.end[1] - paint.start[1]
        t = ((px - paint.start[0]) * ex + (py - paint.start[1]) * ey) / max(ex * ex + ey * ey, 1e-3)
    else:
        t = torch.sqrt(((px - paint.center[0]) / paint.radius[0]) ** 2 + ((py - paint.center[1]) / paint.radius[1]) ** 2)
    offs = [float(np.float32(s.offset)) for s in paint.stops]
    cols = [torch.tensor(s.color.to_tuple(), dtype=_F, device=px.device) for s in paint.stops]
    out = cols[-1].expand(*px.shape, 4)
    for k in reversed(range(len(offs) - 1)):
        u = ((t - offs[k]) / (offs[k + 1] - offs[k]) if offs[k + 1] > offs[k] else torch.zeros_like(t))[..., None]
        on = ((t >= offs[k]) & (t < offs[k + 1]))[..., None]
        out = torch.where(on, cols[k] * (1 - u) + cols[k + 1] * u, out)
    return torch.where((t < offs[0])[..., None], cols[0].expand(*px.shape, 4), out)


def _smooth(d):
    t = ((d + 1.0) * 0.5).clamp(0.0, 1.0)
    return t * t * (3.0 - 2.0 * t)


def _image(scene, opts):
    w, h = scene.width, scene.height
    px, py = _sample_points(w, h, opts, opts.jitter and not opts.use_prefiltering)
    acc = torch.tensor(scene.background.to_tuple(), dtype=_F, device=_DEV)
    acc = torch.cat([acc[:3] * acc[3], acc[3:]]).expand(*px.shape, 4).clone()
    for g in scene.groups:
        grp = _Group(scene, g)
        sw = grp.shape.stroke_width
        reach = 1.0 + (sw + 1.0 if opts.use_prefiltering else 0.0)
        x0, x1 = max(0, math.floor(grp.lo[0] - reach)), min(w, math.ceil(grp.hi[0] + reach) + 1)
        y0, y1 = max(0, math.floor(grp.lo[1] - reach)), min(h, math.ceil(grp.hi[1] + reach) + 1)
        if x0 >= x1 or y0 >= y1:
            continue
        sx, sy = px[y0:y1, x0:x1], py[y0:y1, x0:x1]
        lx, ly = grp.local(sx, sy)
        a = acc[y0:y1, x0:x1]
        need = opts.use_prefiltering or g.stroke is not None
        d = grp.distance(lx, ly) if need else None
        # similarity transforms: a distance in shape space times the scale is the canvas distance
        dc = d * math.sqrt(abs(np.linalg.det(grp.to_canvas[:2, :2]))) if need else None
        for paint, stroke in ((g.stroke, True), (g.fill, False)):
            if paint is None:
                continue
            if opts.use_prefiltering:
                if stroke:
                    cov = _smooth(dc + sw) - _smooth(dc - sw)
                else:
                    dd = dc.clamp(max=1.0)
                    cov = _smooth(torch.where(grp.inside(lx, ly), dd, -dd))
            elif stroke:
                cov = (d < sw).to(_F) if sw > 0 else torch.zeros_like(d)
            else:
                cov = grp.inside(lx, ly).to(_F)
            c = _paint(paint, sx, sy)
            al = (c[..., 3] * cov)[..., None]
            a.copy_(torch.cat([a[..., :3] * (1 - al) + c[..., :3] * al, a[..., 3:] * (1 - al) + al], -1))
    f, r = scene.filter, float(np.float32(scene.filter.radius))
    ri = math.ceil(r)
    num = torch.zeros((h, w, 4), dtype=_F, device=_DEV)
    den = torch.zeros((h, w), dtype=_F, device=_DEV)
    for dy in range(-ri, ri + 1):
        for dx in range(-ri, ri + 1):
            ys, yd = slice(max(0, -dy), min(h, h - dy)), slice(max(0, dy), min(h, h + dy))
            xs, xd = slice(max(0, -dx), min(w, w - dx)), slice(max(0, dx), min(w, w + dx))
            if ys.start >= ys.stop or xs.start >= xs.stop:
                continue
            cx = torch.arange(xd.start, xd.stop, dtype=_F, device=_DEV)[None, :, None] + 0.5
            cy = torch.arange(yd.start, yd.stop, dtype=_F, device=_DEV)[:, None, None] + 0.5
            ox, oy = cx - px[ys, xs], cy - py[ys, xs]
            wt = torch.full_like(ox, 1.0 / (4 * r * r)) if f.filter_type == FilterType.BOX else \
                (2.0 / (math.pi * r * r)) * torch.exp(-2.0 * (ox * ox + oy * oy) / (r * r))
            wt = torch.where((ox.abs() > r) | (oy.abs() > r), torch.zeros_like(wt), wt)
            num[yd, xd] += (acc[ys, xs] * wt[..., None]).sum(2)
            den[yd, xd] += wt.sum(2)
    img = torch.where(den[..., None] > 0, num / den[..., None],
                      torch.tensor(scene.background.to_tuple(), dtype=_F, device=_DEV))
    al = img[..., 3:]
    return torch.cat([torch.where(al > 1e-8, img[..., :3] / al, img[..., :3]), al], -1)


def _sdf(scene, opts):
    px, py = _sample_points(scene.width, scene.height, opts, opts.jitter and not opts.use_prefiltering, sdf=True)
    best = torch.full_like(px, math.inf)
    sign = torch.ones_like(px)
    for g in reversed(scene.groups):
        grp = _Group(scene, g)
        lx, ly = grp.local(px, py)
        d = grp.distance(lx, ly) * math.sqrt(abs(np.linalg.det(grp.to_canvas[:2, :2])))
        near = d < best
        best = torch.where(near, d, best)
        s = torch.where(grp.inside(lx, ly), -1.0, 1.0).to(_F) if g.fill is not None else torch.ones_like(d)
        sign = torch.where(near, s, sign)
    return (best * sign).mean(2)
