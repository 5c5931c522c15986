"""The pass that gathers the image adjoint and the filter-radius adjoint together, for every
filter (the parabolic one, whose adjoint the crate does not scale by the weight's, included), at
radii with one, two and more pixels to a side and sample counts with and without lane groups;
and radii so small that the squares of the weights overflow.

d_filter_radius, one sum over all samples and footprint pixels, against the same sum in f64, over
a canvas of one colour: within 1e-5 of the sum of the terms' magnitudes (some thirty f32
operations of 6e-8 a term, and five times that for the order of the sum)."""
import numpy as np
import pytest

import pyoracle
from dvg import BackwardOptions, Renderer, RenderOptions, Scene, synth
from dvg.scene import Color, Filter, FilterType, Rect, Shape, ShapeGroup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    r = Renderer(0)
    yield r
    r.close()


def _weight(kind, r, x, y):
    """A filter's weight and its derivative by the radius (the crate's, src/backward/filters.rs), the
    latter's terms apart."""
    n = 1.0 / (r * r)
    if kind == FilterType.BOX:
        w, d = np.full(x.shape, 0.25 * n), [np.full(x.shape, -2.0 / (2.0 * r) ** 2)]
    elif kind == FilterType.TENT:
        fx, fy = r - np.abs(x), r - np.abs(y)
        w, d = fx * fy * n * n, [fy * n, fx * n, -4.0 * fx * fy / r ** 5]
    elif kind == FilterType.RADIAL_PARABOLIC:
        w = (16.0 / 9.0) * (1 - (x / r) ** 2) * (1 - (y / r) ** 2)
        d = [-(2 * x * x + 2 * y * y) / r ** 3]
    elif kind == FilterType.HANN:
        ax, ay = 2 * np.pi * (x / (2 * r) + 0.5), 2 * np.pi * (y / (2 * r) + 0.5)
        fx, fy = 0.5 * (1 - np.cos(ax)), 0.5 * (1 - np.cos(ay))
        w = fx * fy * n
        d = [fy * n * np.pi * np.sin(ax) * (-2 * x / (4 * r * r)), fx * n * np.pi * np.sin(ay) * (-2 * y / (4 * r * r)),
             -2 * fx * fy / r ** 3]
    else:
        q = x * x + y * y
        w = 2.0 / (np.pi * r * r) * np.exp(-2.0 * q / (r * r))
        d = [w * 4 * q / r ** 3, -w * 2.0 / r]
    out = (np.abs(x) > r) | (np.abs(y) > r)
    return np.where(out, 0.0, w), [np.where(out, 0.0, v) for v in d]


@pytest.mark.parametrize("spp", [(2, 2), (4, 4), (3, 2)])
@pytest.mark.parametrize("radius", [0.7, 1.6, 3.2])
@pytest.mark.parametrize("kind", list(FilterType))
@pytest.mark.parametrize("prefilter", [False, True])
def test_filter_radius_sum(renderer, kind, radius, spp, prefilter):
    W, H = 45, 37
    color = np.array([0.25, 0.5, 0.75, 1.0])
    sc = Scene(W, H)
    sc.filter = Filter(kind, radius)
    sc.shapes.append(Shape(Rect((-20.0, -20.0), (W + 20.0, H + 20.0))))
    sc.groups.append(ShapeGroup([0], Color(*color), None))
    opts = RenderOptions(samples_x=spp[0], samples_y=spp[1], seed=3, jitter=False, use_prefiltering=prefilter)
    d = np.random.default_rng(2).uniform(-1.0, 1.0, (H, W, 4)).astype(np.float32)
    got = float(renderer.render_backward(sc, opts, BackwardOptions(boundary_samples=1), d).buffers["d_filter_radius"][0])

    r, ri = float(np.float32(radius)), int(np.ceil(radius))
    dt = (d.astype(np.float64) * color).sum(2)
    mag = (np.abs(d.astype(np.float64)) * color).sum(2)
    ys, xs = np.mgrid[0:H, 0:W]
    ws = np.zeros((H, W))
    taps = []
    for sy in range(spp[1]):
        for sx in range(spp[0]):
            ox, oy = (sx + 0.5) / spp[0], (sy + 0.5) / spp[1]
            for j in range(-ri, ri + 1):
                for i in range(-ri, ri + 1):
                    px, py = xs + i, ys + j
                    ok = (px >= 0) & (px < W) & (py >= 0) & (py < H)
                    px, py = px[ok], py[ok]
                    w, dw = _weight(kind, r, np.full(px.shape, i + 0.5 - ox), np.full(px.shape, j + 0.5 - oy))
                    np.add.at(ws, (py, px), w)
                    taps.append((px, py, w, dw))
    total = size = 0.0
    for px, py, w, dw in taps:
        a = np.where(w > 0.0, 1.0, 0.0)
        s = ws[py, px]
        unit = 1.0 if kind == FilterType.RADIAL_PARABOLIC else dt[py, px] * (s - w * (s - w)) / (s * s)
        bound = 1.0 if kind == FilterType.RADIAL_PARABOLIC else mag[py, px] * (s + w * np.abs(s - w)) / (s * s)
        total += float((a * unit * sum(dw)).sum())
        size += float((a * bound * sum(np.abs(v) for v in dw)).sum())
    assert abs(got - total) <= 1e-5 * size, (got, total, size)


@pytest.mark.parametrize("radius", [1e-16, 1e-13])
@pytest.mark.parametrize("prefilter", [False, True])
def test_radius_close_to_zero(renderer, radius, prefilter):
    """One sample at each pixel's centre, the only point within such a radius."""
    sc = synth.plain_scene(4, 24, 20, 3)
    sc.filter = Filter(FilterType.GAUSSIAN, radius)
    opts = RenderOptions(samples_x=1, samples_y=1, seed=3, jitter=False, use_prefiltering=prefilter)
    d = np.ones((20, 24, 4), np.float32)
    bo = BackwardOptions(boundary_samples=100)
    g = renderer.render_backward(sc, opts, bo, d)
    _, ref = pyoracle.render_backward(sc, opts, bo, d)
    assert float(ref["d_filter_radius"][0]) == 0.0
    assert float(g.buffers["d_filter_radius"][0]) == 0.0
