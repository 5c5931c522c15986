"""Per-cell lists at their edges, against the oracle: canvases that end inside a tile and a cell,
paths at the longest listed length and one past it, more list items than a cell holds, one
segment, groups of several shapes, approximate closest points, shapes whose transform is
singular or scales far up or down.  Images <= 1e-5 (one sample that changed side is >= 1/16 of
a colour), gradients <= 1e-4 of their scale, as in test_gpu_parity."""
import math

import numpy as np
import pytest

from dvg import BackwardOptions, Renderer, RenderOptions, Scene
from dvg.scene import Color, FillRule, Filter, FilterType, Mat3, Path, PathGeometry, Shape, ShapeGroup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    r = Renderer(0)
    yield r
    r.close()


def _ring(n, kind, cx, cy, r0, r1, seed):
    """A closed path of n segments (kind 0 lines, 1 quadratics, 2 cubics) wobbling around a circle."""
    rng = np.random.default_rng(seed)
    pts = []
    m = n * (kind + 1)
    for k in range(m):
        a, r = 2.0 * math.pi * k / m, float(rng.uniform(r0, r1))
        pts.append((float(np.float32(cx + r * math.cos(a))), float(np.float32(cy + r * math.sin(a)))))
    return Path([kind] * n, pts, None, True, False)


def _scene(w, h, paths, stroke=0.0, rule=FillRule.NON_ZERO):
    sc = Scene(w, h)
    sc.background = Color(1.0, 1.0, 1.0, 1.0)
    sc.filter = Filter(FilterType.BOX, 0.5)
    for i, p in enumerate(paths):
        s = Shape(PathGeometry(p))
        s.stroke_width = stroke
        sc.shapes.append(s)
        g = ShapeGroup([i], Color(0.2 + 0.1 * i, 0.5, 0.8 - 0.1 * i, 0.7), Color(0.1, 0.9, 0.3, 0.6) if stroke else None)
        g.fill_rule = rule
        sc.groups.append(g)
    return sc


def _check(renderer, sc, spp=(4, 4)):
    import pyoracle

    opts = RenderOptions(samples_x=spp[0], samples_y=spp[1], seed=3, jitter=True, use_prefiltering=False)
    img = renderer.render(sc, opts).pixels
    ref = pyoracle.render(sc, opts)
    assert float(np.max(np.abs(img - ref))) <= 1e-5
    rng = np.random.default_rng(1)
    d = rng.uniform(-1.0, 1.0, img.shape).astype(np.float32)
    bo = BackwardOptions(boundary_samples=2000)
    g = renderer.render_backward(sc, opts, bo, d)
    _, gref = pyoracle.render_backward(sc, opts, bo, d)
    for name in ("d_points", "d_paint_params", "d_shape_stroke_width", "d_shape_transform", "d_group_transform"):
        a, b = g.buffers[name], gref[name]
        scale = float(np.max(np.abs(b))) + 1e-6
        assert float(np.max(np.abs(a - b))) <= 1e-4 * scale + 1e-6, name


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2, 47, 49, 511, 512, 513])
def test_path_lengths(renderer, n, kind):
    if n * (kind + 1) < 3:
        pytest.skip("no area")
    w, h = 37, 43  # neither a multiple of the tile nor of the cell
    _check(renderer, _scene(w, h, [_ring(n, kind, 17.0, 21.0, 6.0, 15.0, n + kind)], 0.75, FillRule.EVEN_ODD))


@pytest.mark.parametrize("spp", [(1, 1), (2, 2), (3, 3), (4, 4), (8, 8), (5, 4)])
def test_crowded_cell(renderer, spp):
    """Sixty segments through one 4x4 cell: more than a cell lists."""
    _check(renderer, _scene(21, 19, [_ring(60, 2, 10.0, 10.0, 0.2, 1.6, 5), _ring(9, 1, 9.0, 9.0, 3.0, 8.0, 6)], 0.3), spp)


@pytest.mark.parametrize("scale", [0.01, 1.0, 100.0])
def test_transforms_and_groups(renderer, scale):
    sc = _scene(45, 33, [_ring(7, 2, 0.0, 0.0, 3.0 / scale, 14.0 / scale, 8), _ring(6, 1, 20.0, 15.0, 3.0, 12.0, 9),
                         _ring(8, 0, 25.0, 17.0, 2.0, 9.0, 10), _ring(5, 2, 14.0, 12.0, 2.0, 9.0, 11)], 0.0)
    sc.groups[0].set_shape_to_canvas(Mat3.translate(22.0, 16.0).mul(Mat3.rotate(0.7)).mul(Mat3.scale(scale, 0.8 * scale)))
    sc.shapes[1].stroke_width = 1.25
    sc.shapes[1].geometry.path.use_distance_approx = True
    sc.groups[1].stroke = Color(0.9, 0.1, 0.2, 0.8)
    sc.shapes[3].transform = Mat3.scale(1.0, 0.0)  # singular: sampled untransformed
    sc.groups[1].shape_indices = [1, 2]  # several shapes in one group
    _check(renderer, sc)


@pytest.mark.parametrize("samples", [1, 31, 33, 127, 129, 5000, 60000])
def test_edge_sample_counts(renderer, samples):
    """The edge pass's segment-ordered sums around a warp's share of 128 samples, on every
    primitive (circle, ellipse, rectangle, mixed path, per-point thickness)."""
    import pyoracle
    from dvg import synth

    sc = synth.primitives_scene()
    opts = RenderOptions(samples_x=2, samples_y=2, seed=5, jitter=True, use_prefiltering=False)
    d = np.random.default_rng(2).uniform(-1.0, 1.0, (sc.height, sc.width, 4)).astype(np.float32)
    bo = BackwardOptions(boundary_samples=samples)
    g = renderer.render_backward(sc, opts, bo, d)
    _, gref = pyoracle.render_backward(sc, opts, bo, d)
    for name in ("d_points", "d_thickness", "d_shape_params", "d_shape_stroke_width", "d_shape_transform",
                 "d_group_transform"):
        a, b = g.buffers[name], gref[name]
        scale = float(np.max(np.abs(b))) + 1e-6
        assert float(np.max(np.abs(a - b))) <= 1e-4 * scale + 1e-6, name


@pytest.mark.parametrize("how", ["scale 0.02", "scale 50", "skewed", "not the inverse", "singular", "two shapes"])
def test_distance_reach(renderer, how):
    """Searches that start from the distance they are asked for: prefiltered image and gradients
    and the signed distance against the oracle's unbounded searches."""
    import pyoracle

    k = {"scale 0.02": 0.02, "scale 50": 50.0}.get(how, 1.0)
    sc = _scene(45, 33, [_ring(7, 2, 0.0, 0.0, 3.0 / k, 14.0 / k, 8), _ring(6, 1, 20.0, 15.0, 3.0, 12.0, 9),
                         _ring(5, 0, 30.0, 12.0, 2.0, 8.0, 10)], 0.0)
    g = sc.groups[0]
    g.set_shape_to_canvas(Mat3.translate(22.0, 16.0).mul(Mat3.rotate(0.7)).mul(Mat3.scale(k, k)))
    sc.shapes[1].stroke_width = 1.5
    sc.groups[1].stroke = Color(0.9, 0.1, 0.2, 0.8)
    if how == "skewed":
        g.set_shape_to_canvas(Mat3.translate(22.0, 16.0).mul(Mat3.rotate(0.7)).mul(Mat3.scale(3.0, 0.2)))
    if how == "not the inverse":
        g.canvas_to_shape = Mat3.scale(0.9, 1.1).mul(g.canvas_to_shape)
    if how == "singular":
        sc.shapes[1].transform = Mat3.scale(0.0, 1.0)
    if how == "two shapes":
        sc.groups[1].shape_indices = [1, 2]
    opts = RenderOptions(samples_x=2, samples_y=2, seed=3, jitter=True, use_prefiltering=True)
    assert float(np.max(np.abs(renderer.render(sc, opts).pixels - pyoracle.render(sc, opts)))) <= 1e-5
    a, b = renderer.render_sdf(sc, opts).values, pyoracle.render_sdf(sc, opts).reshape(33, 45)
    assert float(np.max(np.abs(a - b) / (1.0 + np.abs(b)))) <= 1e-5
    d = np.random.default_rng(1).uniform(-1.0, 1.0, (33, 45, 4)).astype(np.float32)
    gr = renderer.render_backward(sc, opts, BackwardOptions(), d)
    _, ref = pyoracle.render_backward(sc, opts, BackwardOptions(), d)
    for name in ("d_points", "d_paint_params", "d_shape_stroke_width"):
        x, y = gr.buffers[name], ref[name]
        scale = float(np.max(np.abs(y))) + 1e-6
        assert float(np.max(np.abs(x - y))) <= 1e-4 * scale + 1e-6, name


@pytest.mark.parametrize("how", ["plain", "scale 0.02", "scale 50", "even odd", "no stroke width", "crowded",
                                 "two shapes", "past the canvas"])
def test_prefiltered_fill_and_stroke(renderer, how):
    """One search for a group's fill and stroke, and the fill's inside test from the cell lists:
    prefiltered image and gradients against the oracle, which searches and tests for each."""
    import pyoracle

    k = {"scale 0.02": 0.02, "scale 50": 50.0}.get(how, 1.0)
    n = 300 if how == "crowded" else 9
    rule = FillRule.EVEN_ODD if how == "even odd" else FillRule.NON_ZERO
    sc = _scene(45, 33, [_ring(n, 2, 0.0, 0.0, 3.0 / k, 14.0 / k, 8), _ring(6, 1, 20.0, 15.0, 3.0, 12.0, 9),
                         _ring(5, 0, 30.0, 12.0, 2.0, 8.0, 10)], 1.5, rule)
    x, y = (2.0, 30.0) if how == "past the canvas" else (22.0, 16.0)
    sc.groups[0].set_shape_to_canvas(Mat3.translate(x, y).mul(Mat3.rotate(0.7)).mul(Mat3.scale(k, k)))
    if how == "no stroke width":
        sc.shapes[1].stroke_width = 0.0
    if how == "two shapes":
        sc.groups[1].shape_indices = [1, 2]
    opts = RenderOptions(samples_x=2, samples_y=2, seed=3, jitter=True, use_prefiltering=True)
    assert float(np.max(np.abs(renderer.render(sc, opts).pixels - pyoracle.render(sc, opts)))) <= 1e-5
    d = np.random.default_rng(1).uniform(-1.0, 1.0, (33, 45, 4)).astype(np.float32)
    gr = renderer.render_backward(sc, opts, BackwardOptions(), d)
    _, ref = pyoracle.render_backward(sc, opts, BackwardOptions(), d)
    for name in ("d_points", "d_paint_params", "d_shape_stroke_width", "d_group_transform", "d_shape_transform"):
        a, b = gr.buffers[name], ref[name]
        scale = float(np.max(np.abs(b))) + 1e-6
        assert float(np.max(np.abs(a - b))) <= 1e-4 * scale + 1e-6, name


@pytest.mark.parametrize("spp", [(2, 2), (4, 4), (5, 4), (8, 8)])
def test_long_lists(renderer, spp):
    """Cells with many groups of many list items, which a CTA takes entry by entry: in whole
    tiles, in tiles that the canvas cuts, with one cell to a CTA and with several."""
    paths = [_ring(40, i % 3, 20.0 + i, 18.0, 6.0, 17.0, 20 + i) for i in range(8)]
    _check(renderer, _scene(53, 41, paths, 0.7), spp)
