"""Where the distance searches' starting bound must not apply: a stroke width that is no number
(its group's fill takes the stroke's search), and points off the canvas, over which the two maps
of a group have not been compared."""
import numpy as np
import pytest

from dvg import Renderer, RenderOptions, Scene
from dvg.scene import Color, Filter, FilterType, Path, PathGeometry, Shape, ShapeGroup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    r = Renderer(0)
    yield r
    r.close()


def _path(points):
    return Path([0] * len(points), points, None, True, False)


def test_stroke_width_that_is_no_number(renderer):
    """The prefiltered image of the fill alone."""
    def scene(stroke):
        sc = Scene(40, 32)
        sc.background = Color(1.0, 1.0, 1.0, 1.0)
        sc.filter = Filter(FilterType.BOX, 0.5)
        s = Shape(PathGeometry(_path([(7.3, 5.2), (31.6, 9.1), (17.4, 27.7)])))
        s.stroke_width = float("nan") if stroke else 0.0
        sc.shapes.append(s)
        sc.groups.append(ShapeGroup([0], Color(0.2, 0.4, 0.8, 1.0), Color(0.9, 0.1, 0.1, 1.0) if stroke else None))
        return sc

    opts = RenderOptions(samples_x=2, samples_y=2, seed=3, jitter=True, use_prefiltering=True)
    a, b = renderer.render(scene(True), opts).pixels, renderer.render(scene(False), opts).pixels
    assert float(np.max(np.abs(a - b))) <= 1e-5


@pytest.mark.parametrize("x", [8.0, 10000.0])
def test_position_off_the_canvas(renderer, x):
    """Two outlines 1 and 0.3 to the right of a point.  The nearer one's map to its shape space is
    not quite the inverse of the map back: off by 0.007 pixel over a canvas of 16 and by 4 pixels
    at x = 10000, where the shape's edge is 3.7 units from the point's image."""
    sc = Scene(16, 16)
    sc.background = Color(1.0, 1.0, 1.0, 1.0)
    for dx in (0.3, 1.0):
        sc.shapes.append(Shape(PathGeometry(_path([(x + dx, -90.0), (x + dx, 90.0), (x + 110.0, 0.0)]))))
        sc.groups.append(ShapeGroup([len(sc.shapes) - 1], None, Color(0.2, 0.4, 0.8, 1.0)))
    m = sc.groups[0].canvas_to_shape.m.copy()
    m[0, 0] = np.float32(1.0004)
    sc.groups[0].canvas_to_shape.m = m
    got = float(renderer.eval_positions(sc, np.array([[x, 8.0]], np.float32))[0])
    assert abs(abs(got) - 0.3) <= 2e-3  # (an ulp of x is 1e-3 at 10000)
