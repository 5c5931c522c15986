"""The per-cell decisions (diffvg-rs_b200/csrc/cell_classify.cuh) against the oracle's
restatement of the crate's per-sample computation, at random points of random boxes: the
winding contribution of a segment (a constant, steps at levels, parabolas), the segments a
stroke cannot reach a box from, and the chord tests of the others.  Lines, quadratics and cubics; uniform and integer control
points, near-degenerate ones, large coordinates, small segments far from the origin, nearly
flat ones; rows at end points, and points just outside the tolerances.  No decision may differ
from the crate's, and most boxes have to be decided."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ORACLE = os.path.join(os.path.dirname(HERE), "oracle")
LIB = os.path.join(ORACLE, "_build", "libcell_stress.so")
KINDS = ("line", "quadratic", "cubic")
MODES = ("uniform", "integer", "near-degenerate", "large coordinates", "small and far", "nearly flat")


@pytest.fixture(scope="module")
def stress():
    subprocess.run(["make", "-s", "-C", ORACLE], check=True)
    L = C.CDLL(LIB)
    for f in (L.cell_winding_stress, L.cell_point_stress, L.cell_stroke_stress):
        f.argtypes = [C.c_int, C.c_int, C.c_uint64, C.c_uint64, C.c_int, C.POINTER(C.c_ulonglong)]
        f.restype = None

    def run(f, kind, mode, n):
        out = (C.c_ulonglong * 7)()
        getattr(L, f)(kind, mode, 11, n, 16, out)
        return list(out)
    return run


@pytest.mark.parametrize("mode", range(len(MODES)), ids=MODES)
@pytest.mark.parametrize("kind", range(3), ids=KINDS)
def test_cell_winding_never_disagrees(stress, kind, mode):
    boxes, decided, partly, tested, _, wrong, _ = stress("cell_winding_stress", kind, mode, 100_000)
    assert boxes == 100_000 and partly > 0
    assert wrong == 0, f"{wrong} of {tested} points differ from the crate's winding"
    # near-degenerate cubics are left to the per-sample test wherever they are ill conditioned
    assert decided >= (0.5 if mode == 2 and kind == 2 else 0.7) * boxes


@pytest.mark.parametrize("mode", range(len(MODES)), ids=MODES)
@pytest.mark.parametrize("kind", range(3), ids=KINDS)
def test_point_winding_never_disagrees(stress, kind, mode):
    points, decided, crossing, wrong, *_ = stress("cell_point_stress", kind, mode, 100_000)
    assert wrong == 0, f"{wrong} of {points} points differ from the crate's winding"
    assert crossing > 0 and decided >= (0.4 if mode in (1, 2, 5) else 0.55) * points  # half of them lie on or near the curve


@pytest.mark.parametrize("mode", range(len(MODES)), ids=MODES)
@pytest.mark.parametrize("kind", range(3), ids=KINDS)
def test_cell_stroke_never_disagrees(stress, kind, mode):
    boxes, far, full, tested, decided, wrong_miss, wrong_hit = stress("cell_stroke_stress", kind, mode, 100_000)
    assert wrong_miss == 0, f"{wrong_miss} of {tested} points called out of reach are within the stroke"
    # integer coordinates: points for which the crate's bracketing skips the nearest root (1 in 10^7)
    assert wrong_hit <= (3 if kind == 2 and mode == 1 else 0), f"{wrong_hit} points called hits are not"
    assert far >= 0.4 * boxes and decided >= 0.4 * tested
    assert kind == 0 or full > 0
