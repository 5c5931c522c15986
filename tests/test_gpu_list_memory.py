"""Scenes whose cell lists get no memory, some of it or all of it (dvg_context_set_list_memory):
tiles without entries are walked, entries without items keep the full queries, and the results
are those of the full lists.  Images <= 1e-5, gradients <= 1e-4 of their scale, as in
test_gpu_parity (both sides differ by the order of float sums only)."""
import math

import numpy as np
import pytest
import torch

from dvg import BackwardOptions, Batch, Renderer, RenderOptions, Scene, synth
from dvg.abi import scene_with_params
from dvg.scene import Color, Filter, FilterType, Path, PathGeometry, Shape, ShapeGroup

pytestmark = pytest.mark.gpu
ALL = 4 << 30


def _scene(w=61, h=53, rings=5, segs=40):
    """Crowded cells: stroked rings of cubics, quadratics and lines over each other."""
    rng = np.random.default_rng(4)
    sc = Scene(w, h)
    sc.background = Color(1.0, 1.0, 1.0, 1.0)
    sc.filter = Filter(FilterType.GAUSSIAN, 1.0)
    for i in range(rings):
        kind, m = i % 3, segs * (i % 3 + 1)
        ang = 2.0 * math.pi * np.arange(m) / m
        rad = rng.uniform(9.0, 22.0, m)
        pts = [(float(np.float32(w / 2 + i + r * math.cos(a))), float(np.float32(h / 2 + r * math.sin(a)))) for a, r in zip(ang, rad)]
        s = Shape(PathGeometry(Path([kind] * segs, pts, None, True, False)))
        s.stroke_width = 0.6
        sc.shapes.append(s)
        sc.groups.append(ShapeGroup([i], Color(0.2 + 0.1 * i, 0.5, 0.8, 0.7), Color(0.1, 0.9, 0.3, 0.6)))
    return sc


def _bytes(up, share):
    """A share of what the entries and the first guess of the items take."""
    tiles, total = up.tile_count(), int(up.tile_groups().sum())
    return int(tiles * 128 + 1000 + share * total * 16 * (32 + 3 * 16))


@pytest.fixture(scope="module")
def renderer():
    r = Renderer(0)
    yield r
    r.close()


@pytest.fixture
def limited(renderer):
    yield renderer.set_list_memory
    renderer.set_list_memory(ALL)


SHARES = [0.0, 0.02, 0.3, 0.55, 0.8]  # (0.5 has entries for every tile and items for a few)


@pytest.mark.parametrize("share", SHARES)
@pytest.mark.parametrize("prefilter", [False, True])
def test_results_do_not_depend_on_the_room(renderer, limited, share, prefilter):
    sc = _scene()
    opts = RenderOptions(samples_x=4, samples_y=4, seed=3, jitter=True, use_prefiltering=prefilter)
    bo = BackwardOptions(boundary_samples=4000)
    d = np.random.default_rng(1).uniform(-1.0, 1.0, (sc.height, sc.width, 4)).astype(np.float32)
    want, gwant = renderer.render(sc, opts).pixels, renderer.render_backward(sc, opts, bo, d)
    up = renderer.upload(sc)
    nbytes = _bytes(up, share) if share else 0
    up.close()
    limited(nbytes)
    renderer.set_retain(False)
    img, g = renderer.render(sc, opts).pixels, renderer.render_backward(sc, opts, bo, d)
    renderer.set_retain(True)
    assert float(np.max(np.abs(img - want))) <= 1e-5
    for name in ("d_points", "d_paint_params", "d_shape_stroke_width", "d_shape_transform", "d_group_transform"):
        a, b = g.buffers[name], gwant.buffers[name]
        scale = float(np.max(np.abs(b))) + 1e-6
        assert float(np.max(np.abs(a - b))) <= 1e-4 * scale + 1e-6, name


@pytest.mark.parametrize("share", SHARES + [8.0])  # (the last: whole lists, taken in step where they are heavy)
@pytest.mark.parametrize("work_queue", [0, 1])
def test_batch(renderer, limited, share, work_queue):
    scenes = [_scene(), synth.plain_scene(3, 64, 48, 9), _scene(45, 70, 3, 25)]
    opts = RenderOptions(samples_x=4, samples_y=4, seed=3, jitter=True, use_prefiltering=False)
    want = [renderer.render(s, opts).pixels for s in scenes]
    ups = [renderer.upload(s) for s in scenes]
    sizes = [_bytes(u, share) if share else 0 for u in ups]
    for u in ups:
        u.close()
    ups = []
    for s, n in zip(scenes, sizes):
        limited(n)
        ups.append(renderer.upload(s))
    b = Batch(renderer, ups, opts, BackwardOptions(boundary_samples=2000))
    b.set_tuning(1, 4, 16, work_queue)
    for graph in (False, True):
        b.step(graph)
        b.losses()  # waits
        for i, s in enumerate(scenes):
            img = b.buffers(i)[0].cpu().numpy().reshape(s.height, s.width, 4)
            assert float(np.max(np.abs(img - want[i]))) <= 1e-5, i
    b.close()
    for u in ups:
        u.close()


@pytest.mark.parametrize("share", SHARES + [1.0])
@pytest.mark.parametrize("step_share", [0.0, 0.5, 1e6])
def test_optimised_scene(renderer, limited, share, step_share):
    """Room chosen at upload and again when the steps are set up: after some steps the scene's lists
    still render the geometry that it has then (a fresh upload of the same points)."""
    sc = _scene()
    opts = RenderOptions(samples_x=2, samples_y=2, seed=3, jitter=True, use_prefiltering=False)
    probe = renderer.upload(sc)
    nbytes, sbytes = (int(_bytes(probe, x)) if x else 0 for x in (share, step_share))
    probe.close()
    limited(nbytes)
    up = renderer.upload(sc)
    other = Batch(renderer, [up], opts, BackwardOptions(boundary_samples=500))  # holds the tables of now
    b = Batch(renderer, [up], opts, BackwardOptions(boundary_samples=500))
    limited(min(sbytes, ALL))
    b.set_adam(0.5)
    for _ in range(3):
        b.step(True)
    b.losses()
    pts, _ = b.scene_params(0)
    limited(ALL)
    fresh = renderer.upload(scene_with_params(sc, up.packed, pts))
    a, c = (torch.empty(sc.width * sc.height * 4, device="cuda") for _ in range(2))
    up.render_device(opts, a.data_ptr())
    fresh.render_device(opts, c.data_ptr())
    torch.cuda.synchronize()
    assert float((a - c).abs().max()) <= 1e-5
    b.close()
    other.close()
    up.close()
    fresh.close()


def test_room_for_steps_where_the_tile_list_is_full(renderer):
    """A canvas of one tile has every group in its list from the start; its cell lists are still made
    anew, with room for what steps move, when the steps are set up (once)."""
    sc = _scene(16, 16, 3, 10)
    up = renderer.upload(sc)
    assert int(up.tile_groups().sum()) == 3  # the list needs no growth
    b = Batch(renderer, [up], RenderOptions(samples_x=2, samples_y=2, seed=1, use_prefiltering=False))
    n = [renderer.launch_count]
    for _ in range(2):
        b.set_adam(0.1)
        n.append(renderer.launch_count)
    assert n[1] > n[0] and n[2] == n[1]
    b.close()
    up.close()


@pytest.mark.parametrize("share", [0.0, 0.3, 8.0])
def test_two_batches_of_one_scene(renderer, limited, share):
    """A batch made before another one optimises its scene: its steps render the geometry of now, from
    the lists of now (the tile offsets that it reads are written in place)."""
    sc = _scene()
    opts = RenderOptions(samples_x=2, samples_y=2, seed=3, jitter=True, use_prefiltering=False)
    probe = renderer.upload(sc)
    nbytes = _bytes(probe, share) if share else 0
    probe.close()
    limited(nbytes)
    up, more = renderer.upload(sc), renderer.upload(synth.plain_scene(3, 64, 48, 9))
    plain = Batch(renderer, [more, up], opts, BackwardOptions(boundary_samples=500))
    plain.step(True)
    b = Batch(renderer, [up], opts, BackwardOptions(boundary_samples=500))
    b.set_adam(2.0)
    for _ in range(4):
        b.step(True)
    b.losses()
    pts, _ = b.scene_params(0)
    limited(ALL)
    want = renderer.render(scene_with_params(sc, up.packed, pts), opts).pixels.reshape(-1)
    plain.step(True)
    plain.losses()
    assert float(np.max(np.abs(plain.buffers(1)[0].cpu().numpy() - want))) <= 1e-5
    other = renderer.render(more.scene, opts).pixels.reshape(-1)
    assert float(np.max(np.abs(plain.buffers(0)[0].cpu().numpy() - other))) <= 1e-5
    b.close()
    plain.close()
    up.close()
    more.close()
