"""When a scene's cell lists are built: by the first call that reads them, whichever call, context,
thread or capture that is; never for signed distances.  Every image is that of a plain render
(<= 1e-5: the order of float sums)."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from dvg import BackwardOptions, Batch, DeviceGrads, Renderer, RenderOptions, synth
from dvg.abi import RenderOptionsC, render_options_c

pytestmark = pytest.mark.gpu
OPTS = RenderOptions(samples_x=4, samples_y=4, seed=3, jitter=True, use_prefiltering=False)
W, H = 200, 120
N = W * H * 4


@pytest.fixture(scope="module")
def renderer():
    r = Renderer(0)
    yield r
    r.close()


@pytest.fixture(scope="module")
def scene():
    return synth.plain_scene(4, W, H, 14)


@pytest.fixture(scope="module")
def want(renderer, scene):
    return renderer.render(scene, OPTS).pixels.reshape(-1)


def _launches(r, f):
    n = r.launch_count
    f()
    torch.cuda.synchronize()
    return r.launch_count - n


def _same(out, want):
    torch.cuda.synchronize()
    assert float(np.max(np.abs(out.cpu().numpy().reshape(-1) - want))) <= 1e-5


def test_signed_distances_build_none(renderer, scene):
    out = torch.empty(W * H, device="cuda")
    up = renderer.upload(scene)
    first = _launches(renderer, lambda: up.render_sdf_device(OPTS, out.data_ptr()))
    assert first == _launches(renderer, lambda: up.render_sdf_device(OPTS, out.data_ptr()))
    img = torch.empty(N, device="cuda")
    a = _launches(renderer, lambda: up.render_device(OPTS, img.data_ptr()))
    assert a == _launches(renderer, lambda: up.render_device(OPTS, img.data_ptr())) + 1  # the lists, once
    up.close()


@pytest.mark.parametrize("first", ["render", "host", "noalloc", "backward", "shard", "batch", "prefiltered"])
def test_first_reader(renderer, scene, want, first):
    up = renderer.upload(scene)
    out = torch.full((N,), -1.0, device="cuda")
    if first == "host":
        _same(torch.from_numpy(up.render_host(OPTS)), want)
    elif first == "noalloc":
        f = renderer.lib.dvg_render_device_noalloc
        f.argtypes, f.restype = [C.c_void_p, C.c_void_p, C.POINTER(RenderOptionsC), C.c_void_p], C.c_int
        o = render_options_c(OPTS)
        for _ in range(2):
            assert f(renderer.ctx, up.handle, C.byref(o), C.c_void_p(out.data_ptr())) == 0
            _same(out, want)
    elif first == "backward":
        d = torch.ones(N, device="cuda")
        bo = BackwardOptions(boundary_samples=1000)
        got = []
        for _ in range(2):
            g = DeviceGrads(up.packed, torch.device("cuda"))
            up.backward_device(OPTS, bo, d.data_ptr(), g)
            torch.cuda.synchronize()
            got.append(g.flat().cpu().numpy())
        scale = float(np.max(np.abs(got[1])))
        assert float(np.max(np.abs(got[0] - got[1]))) <= 1e-4 * scale
    elif first == "shard":
        acc, ws = torch.zeros(N, device="cuda"), torch.zeros(W * H, device="cuda")
        up.shard_forward(OPTS, (0, up.tile_count()), acc.data_ptr(), ws.data_ptr())
        up.shard_resolve(acc.data_ptr(), ws.data_ptr(), out.data_ptr())
        _same(out, want)
    elif first == "batch":
        b = Batch(renderer, [up, renderer.upload(synth.plain_scene(5, 64, 64, 5))], OPTS, BackwardOptions())
        for graph in (False, True):
            b.step(graph)
            b.losses()
            _same(b.buffers(0)[0], want)
        b.close()
    elif first == "prefiltered":
        po = RenderOptions(samples_x=2, samples_y=2, seed=3, jitter=True, use_prefiltering=True)
        pw = renderer.render(scene, po).pixels.reshape(-1)
        up.render_device(po, out.data_ptr())
        _same(out, pw)
    for _ in range(3):
        up.render_device(OPTS, out.data_ptr())
        _same(out, want)
    up.close()


@pytest.mark.parametrize("warm", [False, True])
def test_first_reader_in_a_capture(renderer, scene, want, warm):
    """Captured before the lists exist, or right after the call that started them; replayed on
    another stream."""
    up = renderer.upload(scene)
    out = torch.full((N,), -1.0, device="cuda")
    other = renderer.upload(scene)
    other.render_device(OPTS, out.data_ptr())  # the context's own buffers are there
    torch.cuda.synchronize()
    if warm:
        up.render_device(OPTS, out.data_ptr())
    lib = torch.cuda.ExternalStream(renderer.stream_handle)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=lib):
        up.render_device(OPTS, out.data_ptr())
    torch.cuda.synchronize()
    out.fill_(-1.0)
    for _ in range(2):
        graph.replay()
        _same(out, want)
    del graph
    up.render_device(OPTS, out.data_ptr())
    _same(out, want)
    up.close()
    other.close()


def test_first_readers_of_several_contexts_and_threads(renderer, scene, want):
    """Four threads, each with a context of its own, meet at one new scene."""
    others = [Renderer(0) for _ in range(4)]
    o = render_options_c(OPTS)
    for _ in range(5):
        up = renderer.upload(scene)
        outs = [torch.full((N,), -1.0, device="cuda") for _ in others]
        torch.cuda.synchronize()
        gate, status = threading.Barrier(len(others)), []

        def work(r, out):
            gate.wait()
            for _ in range(3):
                status.append(r.lib.dvg_render_device(r.ctx, up.handle, C.byref(o), C.c_void_p(out.data_ptr())))

        ts = [threading.Thread(target=work, args=a) for a in zip(others, outs)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert status == [0] * 12
        up.close()  # waits for them
        for out in outs:
            _same(out, want)
    for r in others:
        r.close()


def test_crowded_cells_get_their_room_later(renderer):
    """A scene that asks for more items than the first guess: the first render runs with what fits,
    later ones with all, and a batch made in between keeps the tables that it was made with."""
    import test_gpu_list_memory as lm

    sc = lm._scene(rings=8, segs=90)
    ref = renderer.render(sc, OPTS).pixels.reshape(-1)
    up = renderer.upload(sc)
    out = torch.empty(ref.size, device="cuda")
    up.render_device(OPTS, out.data_ptr())
    _same(out, ref)
    b = Batch(renderer, [up], OPTS, BackwardOptions(boundary_samples=500))
    for _ in range(3):
        up.render_device(OPTS, out.data_ptr())
        _same(out, ref)
        b.step(True)
        b.losses()
        _same(b.buffers(0)[0], ref)
    b.close()
    up.close()


@pytest.mark.parametrize("spp", [(1, 1), (2, 2), (4, 4)])
def test_small_first_render_walks_the_tiles(renderer, spp):
    """Up to 74 CTAs (16 tiles here: 16, 64 and 256) a first render leaves the lists to the second
    reader; in a fused step they are built for its backward pass."""
    sc = synth.plain_scene(3, 64, 64, 10)
    opts = RenderOptions(samples_x=spp[0], samples_y=spp[1], seed=3, jitter=True, use_prefiltering=False)
    out = [torch.empty(64 * 64 * 4, device="cuda") for _ in range(3)]
    up = renderer.upload(sc)
    n = [_launches(renderer, lambda o=o: up.render_device(opts, o.data_ptr())) for o in out]
    small = 16 * spp[0] * spp[1] <= 74
    assert n[1] - n[2] == (1 if small else 0) and n[0] - n[2] == (0 if small else 1)
    for o in out[:2]:
        _same(o, out[2].cpu().numpy())
    up.close()
    one = renderer.render(sc, opts).pixels.reshape(-1)
    _same(out[2], one)
    up = renderer.upload(sc)
    g = DeviceGrads(up.packed, torch.device("cuda"))
    img, loss = torch.empty(64 * 64 * 4, device="cuda"), torch.empty(1, device="cuda")
    for _ in range(2):
        up.fwd_bwd_l2_device(opts, BackwardOptions(), out[2].data_ptr(), img.data_ptr(), loss.data_ptr(), g)
        _same(img, one)
    up.close()
