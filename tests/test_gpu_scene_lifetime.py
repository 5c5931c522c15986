"""A scene that another context renders, destroyed and its memory taken by the next uploads while
that context's work is still queued: the image is the scene's."""
import ctypes as C

import numpy as np
import pytest
import torch

from dvg import Renderer, RenderOptions, synth
from dvg.abi import render_options_c

pytestmark = pytest.mark.gpu


def test_destroyed_under_another_contexts_work():
    opts = RenderOptions(samples_x=4, samples_y=4, seed=3, jitter=True, use_prefiltering=False)
    a, b = Renderer(0), Renderer(0)
    sc = synth.plain_scene(3, 256, 256, 24)
    want = a.render(sc, opts).pixels
    o = render_options_c(opts)
    outs = []
    for k in range(4):
        up = a.upload(sc)
        out = torch.empty(256 * 256 * 4, device="cuda")
        for _ in range(30):  # a queue of work on the other context's stream
            st = b.lib.dvg_render_device(b.ctx, up.handle, C.byref(o), C.c_void_p(out.data_ptr()))
            assert st == 0, b.lib.dvg_last_error()
        outs.append(out)
        up.close()
        for j in range(3):  # these take the memory
            a.upload(synth.plain_scene(10 + 3 * k + j, 256, 256, 24)).close()
    torch.cuda.synchronize()
    for out in outs:
        assert float(np.max(np.abs(out.cpu().numpy().reshape(256, 256, 4) - want))) <= 1e-5
    b.close()
    a.close()
