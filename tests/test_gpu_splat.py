"""The splat summed over a pixel's lanes (4 or 16 samples next to each other) at filter radii of
several pixels, against the per-sample splat (the layout with one sub-sample to a warp), and the
counts that have no lane groups.  Both sides sum the same N = samples * (2 * ceil(r) + 1)^2 terms in
other orders: within N * 6e-8, at most one rounding a term."""
import math

import numpy as np
import pytest
import torch

from dvg import Renderer, RenderOptions, synth
from dvg.scene import Filter, FilterType

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [(2, 2), (4, 4), (4, 2), (8, 4)])
@pytest.mark.parametrize("radius", [0.5, 1.6, 3.2, 7.9])
@pytest.mark.parametrize("kind", [FilterType.BOX, FilterType.TENT, FilterType.GAUSSIAN])
@pytest.mark.parametrize("prefilter", [False, True])
def test_lane_groups(kind, radius, spp, prefilter):
    r = Renderer(0)
    sc = synth.plain_scene(4, 45, 37, 5)
    sc.filter = Filter(kind, radius)
    opts = RenderOptions(samples_x=spp[0], samples_y=spp[1], seed=3, jitter=True, use_prefiltering=prefilter)
    up = r.upload(sc)
    out = [torch.empty(45 * 37 * 4, device="cuda") for _ in range(2)]
    for layout in (0, 1):
        up.set_tuning(layout, 4)
        up.render_device(opts, out[layout].data_ptr())
    torch.cuda.synchronize()
    n = spp[0] * spp[1] * (2 * math.ceil(radius) + 1) ** 2
    a, b = out[0].cpu().numpy(), out[1].cpu().numpy()
    up.close()
    r.close()
    assert float(np.max(np.abs(a - b))) <= n * 6e-8
