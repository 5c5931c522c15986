"""Sizes and index arithmetic at limits that no test can reach on a device."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ORACLE = os.path.join(os.path.dirname(HERE), "oracle")


@pytest.fixture(scope="module")
def limits():
    subprocess.run(["make", "-s", "-C", ORACLE], check=True)
    return C.CDLL(os.path.join(ORACLE, "_build", "liblimits.so"))


@pytest.mark.parametrize("radii", [[1], [8], [9], [1, 3, 8], [9, 1], [1, 9, 3], [40, 8, 200], [0], [9, 0, 9]])
def test_splat_room_for_every_scene(limits, radii):
    """A batch's scenes whose own radius fits accumulate in shared memory, so there has to be room
    for the largest of them next to any that does not fit; the lane-group splat needs all to fit."""
    f = limits.limits_splat
    f.restype = C.c_size_t
    all_fit = C.c_int()
    got = f((C.c_int * len(radii))(*radii), len(radii), C.byref(all_fit))
    need = max([(16 + 2 * r) ** 2 * 20 for r in radii if r <= 8], default=0)
    assert got == need
    assert bool(all_fit.value) == all(r <= 8 for r in radii)


def test_place_in_the_tile_list(limits):
    """Cell entries keep their group's place next to eight flags; a walk over a longer tile list than
    that leaves room for has to give its own step (2^23 shifted by eight is negative)."""
    top = limits.limits_cell_list_max()
    for place in (0, 1, 32767, top - 1):
        for flags in (0, 1, 20, 255):
            assert limits.limits_place(1, place, flags) == place
    for place in (0, top, (1 << 23) - 1, 1 << 23, 9_000_000, (1 << 24) + 5, (1 << 31) - 1):
        assert limits.limits_place(0, place, 20) == place


@pytest.mark.parametrize("tiles, groups", [(512 * 512, 1025), (256 * 256, 4100), (1024, 1 << 21), (64, 3), (1, 0)])
def test_room_is_given_once(limits, tiles, groups):
    """Scenes whose cell entries (16 per tile and group) or items pass 2^32: canvases of 8192 and 4096
    pixels full of groups.  Only the room there is is given, and none of it twice."""
    f = limits.limits_room
    f.argtypes, f.restype = [C.c_longlong, C.c_int, C.c_int], C.c_longlong
    for cap in (1 << 30, (1 << 31) - 1, 1000, 0):
        need = 16 * groups
        assert f(tiles, need, cap) == (min(tiles, cap // need) if need else tiles)


@pytest.mark.parametrize("tiles, entries", [(0, 0), (1, 0), (16, 40), (4096, 110_700), (16384, 16_400_000),
                                            (262144, 1 << 31)])
def test_cell_list_memory_within_its_limit(limits, tiles, entries):
    """1,000 canvas-wide groups at 2048x2048 wanted 21 GB for lists that are an optimisation."""
    f = limits.limits_cell_room
    f.argtypes, f.restype = [C.c_uint64] * 4 + [C.c_void_p], None
    want = (min(max(entries, 1) * 16, 1 << 30), min(max(48 * entries, 1), 1 << 30))
    for budget in (0, 1, 1000, 1 << 16, 1 << 20, 1 << 30, 4 << 30, 1 << 40):
        out = (C.c_uint64 * 6)()
        f(tiles, entries, 48 * entries, budget, out)
        ents, items, at_ents, at_items, at_counters, total = out
        if total == 0:
            assert tiles == 0 or budget < tiles * 128 + 1000
            continue
        assert total <= budget and 1 <= ents <= want[0] and 1 <= items <= want[1]
        assert at_ents >= tiles * 128 and at_ents % 16 == 0
        assert at_items >= at_ents + ents * 32 and at_counters >= at_items + items * 16 and at_counters % 8 == 0
        assert total >= at_counters + 16
        if budget == 1 << 40:
            assert (ents, items) == want


def test_steps_of_an_entry(limits):
    """The count that makes a cell heavy (from 24 steps): a primitive's edge, marked by 63 in the place of
    a number of segments, does so by itself and no more than that."""
    assert limits.limits_entry_steps(2, 3, 4, 5) == 14
    assert limits.limits_entry_steps(0, 0, 63, 0) == 24
    assert limits.limits_entry_steps(0, 0, 48, 2) == 50


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [(2, 2), (4, 4), (3, 2)])
@pytest.mark.parametrize("prefilter", [False, True])
@pytest.mark.parametrize("work_queue", [0, 1])
def test_batch_of_mixed_filter_radii(work_queue, prefilter, spp):
    """Radii on both sides of what shared memory holds in one batch, against single renders."""
    import numpy as np
    from dvg import Batch, Renderer, RenderOptions, synth
    from dvg.scene import Filter, FilterType

    scenes = []
    for i, r in enumerate((0.5, 9.5, 2.5)):
        sc = synth.plain_scene(i, 40 + 3 * i, 33, 4)
        sc.filter = Filter(FilterType.GAUSSIAN, r)
        scenes.append(sc)
    opts = RenderOptions(samples_x=spp[0], samples_y=spp[1], seed=3, jitter=True, use_prefiltering=prefilter)
    rn = Renderer(0)
    ups = [rn.upload(s) for s in scenes]
    b = Batch(rn, ups, opts)
    b.set_tuning(1, 4, 16, work_queue)
    b.step(use_graph=False)
    b.losses()  # waits
    for i, s in enumerate(scenes):
        img = b.buffers(i)[0].cpu().numpy().reshape(s.height, s.width, 4)
        assert float(np.max(np.abs(img - rn.render(s, opts).pixels))) <= 1e-5
    b.close()
    rn.close()
