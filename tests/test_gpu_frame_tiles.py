"""Whole frames, which list their hits and shading rays where they have them at hand: with tiles
that leave a warp broken, whose lists have kernels of their own, the same bits as with
tiles of whole warps; around the size from which shading's list has its own kernel, the bits
of the same frames run stage by stage."""
import numpy as np
import pytest

from conftest import assert_records_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model, size", [("area", (77, 41)), ("point", (77, 41)), ("area", (1, 1)), ("area", (33, 130))])
def test_whole_frames_whatever_the_tile(lib, cuda_device, scene0, model, size):
    w, _ = scene0
    want = None
    for tile in ((16, 8), (10, 10), (5, 5), (33, 1), (1, 1), (7, 36), (8, 4)):
        v = lib.View(w, lib.view_desc(*size, lib.LIGHTS_POINT if model == "point" else lib.LIGHTS_AREA, accumulate=1,
                                      rng_seed=11, tile_x=tile[0], tile_y=tile[1]))
        try:
            for f in range(3):
                v.lookat((60.0 + 3 * f, 120.0, 40.0), (150.0, 60.0, 170.0))
                v.render()
            v.wait()
            got = (v.read_gbuffer(0), v.read_reservoirs(0), v.read_reservoirs(1), v.read_accum(), v.work_counts())
        finally:
            v.close()
        if want is None:
            want = got
            assert size == (1, 1) or 0 < min(got[4]) and max(got[4]) == got[4][0]
        for a, b, name in zip(got, want, ("G-buffer", "candidates", "reservoirs", "image")):
            assert_records_equal(name, a, b, f"[tile {tile}]")
        assert tuple(got[4]) == tuple(want[4])


@pytest.mark.parametrize("size", [(512, 512), (513, 512), (1021, 257)])
def test_whole_frames_around_the_request_line(lib, cuda_device, scene0, size):
    w, _ = scene0
    views = [lib.View(w, lib.view_desc(*size, lib.LIGHTS_AREA, accumulate=1, num_candidates=4, rng_seed=7)) for _ in range(2)]
    try:
        for f in range(2):
            for v in views:
                v.lookat((60.0 + 3 * f, 120.0, 40.0), (150.0, 60.0, 170.0))
            views[0].render()
            views[1].begin_frame()
            for s in (lib.STAGE_ALBEDO, lib.STAGE_CANDIDATES, lib.STAGE_SPATIAL, lib.STAGE_SHADE, lib.STAGE_ACCUMULATE):
                views[1].stage(s)
            views[1].end_frame()
        for v in views:
            v.wait()
        assert_records_equal("reservoirs", views[0].read_reservoirs(1), views[1].read_reservoirs(1))
        assert_records_equal("image", views[0].read_accum(), views[1].read_accum())
        assert tuple(views[0].work_counts()) == tuple(views[1].work_counts())
    finally:
        for v in views:
            v.close()
