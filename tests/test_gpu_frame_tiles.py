"""Whole frames with tiles that leave a warp broken, which list their hits and shading rays in
kernels of their own: the same bits as tiles of whole warps, over three frames with reuse."""
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
