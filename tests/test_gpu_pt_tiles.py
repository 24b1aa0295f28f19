"""The path tracer deals a block's second rays out again by the axis of the face they leave:
the same image with tiles of whole warps, of broken ones (which do not), of one warp, and with
resident blocks, at sizes that are no multiple of any."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(77, 41), (33, 7), (1, 1)])
def test_path_tracer_whatever_the_tile(lib, cuda_device, scene0, size):
    w, _ = scene0
    images = []
    for tile, persistent in (((10, 10), 0), ((16, 8), 0), ((16, 16), 0), ((8, 4), 0), ((16, 8), 1)):
        v = lib.View(w, lib.view_desc(*size, lib.LIGHTS_AREA, tile_x=tile[0], tile_y=tile[1]))
        try:
            if persistent:
                v.set_tuning(lib.tuning(persistent=1))
            v.lookat((60.0, 120.0, 40.0), (150.0, 60.0, 170.0))
            frames = []
            for _ in range(2):
                v.begin_frame()
                v.stage(lib.STAGE_PATH_TRACE)
                frames.append(v.read_frame())
                v.end_frame()
                v.wait()
            images.append(np.stack(frames))
        finally:
            v.close()
    if size != (1, 1):
        assert (images[0][..., 3] < 1e19).any()
    for im in images[1:]:
        assert np.array_equal(im.view(np.uint32), images[0].view(np.uint32))
