"""The candidate pass of worlds with 32,768 emitters and more, which asks for no ray that
cannot reach its emitter: every stage bit for bit with the oracle on both sides of the line,
at image sizes that are no multiple of a warp, with both light models."""
import numpy as np
import pytest

from oracle import binding as ob
from test_gpu_parity import _run_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emitters, point, size", [(32767, False, (77, 41)), (32768, False, (77, 41)), (40000, True, (77, 41)),
                                                   (40000, False, (160, 90)), (40000, False, (1, 1))])
def test_stages_around_the_line(lib, cuda_device, emitters, point, size):
    w = lib.World()
    try:
        d = lib.scene_preset(3, emitters=emitters)   # blobs of emitters in a 1024^3 world
        w.generate(d)
        g, b, l = w.arrays()
        assert len(l) == emitters
        _run_parity(lib, (w, d), ob.WorldArrays(g, b, l), *size, point, 3, lambda f: lib.camera_path(d, 1, 60 + f, 120))
    finally:
        w.close()


def test_decided_rays_are_counted(lib, cuda_device):
    """work_counts counts the rays that the candidate pass decides as well as the traced ones."""
    w = lib.World()
    d = lib.scene_preset(3, emitters=40000)
    w.generate(d)
    v = lib.View(w, lib.view_desc(320, 180, lib.LIGHTS_AREA, temporal=0, spatial=0, accumulate=0))
    try:
        v.lookat(*lib.camera_path(d, 1, 60, 120))
        v.render()
        v.wait()
        hits, rays, _ = v.work_counts()
        # a pixel whose reservoir holds an emitter asked for its ray, visible or not
        held = v.read_reservoirs(0)
        assert 0 < np.count_nonzero(held["pHat"] > 0) <= rays <= hits
    finally:
        v.close()
        w.close()
