"""The candidate pass of worlds with 32,768 emitters and more, which asks for no ray that
cannot reach its emitter: every stage bit for bit with the oracle on both sides of the line,
at image sizes that are no multiple of a warp, with both light models."""
import numpy as np
import pytest

from conftest import assert_records_equal
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
    """work_counts counts the rays that the candidate pass decides as well as the traced ones; a
    whole frame, whose primary rays list the hits, is the one of the stages."""
    w = lib.World()
    d = lib.scene_preset(3, emitters=40000)
    w.generate(d)
    v, staged = (lib.View(w, lib.view_desc(320, 180, lib.LIGHTS_AREA, temporal=0, spatial=0, accumulate=0)) for _ in range(2))
    try:
        v.lookat(*lib.camera_path(d, 1, 60, 120))
        v.render()
        v.wait()
        hits, rays, _ = v.work_counts()
        # a pixel whose reservoir holds an emitter asked for its ray, visible or not
        held = v.read_reservoirs(0)
        assert 0 < np.count_nonzero(held["pHat"] > 0) <= rays <= hits
        staged.lookat(*lib.camera_path(d, 1, 60, 120))
        staged.begin_frame()
        for s in (lib.STAGE_ALBEDO, lib.STAGE_CANDIDATES, lib.STAGE_SPATIAL, lib.STAGE_SHADE):
            staged.stage(s)
        staged.end_frame()
        staged.wait()
        assert_records_equal("candidates", v.read_reservoirs(0), staged.read_reservoirs(0))
        assert_records_equal("frame", v.read_frame(), staged.read_frame())
    finally:
        v.close()
        staged.close()
        w.close()


@pytest.mark.parametrize("candidates, tile", [(15, (16, 8)), (16, (16, 16)), (31, (32, 4)), (32, (10, 10)), (32, (16, 8)), (33, (16, 8))])
def test_candidates_behind_the_surface(lib, cuda_device, candidates, tile):
    """Most emitters below the visible faces (a layer under the terrain): the candidate pass works
    out those in front alone. Reservoirs and random states as the oracle's, below, at and above
    the candidate counts it scans, with tiles of whole and of broken warps."""
    w = lib.World()
    d = lib.scene_preset(4, extent=256, emitters=40000)
    w.generate(d)
    g, b, l = w.arrays()
    assert len(l) == 40000
    W, H = 77, 41
    view = lib.View(w, lib.view_desc(W, H, lib.LIGHTS_AREA, accumulate=0, spatial=0, temporal=0, num_candidates=candidates,
                                     tile_x=tile[0], tile_y=tile[1]))
    port = ob.Renderer("port", ob.WorldArrays(g, b, l), W, H, False)
    try:
        for f in range(2):
            view.lookat(*lib.camera_path(d, 1, 60 + f, 120))
            k = view.begin_frame()
            assert k.numberOfCandidates == candidates
            port.frame_start()
            for s in (1, 2):
                view.stage(s)
                port.stage(k, s)
            hits = np.count_nonzero(port.gbuffer(0)["voxel"])
            assert view.work_counts()[0] == hits
            assert (view.read_gbuffer(0)["voxel"] != 0).mean() > 0.2
            assert_records_equal("candidates", view.read_reservoirs(0), port.reservoirs(0), f"[frame {f}]")
            assert_records_equal("seed", view.read_gbuffer(0)["seed"], port.gbuffer(0)["seed"], f"[frame {f}]")
            view.end_frame()
            view.wait()
    finally:
        port.close()
        view.close()
        w.close()
