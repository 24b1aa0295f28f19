"""vxr_render_frame_noalloc on both sides of the brick count up to which it makes brick boxes
in its scratch (32,768): the same pixels as a view, for both light models."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("point", [False, True], ids=["area", "point"])
def test_noalloc_with_and_without_boxes(lib, cuda_device, scene0, point):
    torch = pytest.importorskip("torch")
    world, _ = scene0
    W, H = 77, 41
    g, b, l = world.arrays()
    bricks = np.zeros((32769, 512), np.uint32)   # a pool of more bricks than the grid refers to
    bricks[:len(b)] = b.reshape(-1, 512)
    dev = [torch.from_numpy(np.ascontiguousarray(a).view(np.int32).reshape(-1).copy()).to("cuda")
           for a in (g, bricks, l.view(np.uint32))]
    out = torch.zeros(W * H * 4, dtype=torch.float32, device="cuda")
    model = lib.LIGHTS_POINT if point else lib.LIGHTS_AREA
    view = lib.View(world, lib.view_desc(W, H, model, temporal=0, accumulate=0))
    L = lib.load()
    try:
        view.lookat((60.0, 120.0, 40.0), (150.0, 60.0, 170.0))
        k = view.begin_frame()
        for s in (lib.STAGE_ALBEDO, lib.STAGE_CANDIDATES, lib.STAGE_SPATIAL, lib.STAGE_SHADE):
            view.stage(s)
        view.end_frame()
        view.wait()
        want = view.read_frame()
        assert (want[:, :3] > 0).any()
        for n in (len(b), 32768, 32769):
            out.zero_()
            torch.cuda.synchronize()
            rc = L.vxr_render_frame_noalloc(*(C.c_void_p(t.data_ptr()) for t in dev[:2]), n, C.c_void_p(dev[2].data_ptr()), len(l),
                                            model, C.byref(k), C.c_void_p(out.data_ptr()), None)
            assert rc == 0, L.vxr_last_error().decode()
            got = out.cpu().numpy().reshape(-1, 4)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), n
    finally:
        view.close()
