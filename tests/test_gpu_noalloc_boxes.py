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


@pytest.mark.parametrize("pool", [1, 32769], ids=["boxes", "no boxes"])
def test_a_bad_grid_is_refused_and_draws_nothing(lib, cuda_device, scene0, pool):
    """A cell that points past the bricks: refused, the caller's image as it was, and the next
    call draws again."""
    torch = pytest.importorskip("torch")
    world, _ = scene0
    W, H = 77, 41
    g, b, l = world.arrays()
    n = max(len(b), pool)
    bricks = np.zeros((n, 512), np.uint32)
    bricks[:len(b)] = b.reshape(-1, 512)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32).reshape(-1).copy()).to("cuda")  # noqa: E731
    bad = g.copy()
    bad[np.nonzero(bad & 1)[0][0]] = (n << 1) | 1
    good, bad, bricks, lights = to(g), to(bad), to(bricks), to(l.view(np.uint32))
    out = torch.full((W * H * 4,), 7.0, dtype=torch.float32, device="cuda")
    cam = lib.Camera()
    cam.lookat((60.0, 120.0, 40.0), (150.0, 60.0, 170.0))
    k = cam.begin_frame(W, H)
    k.numberOfLights, k.numberOfCandidates, k.spatialRadius, k.spatialTaps, k.spatial = len(l), 32, 30, 5, 1
    L = lib.load()
    torch.cuda.synchronize()

    def draw(grid):
        return L.vxr_render_frame_noalloc(C.c_void_p(grid.data_ptr()), C.c_void_p(bricks.data_ptr()), n,
                                          C.c_void_p(lights.data_ptr()), len(l), lib.LIGHTS_AREA, C.byref(k),
                                          C.c_void_p(out.data_ptr()), None)
    assert draw(good) == 0, L.vxr_last_error().decode()
    first = out.clone()
    assert (first != 7.0).any()
    out.fill_(7.0)
    torch.cuda.synchronize()
    assert draw(bad) == lib.vxr.VXR_E_INVALID and b"brick" in L.vxr_last_error()
    assert bool((out == 7.0).all())
    assert draw(good) == 0
    assert torch.equal(out.view(torch.int32), first.view(torch.int32))
