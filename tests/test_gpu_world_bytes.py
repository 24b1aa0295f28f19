"""vxr_world_device_bytes: what the world's GPU copy holds."""
import pytest

pytestmark = pytest.mark.gpu

CELLS = 128 ** 3 * (4 + 2 * 8) + 32 ** 3 * (1 + 16 + 8)   # grid with two box tables, uber cells with two mask tables
BRICK = 512 * 4 + 2 * 4 + 2 * 64                          # voxels, boxes, masks of the opaque and the non-zero voxels
LIGHT = 16 + 2 * 16                                       # record, geometry, emission


@pytest.mark.parametrize("extent, emitters", [(64, 0), (256, 64), (512, 5000)])
def test_device_bytes_counts_every_table(lib, cuda_device, extent, emitters):
    import torch
    w = lib.World()
    try:
        w.generate(lib.scene_preset(0, extent=extent, emitters=emitters))
        _, bricks, lights = w.arrays()
        assert w.device_bytes() == 0
        torch.cuda.init()
        free = torch.cuda.mem_get_info()[0]
        w.upload()
        taken = free - torch.cuda.mem_get_info()[0]
        pool = len(bricks) + len(bricks) // 8 + 256           # the pool's headroom for later edits
        want = CELLS + pool * BRICK + max(1, len(lights)) * LIGHT
        assert w.device_bytes() == want
        # the driver hands memory out in blocks of 2 MB, small tables from blocks in part used
        assert abs(taken - want) <= 11 * (2 << 20)
        # an edit within the pool brings its staging buffer: 64 bricks and their indices
        w.set(1, 1, 1, 0xF123)
        assert w.commit()[1] is False
        assert w.device_bytes() == want + 64 * (512 * 4 + 4)
    finally:
        w.close()
