"""Who takes which device error flag: a call that reports one leaves the others to be reported,
and frames in flight keep theirs. Flags are raised without a fault: a reservoir that names an
emitter beyond the list (2 in the temporal pass, 8 in shading), tensor-core waits that run
out by the test hook (16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cam(f):
    return (128.0 + 4.0 * f, 160.0, 10.0 + f), (128.0, 120.0, 128.0)


def _learned(lib, W=96, H=64):
    w = lib.World()
    w.generate(lib.scene_preset(0, emitters=2048, emitter_mode=1))
    w.cluster_lights(256, seed=3, iters=6)
    v = lib.View(w, lib.view_desc(W, H, lib.LIGHTS_AREA, num_candidates=8))
    v.proposal_enable(seed=7, batch=4096, inference=2)
    v.proposal_use(True)
    return w, v


def _name_missing_emitter(v, role, n):
    h = v.read_reservoirs(role)
    live = (h["streamLength"] > 0) & (h["sumOfWeights"] > 0) & (h["pHat"] > 0)
    assert live.sum() > 10
    h["lightIndex"][live] = n + 7
    v.write_reservoirs(role, h)


def test_probs_take_their_own_flag_alone(lib, cuda_device):
    w, v = _learned(lib)
    try:
        v.lookat(*_cam(0))
        v.render()
        v.wait()
        v.proposal_test_timeout(True)
        v.lookat(*_cam(1))
        v.begin_frame()
        for s in (lib.STAGE_ALBEDO, lib.STAGE_CANDIDATES):       # raises 16
            v.stage(s)
        v.proposal_test_timeout(False)
        v.stage(lib.STAGE_SPATIAL)
        _name_missing_emitter(v, 1, len(w.arrays()[2]))
        v.stage(lib.STAGE_SHADE)                                 # raises 8
        v.end_frame()
        with pytest.raises(lib.VxrError, match="tensor-core wait gave up"):
            v.proposal_probs(np.zeros((16, 4), np.float32))
        with pytest.raises(lib.VxrError, match=r"device error flags 0x8 \("):
            v.wait()
        v.wait()
        v.proposal_probs(np.zeros((16, 4), np.float32))
    finally:
        v.close()
        w.close()


def test_pipelined_images_report_each_time(lib, cuda_device):
    """A flag is reported with the first image waited for, for all frames enqueued by then; one
    that later frames raise is reported again."""
    w, v = _learned(lib)
    bufs = [lib.PinnedBuffer(96 * 64 * 4) for _ in range(3)]
    try:
        for turn in range(3):
            v.proposal_test_timeout(True)
            t = [v.render_to_host_async(*_cam(3 * turn + i), bufs[i].array) for i in range(3)]
            with pytest.raises(lib.VxrError, match=r"device error flags 0x10 \("):
                v.image_wait(t[0])
            for x in t[1:]:
                v.image_wait(x)
            v.proposal_test_timeout(False)
            for i in range(3):
                v.image_wait(v.render_to_host_async(*_cam(3 * turn + i), bufs[i].array))
            assert np.isfinite(bufs[2].array).all()
    finally:
        v.close()
        w.close()
        for b in bufs:
            b.close()


def test_batch_reports_the_flags_of_its_views(lib, cuda_device, scene0):
    w, _ = scene0
    views = [lib.View(w, lib.view_desc(64, 48, lib.LIGHTS_AREA, rng_seed=3 + i)) for i in range(2)]
    batch = lib.Batch(views, graph=True)

    def frame(f):
        for v in views:
            v.lookat(*_cam(f))
        batch.render()

    try:
        frame(0)
        batch.wait()
        _name_missing_emitter(views[1], 1, len(w.arrays()[2]))
        frame(1)
        with pytest.raises(lib.VxrError, match=r"device error flags 0x[2-9a-f] \("):
            batch.wait()
        for v in views:
            v.wait()                                             # reported once
        # (the index stays in the history that the next temporal pass reads: empty it)
        views[1].write_reservoirs(1, np.zeros_like(views[1].read_reservoirs(1)))
        frame(2)
        batch.wait()
    finally:
        batch.close()
        for v in views:
            v.close()
