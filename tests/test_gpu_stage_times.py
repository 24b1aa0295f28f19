"""Stage times: vxr_view_stage_times answers for the last waited frame whatever ran since, and
no frame pays for the times of those before it."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RING = 256   # frames whose stage events a view keeps


def _frame(v, f):
    v.lookat((110.0 + f % 7, 150.0, 10.0), (128.0, 120.0, 128.0))
    v.render()


def test_stage_times_stay_those_of_the_waited_frame(lib, cuda_device, scene0):
    w, _ = scene0
    v = lib.View(w, lib.view_desc(1280, 720, lib.LIGHTS_AREA, num_candidates=64))
    try:
        for f in range(3):
            _frame(v, f)
            v.wait()
        long = v.stage_times()[1]                 # 64 candidates (the scene's emitters)
        _frame(v, 3)
        v.wait()                                  # the last waited frame
        v.set_params(lib.view_desc(1280, 720, lib.LIGHTS_AREA, num_candidates=1))
        for f in range(200):
            _frame(v, f)
        v.stage_stats()                           # waits for the view, and is no vxr_view_wait
        for f in range(RING):                     # every ring entry taken again
            _frame(v, f)
        assert v.stage_times()[1] > 0.5 * long
        v.wait()
        assert 0.0 < v.stage_times()[1] < 0.5 * long   # one candidate
    finally:
        v.close()


def test_stage_times_of_a_frame_in_progress(lib, cuda_device, scene0):
    w, _ = scene0
    v = lib.View(w, lib.view_desc(160, 90, lib.LIGHTS_AREA))
    try:
        _frame(v, 0)
        v.wait()
        v.begin_frame()
        v.stage(lib.STAGE_ALBEDO)
        v.wait()
        t = v.stage_times()
        assert t[0] > 0.0 and not any(t[1:])      # only what this frame ran
        v.stage(lib.STAGE_CANDIDATES)
        v.end_frame()
        v.wait()
        t = v.stage_times()
        assert t[0] > 0.0 and t[1] > 0.0 and not any(t[2:])
        sums, counts = v.stage_stats(reset=True)
        assert list(counts[:3]) == [2, 2, 1] and sums[0] >= t[0]
        v.wait()                                  # nothing new
        assert list(v.stage_times()) == list(t)
    finally:
        v.close()


def test_no_frame_pays_for_the_times_of_others(lib, cuda_device, scene0):
    """The host time of the frames that take a ring entry anew, at every turn of the ring,
    against the median frame's: twice is far above what one frame's few queries cost and below
    a thousand of them."""
    w, _ = scene0
    v = lib.View(w, lib.view_desc(64, 48, lib.LIGHTS_AREA))
    try:
        t = np.zeros(4 * RING + 1)
        for f in range(len(t)):
            v.lookat((110.0, 150.0, 10.0), (128.0, 120.0, 128.0))
            t0 = time.perf_counter()
            v.render()
            t[f] = time.perf_counter() - t0
            v.wait()
        assert t[RING::RING].min() <= 2.0 * np.median(t)
    finally:
        v.close()


def test_stage_stats_keep_the_last_frames_between_waits(lib, cuda_device, scene0):
    """300 frames, a wait, 300 frames: of either the last 256 count, whoever harvests them; frames
    that end otherwise (begun and dropped, without stages) leave nothing behind."""
    w, _ = scene0
    v = lib.View(w, lib.view_desc(64, 48, lib.LIGHTS_AREA))
    try:
        for f in range(300):
            _frame(v, f)
        v.wait()
        for f in range(300):
            _frame(v, f)
        _, counts = v.stage_stats(reset=True)
        assert list(counts) == [2 * RING] * 4 + [0]
        v.begin_frame()
        v.stage(lib.STAGE_ALBEDO)
        v.begin_frame()                           # the frame before is dropped
        v.end_frame()
        v.wait()
        assert not any(v.stage_times())
        assert not any(v.stage_stats()[1])
    finally:
        v.close()
