"""The split shadow DDA (GridWalk and its tasks, device.cuh) compiled for the CPU, against the
resumable walker: the same status, distance bits, side and visibility for every ray, tasks
finished at once or after the walk, with and without brick boxes and masks. The first-voxel trace over cell masks (trace_first)
against the three-level DDA it stands for. And the one-call
area-light candidate (area_candidate) against the sample and target functions it stands for."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import binding as ob
from test_device_code_host import (_candidate_shadow_rays, _f3, _rays, _surface_rays, brick_boxes, dh,  # noqa: F401
                                   uber_boxes0)

NATIVE = os.path.join(ROOT, "tests", "native")


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("split") / "libsplit.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math", "-w", "-I" + cuda,
                    "-I" + os.path.join(ROOT, "smallproject_gb300", "csrc"), os.path.join(NATIVE, "devhost_split.cpp"), "-o", so],
                   check=True)
    lib = C.CDLL(so)
    P, F = C.c_void_p, C.POINTER(C.c_float)
    lib.dh_shadow_split.argtypes = [P, P, P, P, P, F, F, C.c_uint32, C.c_uint32, C.c_int, C.c_int, C.POINTER(C.c_int), F,
                                    C.POINTER(C.c_uint32)]
    return lib


def uber_cells(grid, bricks, boxes):
    """World::ucell as the GPU builds it (build_uber_boxes_kernel); boxes None: every brick
    counts as one that can stop a ray."""
    g = grid.reshape(128, 128, 128)                                    # [y, z, x]
    brick = (g & 1) == 1
    stops = ~brick & ((((g >> 1) >> 12) & 15) == 15)
    stops[brick] = True if boxes is None else boxes[g[brick] >> 1] != 0xFFFFFFFF
    out = np.zeros((32, 32, 32, 2), np.uint32)                         # [uy, uz, ux]
    for b in range(64):
        s = stops[b >> 4::4, (b >> 2) & 3::4, b & 3::4].astype(np.uint32)
        out[..., b >> 5] |= s << np.uint32(b & 31)
    occupied = (g != 0).reshape(32, 4, 32, 4, 32, 4).any(axis=(1, 3, 5))
    out[..., 0] |= (occupied & ~out.any(axis=-1)).astype(np.uint32)
    return np.ascontiguousarray(out.reshape(-1, 2))


def uber_cells0(grid, bricks, boxed):
    """World::ucell0 and gbox0 as the GPU builds them (build_cells_kernel); boxed False: every
    brick counts as one that can stop a ray, and there is no gbox0."""
    g = grid.reshape(128, 128, 128)
    box = brick_boxes(bricks, nonzero=True)
    brick = (g & 1) == 1
    stops = g != 0
    if boxed:
        stops[brick] = box[g[brick] >> 1] != 0xFFFFFFFF
    out = np.zeros((32, 32, 32, 4), np.uint32)
    for b in range(64):
        s = stops[b >> 4::4, (b >> 2) & 3::4, b & 3::4].astype(np.uint32)
        out[..., b >> 5] |= s << np.uint32(b & 31)
    occupied = (g != 0).reshape(32, 4, 32, 4, 32, 4).any(axis=(1, 3, 5))
    out[..., 2] = uber_boxes0(grid, bricks).reshape(32, 32, 32)
    out[..., 0] |= (occupied & ~out[..., :2].any(axis=-1)).astype(np.uint32)
    gbox = np.stack([grid, np.where(grid & 1, box[np.where(grid & 1, grid >> 1, 0)], 0).astype(np.uint32)], 1) if boxed else None
    return np.ascontiguousarray(out.reshape(-1, 4)), gbox


def brick_masks(bricks, nonzero=False):
    """World::bmask (nonzero: bmask0) as the GPU builds it (build_brick_boxes_kernel)."""
    v = bricks.reshape(-1, 16, 32)
    op = v != 0 if nonzero else ((v >> 12) & 15) == 15
    return (op.astype(np.uint32) << np.arange(32, dtype=np.uint32)).sum(axis=2, dtype=np.uint32)


def _compare(dh, split, wa, O, D, pos, size, stepss):  # noqa: F811
    boxes, masks = brick_boxes(wa.bricks), brick_masks(wa.bricks)
    P = lambda a: a.ctypes.data  # noqa: E731
    hits = visible = 0
    stats = (C.c_int * 4)()
    for bx, mk in ((boxes, masks), (None, None)):
        uc = uber_cells(wa.grid, wa.bricks, bx)
        for i in range(len(O)):
            o, d, steps = _f3(O[i]), _f3(D[i]), int(stepss[i])
            da, sa, nv = C.c_float(0), C.c_uint32(0), C.c_int(0)
            st = dh.dh_walk_skip(P(wa.grid), P(wa.uber), P(wa.bricks), P(boxes), o, d, steps, C.byref(da), C.byref(sa),
                                 C.byref(nv))
            want = dh.dh_shadow(P(wa.grid), P(wa.uber), P(wa.bricks), P(boxes), o, d, int(pos[i]), int(size[i]), 0,
                                C.byref(nv)) if steps == 128 else None
            for deferred in (0, 1):
                db, sb = C.c_float(0), C.c_uint32(0)
                got = split.dh_shadow_split(P(wa.grid), P(wa.bricks), P(bx) if bx is not None else None, P(uc),
                                            P(mk) if mk is not None else None, o, d, int(pos[i]), int(size[i]), steps, deferred, stats, C.byref(db), C.byref(sb))
                assert (sb.value != 3) == (st == 1), (i, O[i], D[i], steps)
                assert np.float32(da.value).view(np.uint32) == np.float32(db.value).view(np.uint32), (i, O[i], D[i])
                assert st != 1 or sa.value == sb.value, (i, O[i], D[i])
                assert want is None or got == want, (i, O[i], D[i])
            hits += st == 1
            visible += bool(want)
    return hits, visible, list(stats)


def test_split_walk_matches_walker(dh, split, world0_arrays):  # noqa: F811
    """Rays through and past the map, axis-aligned ones among them, rays leaving the terrain,
    budgets from 1 to endless; the emitter is drawn at random (the hit decides) and a NaN
    direction ends as the walker's does."""
    wa = world0_arrays
    o1, d1, rng = _rays(2500, 77)
    o2, d2, _ = _surface_rays(wa, 2500, 78)
    o3 = np.tile(np.float32([[128.5, 200.5, 128.5]]), (3, 1))
    d3 = np.float32([[0, -1, 0], [np.nan, np.nan, np.nan], [np.inf, 0, 0]])
    O, D = np.concatenate([o1, o2, o3]), np.concatenate([d1, d2, d3])
    steps = rng.choice([128, 128, 128, 5000, 9, 5, 4, 1], len(O))
    li = rng.integers(0, len(wa.lights), len(O))
    hits, _, _ = _compare(dh, split, wa, O, D, wa.lights["position"][li], wa.lights["size"][li], steps)
    assert hits > 500


@pytest.mark.parametrize("point", [False, True])
def test_split_walk_matches_walker_on_candidate_rays(dh, split, world0_arrays, point):  # noqa: F811
    wa = world0_arrays
    O, D, LI = _candidate_shadow_rays(wa, wa.lights, 96, 54,
                                      lambda f: ((128.0 + 40.0 * f, 170.0, -60.0 + 30.0 * f), (128.0, 100.0, 128.0)), point)
    hits, visible, _ = _compare(dh, split, wa, O, D, wa.lights["position"][LI], wa.lights["size"][LI], np.full(len(O), 128))
    assert hits > 500 and visible > 100


def test_split_walk_finds_solid_cells(dh, split):  # noqa: F811
    """Brick-less cells: opaque ones stop a ray at their entry point, translucent ones do not
    (nor does an uber cell that holds nothing else, but its cells still cost budget)."""
    import smallproject_gb300 as vx
    w = vx.World()
    rng = np.random.default_rng(5)
    for b in rng.integers(0, 16, (160, 3)):
        w.add_brick(int(b[0]), int(b[1]), int(b[2]), 0xF123 if rng.random() < 0.5 else 0x8123)
    for b in rng.integers(0, 128, (400, 3)):
        w.set(int(b[0]), int(b[1]), int(b[2]), 0xFFFF if rng.random() < 0.7 else 0x7ABC)
    g, bricks, lights = w.arrays()
    wa = ob.WorldArrays(g, bricks, lights)
    O, D, rng = _rays(2500, 6, lo=-40.0, hi=170.0, inside=(0.0, 128.0))
    n = len(O)
    hits, _, _ = _compare(dh, split, wa, O, D, rng.integers(0, 1 << 30, n), rng.choice([1, 8], n),
                          rng.choice([128, 30, 9], n))
    assert hits > 300


def _compare_reach(dh, split, wa, O, D, pos, size):  # noqa: F811
    """Rays shadow_can_reach rules out are occluded for the walker; returns (rays, ruled out,
    visible)."""
    boxes = brick_boxes(wa.bricks)
    P = lambda a: a.ctypes.data  # noqa: E731
    split.dh_can_reach.argtypes = [C.c_void_p, C.POINTER(C.c_float), C.POINTER(C.c_float), C.c_uint32, C.c_uint32, C.c_int]
    nv, out, visible = C.c_int(0), 0, 0
    for i in range(len(O)):
        o, d = _f3(O[i]), _f3(D[i])
        can = split.dh_can_reach(P(wa.uber), o, d, int(pos[i]), int(size[i]), 128)
        if not can or i % 4 == 0:
            v = dh.dh_shadow(P(wa.grid), P(wa.uber), P(wa.bricks), P(boxes), o, d, int(pos[i]), int(size[i]), 0, C.byref(nv))
            assert can or not v, (i, O[i], D[i], pos[i], size[i])
            visible += v
        out += not can
    return len(O), out, visible


def test_rays_out_of_reach_are_occluded(dh, split):  # noqa: F811
    """Candidate shadow rays of the 1,024-voxel benchmark scene, and the same rays pointed at
    other emitters and at solid ones of 8 voxels; axis-aligned rays, rays from outside the map
    and of numbers that are not finite are left to the walk."""
    hs = ob.HostScene(3)
    wa = ob.WorldArrays(hs.grid, hs.bricks, hs.lights)
    O, D, LI = _candidate_shadow_rays(wa, hs.lights, 112, 63, lambda f: hs.camera_path(1, 150 + f, 300), False)
    pos, size = hs.lights["position"], hs.lights["size"]
    n, out, visible = _compare_reach(dh, split, wa, O, D, pos[LI], size[LI])
    assert out > 0.1 * n and visible > 100
    rng = np.random.default_rng(4)
    li = rng.integers(0, len(pos), len(O))
    to = np.stack([pos[li] % 1024, pos[li] // 1048576, (pos[li] // 1024) % 1024], 1).astype(np.float32) + np.float32(0.5)
    size = np.where(rng.random(len(O)) < 0.3, 8, 1)
    D2 = to - O
    D2 = (D2 / np.linalg.norm(D2, axis=1, keepdims=True)).astype(np.float32)
    D2[::9] = D[::9]                                     # a ray that does not head for its emitter
    D2[1::50, 0] = 0.0
    D2[2::50] = np.nan
    O[3::50] -= 2000.0
    n, out, _ = _compare_reach(dh, split, wa, O, D2, pos[li], size)
    assert out > 0.1 * n


def _compare_first(dh, split, wa, O, D, stepss):  # noqa: F811
    P = lambda a: a.ctypes.data if a is not None else None  # noqa: E731
    split.dh_trace_first.restype = C.c_uint32
    split.dh_trace_first.argtypes = [C.c_void_p] * 6 + [C.POINTER(C.c_float)] * 2 + [C.c_int, C.c_int, C.POINTER(C.c_float),
                                                                                     C.POINTER(C.c_uint32)]
    hits = 0
    for boxed, bits in ((True, None), (False, None), (True, brick_masks(wa.bricks, nonzero=True))):
        uc, gb = uber_cells0(wa.grid, wa.bricks, boxed)
        for i in range(len(O)):
            o, d, steps = _f3(O[i]), _f3(D[i]), int(stepss[i])
            da, sa, db, sb = C.c_float(0), C.c_uint32(0), C.c_float(0), C.c_uint32(0)
            a = dh.dh_trace(0, P(wa.grid), P(wa.uber), P(wa.bricks), o, d, steps, 0, 0, C.byref(da), C.byref(sa))
            b = split.dh_trace_first(P(wa.grid), P(wa.uber), P(wa.bricks), P(uc), P(gb), P(bits), o, d, int(steps < 999999), steps, C.byref(db),
                                     C.byref(sb))
            assert (a, sa.value) == (b, sb.value) and \
                np.float32(da.value).view(np.uint32) == np.float32(db.value).view(np.uint32), (i, O[i], D[i], steps)
            hits += a != 0
    return hits


def test_trace_first_matches_trace(dh, split, world0_arrays):  # noqa: F811
    """Terrain with emitters: rays from inside and outside the map, leaving the surface, axis
    aligned and of numbers that are not finite, endless and with budgets down to one step."""
    wa = world0_arrays
    o1, d1, rng = _rays(2500, 91)
    o2, d2, _ = _surface_rays(wa, 1500, 92)
    n, i = np.nan, np.inf
    d3 = np.float32([[0, -1, 0], [n, n, n], [i, 0, 0], [n, 0, -1], [i, n, n], [0, i, 0], [0.6, n, 0.8], [0, 0, 0]])
    o3 = np.tile(np.float32([[128.5, 200.5, 128.5]]), (len(d3), 1))
    o4, d4 = np.float32([[n, n, n], [i, 5, 5], [-i, i, n], [5, 5, -1e35]]), np.tile(np.float32([[0.6, 0, 0.8]]), (4, 1))
    O, D = np.concatenate([o1, o2, o3, o4]), np.concatenate([d1, d2, d3, d4])
    steps = rng.choice([999999, 999999, 128, 128, 9, 5, 4, 1], len(O))
    steps[-12:] = 999999
    assert _compare_first(dh, split, wa, O, D, steps) > 1500


def _compare_opaque(dh, split, wa, O, D, stepss):  # noqa: F811
    P = lambda a: a.ctypes.data  # noqa: E731
    split.dh_trace_opaque.restype = C.c_uint32
    split.dh_trace_opaque.argtypes = [C.c_void_p] * 6 + [C.POINTER(C.c_float)] * 2 + [C.c_int, C.POINTER(C.c_float), C.POINTER(C.c_uint32)]
    boxes, masks = brick_boxes(wa.bricks), brick_masks(wa.bricks)
    uc = uber_cells(wa.grid, wa.bricks, boxes)
    gb = np.stack([wa.grid, np.where(wa.grid & 1, boxes[np.where(wa.grid & 1, wa.grid >> 1, 0)], 0).astype(np.uint32)], 1)
    hits = 0
    for i in range(len(O)):
        o, d, steps = _f3(O[i]), _f3(D[i]), int(stepss[i])
        da, sa, db, sb = C.c_float(0), C.c_uint32(0), C.c_float(0), C.c_uint32(0)
        a = dh.dh_trace(1, P(wa.grid), P(wa.uber), P(wa.bricks), o, d, steps, 0, 0, C.byref(da), C.byref(sa))
        b = split.dh_trace_opaque(P(wa.grid), P(wa.uber), P(wa.bricks), P(uc), P(gb), P(masks), o, d, steps, C.byref(db), C.byref(sb))
        assert a == b, (i, O[i], D[i], steps)
        if a:
            assert sa.value == sb.value and np.float32(da.value).view(np.uint32) == np.float32(db.value).view(np.uint32), (i, O[i])
        hits += a != 0
    return hits


def test_opaque_trace_over_masks_matches_trace(dh, split, world0_arrays):  # noqa: F811
    """The sky light's ray: terrain, from inside and outside the map and leaving the surface, with
    its budget of 10, smaller and larger ones; numbers that are not finite."""
    wa = world0_arrays
    o1, d1, rng = _rays(1500, 95)
    o2, d2, _ = _surface_rays(wa, 2500, 96)
    n, i = np.nan, np.inf
    d3 = np.float32([[0, -1, 0], [n, n, n], [i, 0, 0], [n, 0, -1], [0.6, n, 0.8], [0, 0, 0]])
    o3 = np.tile(np.float32([[128.5, 200.5, 128.5]]), (len(d3), 1))
    O, D = np.concatenate([o1, o2, o3]), np.concatenate([d1, d2, d3])
    steps = rng.choice([10, 10, 128, 9, 5, 4, 1], len(O))
    assert _compare_opaque(dh, split, wa, O, D, steps) > 300


def test_trace_first_matches_trace_on_solid_cells(dh, split):  # noqa: F811
    """Brick-less cells, bricks without a non-zero voxel, single voxels in the air."""
    import smallproject_gb300 as vx
    w = vx.World()
    rng = np.random.default_rng(8)
    for b in rng.integers(0, 16, (160, 3)):
        w.add_brick(int(b[0]), int(b[1]), int(b[2]), 0xF123 if rng.random() < 0.5 else 0x8123)
    for k, b in enumerate(rng.integers(0, 128, (400, 3))):
        w.set(int(b[0]), int(b[1]), int(b[2]), 0xFFFF)
        if k % 3 == 0:
            w.set(int(b[0]), int(b[1]), int(b[2]), 0)
    g, bricks, lights = w.arrays()
    wa = ob.WorldArrays(g, bricks, lights)
    O, D, rng = _rays(2500, 16, lo=-40.0, hi=170.0, inside=(0.0, 128.0))
    assert _compare_first(dh, split, wa, O, D, rng.choice([999999, 128, 30, 9], len(O))) > 800


def test_area_candidate_matches_sample_and_target(split):
    """Wherever area_candidate answers, it gives the draws and the target value of
    sample_area_light and phat bit for bit, and with a non-zero target the same point, weight
    and face; it answers for nearly every ordinary candidate. Shading points far and near,
    on face planes and inside the cube; huge and zero sizes, black and non-finite emission,
    an RNG state of zero, points at infinity."""
    rng = np.random.default_rng(17)
    P = C.POINTER(C.c_float)
    split.dh_area_candidate.argtypes = [P, C.c_uint32, C.c_uint32, P]
    out = np.zeros((2, 7), np.float32)
    answered = ordinary = lit = 0
    for i in range(60000):
        size = np.float32(rng.choice([1.0, 1.0, 8.0]))
        c = np.floor(rng.uniform(0, 1000, 3)).astype(np.float32) + np.float32(0.5) * size
        mode = i % 6
        sp = rng.uniform(0, 1024, 3) if mode < 3 else c + rng.normal(0, 3 * size, 3)
        if mode == 4:      # inside slabs, on face planes
            sp = c + np.where(rng.random(3) < 0.5, rng.choice([-0.5, 0.5, 0.25], 3) * size, rng.normal(0, 9, 3))
        em, brdf = rng.uniform(0, 30, 3), rng.uniform(0, 0.32, 3)
        side, sign, seed = int(rng.integers(3)), float(rng.choice([-1.0, 1.0])), int(rng.integers(1, 2 ** 32))
        if mode == 5:
            k = i // 6 % 7
            if k == 0: size = np.float32(rng.choice([0.0, 3.0, 5e5, 4e9]))   # noqa: E701
            if k == 1: em = em * rng.choice([0.0, np.inf, np.nan, 1e30])     # noqa: E701
            if k == 2: brdf = brdf * rng.choice([0.0, 1e-25, 1e25])          # noqa: E701
            if k == 3: seed = 0                                              # noqa: E701
            if k == 4: sp[int(rng.integers(3))] = rng.choice([np.inf, -np.inf, np.nan, 1e9])   # noqa: E701
            if k == 5: sp = c.copy()                                         # noqa: E701
        sp = sp.astype(np.float32)
        spo = sp.copy()
        spo[side] += np.float32(0.1) * np.float32(sign)
        args = np.concatenate([c, [size], em, sp, spo, [sign], brdf]).astype(np.float32)
        ok = split.dh_area_candidate(args.ctypes.data_as(P), side, seed, out.ctypes.data_as(P))
        a, b = out.view(np.uint32)
        if ok:
            assert a[0] == b[0] and a[1] == b[1], (i, args, out)
            assert out[0, 0] == 0.0 or (a[2:] == b[2:]).all(), (i, args, out)
        answered += ok and mode < 3
        ordinary += mode < 3
        lit += bool(ok and out[0, 0] > 0)
    assert answered > 0.999 * ordinary and lit > 10000
