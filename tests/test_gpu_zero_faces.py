"""Rays that end on a face at coordinate zero, coming down the axis (a floor
whose top is z = 0): the same answers as the oracle's, zeros' signs included,
from one search like any other face."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import MISS, same_points

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def vg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as m
    return m


def _floor(axis, top, side=128, depth=6, seed=3):
    """A slab of cells below `top` on `axis`, with holes."""
    r = np.random.RandomState(seed)
    cells = np.argwhere(r.random_sample((side, side, depth)) < 0.7).astype(np.float32)
    cells[:, 2] += top - depth
    return np.ascontiguousarray(np.roll(cells, axis - 2, axis=1))


def _rays(axis, top, n, side=128, seed=4):
    """Rays from above the slab, at its whole area."""
    r = np.random.RandomState(seed)
    o = np.concatenate([side * r.random_sample((n, 2)) * 1.4 - 0.2 * side, np.full((n, 1), 90.0 + top)], 1)
    to = np.concatenate([side * r.random_sample((n, 2)), np.full((n, 1), float(top))], 1)
    return tuple(np.ascontiguousarray(np.roll(x, axis - 2, axis=1).astype(np.float32)) for x in (o, to - o))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("zero", [0.0, -0.0])
def test_points_on_zero_faces(vg, axis, zero):
    vox = _floor(axis, 0)
    vox[vox == 0] = zero
    ht = vg.HostTree.from_voxels(vox)
    o, d = _rays(axis, 0, 20000)
    o[::3, axis - 1] = zero          # and points with a zero that comes from the origin
    d[::3, axis - 1] = 1e-9
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    assert ((opts[:, axis] == 0) & (oleaf != MISS)).mean() > 0.2
    for dt in (vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)):
        leaf, slot, pts = dt.rays(o, d)
        assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
        ok, bad = same_points(pts, opts, leaf != MISS)
        assert ok, f"{bad} points differ"


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_zero_faces_cost_what_others_do(vg, axis):
    """A frame of the slab with its top at 0, and at 1: 1.0 expected (the same
    searches, but for the last bits of the points); where each ray that ends on
    the zero face is searched twice, 1.8."""
    from voxvision_gb300.cameras import HostCamera
    w, h, took, draws = 1920, 1080, {}, {}
    tex = torch.zeros(32 * 32 * 32, dtype=torch.uint8, device="cuda")
    for top in (0, 1):
        tree = vg.DeviceTree.build(_floor(axis, top, side=256))
        cam = HostCamera(0)
        cam.set_fov(1.0)
        cam.set_window_size(w, h)
        cam.set_position(np.roll(np.array([128, -60, 120 + top], np.float32), axis - 2))
        cam.look_at(np.roll(np.array([128, 128, top], np.float32), axis - 2))
        draws[top] = tree, cam.gpu_struct(), w, h, tex, torch.zeros((h, w), dtype=torch.int32, device="cuda")
    for _ in range(15):
        for top in (0, 1):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                draws[top][0].render_device(*draws[top][1:])
            b.record()
            b.synchronize()
            took.setdefault(top, []).append(a.elapsed_time(b))
    assert (draws[0][5] != 0).float().mean() > 0.2
    assert min(took[0]) < 1.3 * min(took[1]), {k: min(v) for k, v in took.items()}


def _about_the_origin(side=96, seed=5):
    r = np.random.RandomState(seed)
    return np.ascontiguousarray((np.argwhere(r.random_sample((side, side, side)) < 0.1) - side // 2).astype(np.float32))


@pytest.mark.parametrize("zero", [0.0, -0.0])
def test_points_on_planes_at_zero(vg, zero):
    """Rays whose crossings of the planes at zero cancel, from origins with zeros of either sign, inside and outside."""
    vox = _about_the_origin(40)
    vox[vox == 0] = zero
    ht = vg.HostTree.from_voxels(vox)
    r = np.random.RandomState(6)
    n = 60000
    o = (r.randint(-25, 26, (n, 3)) * r.choice([1.0, 0.5, 0.25], (n, 1))).astype(np.float32)
    o[(o == 0) & (r.random_sample((n, 3)) < 0.5)] = -0.0
    d = r.randint(1, 9, (n, 3)) * r.choice([-1.0, 1.0], (n, 3)) * 2.0 ** r.randint(-3, 4, (n, 1))
    to = r.uniform(-20, 20, (n, 3))
    d[::2] = (to - o)[::2]
    d = np.ascontiguousarray(d.astype(np.float32))
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    hit = oleaf != MISS
    assert ((opts == 0).any(1) & hit).sum() > 1000 and (np.signbit(opts) & (opts == 0) & hit[:, None]).any()
    for dt in (vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)):
        leaf, slot, pts = dt.rays(o, d)
        assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
        ok, bad = same_points(pts, opts, hit)
        assert ok, f"{bad} points differ"


def test_boxes_that_end_at_minus_zero(vg):
    """No tree is made with one, but a caller's own may have it: the point's zero keeps its sign."""
    import ctypes as C
    vox = _floor(2, 0, side=40)
    ht = vg.HostTree(vg.lib().vox_make_tree_host(vox.copy().ctypes.data_as(C.c_void_p), len(vox)))
    stack, turned = [ht.ptr], 0
    while stack:
        p = stack.pop()
        top = C.c_float.from_address(p + 20)
        if top.value == 0.0:
            top.value = -0.0
            turned += 1
        if not C.c_uint.from_address(p + 24).value & 3:
            stack += [c for c in (C.c_void_p.from_address(p + 48 + 8 * o).value for o in range(8)) if c]
    assert turned
    o, d = _rays(2, 0, 20000, side=40)
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    leaf, slot, pts = vg.DeviceTree(ht.ptr).rays(o, d)
    assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
    ok, bad = same_points(pts, opts, leaf != MISS)
    assert ok, f"{bad} points differ"


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_planes_at_zero_cost_what_others_do(vg, axis):
    """Frames of a wall that ends at zero, in the middle of a tree about the origin, so that rays end on it where they
    cross the dividing plane at zero; and of the same tree further along: 1.0 expected."""
    from voxvision_gb300.cameras import HostCamera
    w, h, side, took, draws = 640, 480, 96, {}, {}
    tex = torch.zeros(32 * 32 * 32, dtype=torch.uint8, device="cuda")
    r = np.random.RandomState(5)
    wall = np.argwhere(r.random_sample((1, side, side)) < 0.7) + (side // 2 - 1, 0, 0)
    vox = np.unique(np.concatenate([np.argwhere(r.random_sample((side,) * 3) < 0.002), wall]), axis=0) - side // 2
    for shift in (0, side):
        tree = vg.DeviceTree.build(np.ascontiguousarray(np.roll(vox.astype(np.float32), axis, axis=1) + np.float32(shift)))
        cam = HostCamera(0)
        cam.set_fov(1.0)
        cam.set_window_size(w, h)
        cam.set_position(np.roll(np.float32([40, 3.3, 2.2]), axis) + np.float32(shift))
        cam.look_at(np.full(3, shift, np.float32))
        draws[shift] = tree, cam.gpu_struct(), w, h, tex, torch.zeros((h, w), dtype=torch.int32, device="cuda")
    for _ in range(15):
        for shift in draws:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(8):
                draws[shift][0].render_device(*draws[shift][1:])
            b.record()
            b.synchronize()
            took.setdefault(shift, []).append(a.elapsed_time(b))
    assert (draws[0][5] != 0).float().mean() > 0.2
    assert min(took[0]) < 1.3 * min(took[side]), {k: min(v) for k, v in took.items()}
