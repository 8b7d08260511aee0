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
