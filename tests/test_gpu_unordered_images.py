"""Images whose boxes are not ordered, which every search takes in its general
form: frames of every quality, lit, from a ray buffer and in batches, and ray
batches, equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import MISS, same_points

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
W, H = 336, 200


class Scene:
    def __init__(self):
        import voxvision_gb300 as vg
        from voxvision_gb300 import workloads as wl
        from voxvision_gb300.cameras import HostCamera
        self.vg = vg
        vg.set_voxel_size((1, 1, 1))
        orc.set_voxel((1, 1, 1))
        vox = wl.voxels_from_mask(wl.blobs_volume(64, 20, 1, 0.20))
        self.ht = vg.HostTree(vg.lib().vox_make_tree_host(vox.copy().ctypes.data_as(C.c_void_p), len(vox)))
        stack, turned = [self.ht.ptr], 0
        while stack and turned < 12:   # some inner nodes' boxes are turned round
            p = stack.pop(0)
            if C.c_uint.from_address(p + 24).value & 3:
                continue
            kids = [c for c in (C.c_void_p.from_address(p + 48 + 8 * o).value for o in range(8)) if c]
            stack += kids
            if p != self.ht.ptr and turned < 12 and turned % 2 == 0:
                lo, hi = C.c_float.from_address(p + 4 * (turned % 3)), C.c_float.from_address(p + 12 + 4 * (turned % 3))
                lo.value, hi.value = hi.value, lo.value
            turned += 1
        self.dt = vg.DeviceTree(self.ht.ptr)
        self.cam = HostCamera(0)
        self.cam.set_window_size(W, H)
        self.cam.set_position((150.0, -90.0, 100.0))
        self.cam.look_at(np.array([32.0, 32.0, 32.0], np.float32))
        self.tex = wl.texture32(7)


@pytest.fixture(scope="module")
def scene():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    return Scene()


@pytest.mark.parametrize("quality", [0, 1, 2, 2 | 4, 2 | 8])
def test_frames(scene, quality):
    s = scene
    ref, _ = orc.render_quality(s.ht.ptr, s.cam.state(), W, H, quality, s.tex)
    assert (ref != 0).sum() > 1500
    assert np.array_equal(s.dt.render_quality(s.cam.gpu_struct(), W, H, quality, s.tex), ref)
    if quality == 0:
        assert np.array_equal(s.dt.render(s.cam.gpu_struct(), W, H, s.tex), ref)
        assert np.array_equal(s.dt.render_frames([s.cam.gpu_struct()], W, H, s.tex)[0], ref)
    dev, dtex = torch.zeros((H, W), dtype=torch.int32, device="cuda"), torch.from_numpy(s.tex).cuda()
    dirs = np.array([[orc.screen2world(s.cam.state(), x, y) for x in range(W)] for y in range(H)], np.float32)
    s.dt.render_rays_device(s.cam.state()["position"], torch.from_numpy(dirs).cuda(), W, H, quality, dtex, dev)
    assert np.array_equal(dev.cpu().numpy().view(np.uint32), ref)
    if quality == 0:
        b = s.vg.FrameBatch([(s.dt, s.cam.gpu_struct(), W, H, dtex, dev)])
        dev.zero_()
        b.launch()
        assert np.array_equal(dev.cpu().numpy().view(np.uint32), ref)


@pytest.mark.parametrize("quality", [0, 2])
def test_lit_frames(scene, quality):
    s = scene
    m, o = s.vg.LightManager(), orc.OracleLights()
    r = np.random.RandomState(4)
    for x in (m, o):
        x.ambient((0.2, 0.2, 0.25))
    for _ in range(12):
        c, rad, col = r.uniform(0, 64, 3).astype(np.float32), float(r.uniform(5, 30)), r.uniform(0, 1, 3).astype(np.float32)
        m.insert(c, rad, col)
        o.insert(c, rad, col)
    ref = orc.render_lit(s.ht.ptr, s.cam.state(), W, H, quality, s.tex, o)
    assert np.array_equal(s.dt.render_lit(s.cam.gpu_struct(), W, H, quality, s.tex, m.upload()), ref)


@pytest.mark.parametrize("n,launches", [(262143, 1), (262144, 4), (300000, 4), (393216, 4)])
def test_ray_batches_are_sorted_where_it_pays(scene, n, launches):
    """From 262,144 rays on these batches are traced grouped (three kernels more), and answer the same."""
    s = scene
    r = np.random.RandomState(n)
    o = r.uniform(-40, 104, (n, 3)).astype(np.float32)
    d = r.standard_normal((n, 3)).astype(np.float32)
    do, dd = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    leaf = torch.zeros(n, dtype=torch.int32, device="cuda")
    slot, pts = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.zeros((n, 3), device="cuda")
    before = s.vg.lib().vox_cuda_launch_count()
    s.dt.rays_device(do, dd, leaf, slot, pts)
    torch.cuda.synchronize()
    assert s.vg.lib().vox_cuda_launch_count() - before == launches
    oleaf, oslot, opts, _ = orc.ray_batch(s.ht.ptr, o, d)
    got = leaf.cpu().numpy().view(np.uint32)
    assert np.array_equal(got, oleaf) and np.array_equal(slot.cpu().numpy(), oslot)
    ok, bad = same_points(pts.cpu().numpy(), opts, got != MISS)
    assert ok, f"{bad} points differ"
