"""A frame batch whose tree was refreshed draws the tree as it is now, at the
next launch and without a new batch: the frames are those of the single-frame
call, which are compared with the oracle's."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
W, H = 320, 240


@pytest.fixture(scope="module")
def vg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as m
    m.set_voxel_size((1, 1, 1))
    orc.set_voxel((1, 1, 1))
    return m


class Scene:
    def __init__(self, vg):
        from voxvision_gb300 import workloads as wl
        from voxvision_gb300.cameras import HostCamera
        self.vg, self.L = vg, vg.lib()
        vox = np.ascontiguousarray(wl.voxels_from_mask(wl.blobs_volume(48, 12, 1, 0.20))).copy()
        self.root = C.c_void_p(self.L.vox_make_tree_host(vox.ctypes.data_as(C.c_void_p), vox.shape[0]))
        self.tree = vg.DeviceTree(self.root.value)
        self.cams = []
        for at in ((130.0, -70.0, 90.0), (-60.0, 20.0, 60.0)):
            c = HostCamera(0)
            c.set_window_size(W, H)
            c.set_position(at)
            c.look_at(np.array([24.0, 24.0, 24.0], np.float32))
            self.cams.append(c)
        self.tex = wl.texture32(7)
        self.dtex = torch.from_numpy(self.tex).cuda()
        self.out = torch.zeros((2, H, W), dtype=torch.int32, device="cuda")
        self.batch = vg.FrameBatch([(self.tree, c.gpu_struct(), W, H, self.dtex, self.out[i])
                                    for i, c in enumerate(self.cams)])

    def check(self):
        self.out.zero_()
        self.batch.launch()
        torch.cuda.synchronize()
        got = self.out.cpu().numpy().view(np.uint32)
        for i, c in enumerate(self.cams):
            ref, _ = orc.render_best(self.root.value, c.state(), W, H, self.tex)
            assert np.array_equal(self.tree.render(c.gpu_struct(), W, H, self.tex), ref)
            assert np.array_equal(got[i], ref), f"frame {i}: {(got[i] != ref).sum()} pixels differ"

    def refresh(self):
        self.vg.check(self.L.vox_cuda_tree_refresh(self.tree.h, self.root), "vox_cuda_tree_refresh")


def test_boxes_no_longer_ordered(vg):
    s = Scene(vg)
    s.check()
    for o in range(8):   # every inner child of the root: its box turned round on x
        child = C.c_void_p.from_address(s.root.value + 48 + 8 * o).value
        if child and not (C.c_uint.from_address(child + 24).value & 3):
            lo, hi = C.c_float.from_address(child), C.c_float.from_address(child + 12)
            lo.value, hi.value = hi.value, lo.value
    s.refresh()
    s.check()


def test_tree_grows_and_shrinks(vg):
    s = Scene(vg)
    s.check()
    rng = np.random.default_rng(3)
    for lo, hi, n in ((-20, 70, 4000), (23, 25, 300), (10, 40, 200)):
        for _ in range(n):   # past the old buffers and box, then deeper
            a = rng.uniform(lo, hi, 3).astype(np.float32) if hi - lo < 5 else rng.integers(lo, hi, 3).astype(np.float32)
            s.L.vox_insert_voxel(C.byref(s.root), a.ctypes.data_as(C.c_void_p))
        s.refresh()
        s.check()
