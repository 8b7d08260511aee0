"""Trees built by several threads at once, beside frames of the trees just
built: every image is the host build's."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _set(i):
    r = np.random.RandomState(i)
    n = (40, 900, 7000, 33000, 120000, 400000)[i % 6]
    if i % 2:
        side = int(round((8 * n) ** (1 / 3))) + 2
        v = r.choice(side ** 3, n, replace=False)
        v = np.stack([v // side // side, v // side % side, v % side], 1)
    else:
        v = r.random_sample((n, 3)) * 10.0 ** r.randint(-3, 4, (n, 1))
    return np.ascontiguousarray(v.astype(np.float32))


def test_builds_at_once():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as vg
    from voxvision_gb300.cameras import HostCamera
    sets = [_set(i) for i in range(12)]
    want = []
    for v in sets:
        copy = v.copy()
        ht = vg.HostTree(vg.lib().vox_make_tree_host(copy.ctypes.data_as(C.c_void_p), len(copy)))
        want.append(vg.DeviceTree(ht.ptr).image())
    cam = HostCamera(0)
    cam.set_window_size(320, 240)
    cam.set_position((150.0, -90.0, 100.0))
    cam.look_at(np.array([32.0, 32.0, 32.0], np.float32))
    tex = np.zeros(32768, np.uint8)
    frames = {}
    for i, v in enumerate(sets):
        frames[i] = vg.DeviceTree.build(v).render(cam.gpu_struct(), 320, 240, tex)
    dev = [torch.from_numpy(v).cuda() for v in sets]
    torch.cuda.synchronize()
    wrong = []

    def work(t):
        try:
            for k in range(24):
                i = (5 * t + 7 * k) % len(sets)
                tree = vg.DeviceTree.build_device(dev[i]) if k % 3 else vg.DeviceTree.build(sets[i])
                u, ids = tree.image()
                if not (np.array_equal(u, want[i][0]) and np.array_equal(ids, want[i][1])):
                    wrong.append(("image", t, k, i))
                if not np.array_equal(tree.render(cam.gpu_struct(), 320, 240, tex), frames[i]):
                    wrong.append(("frame", t, k, i))
                if k % 2:
                    tree.close()
        except Exception as e:   # reported by the test's own thread
            wrong.append((t, repr(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not wrong, wrong[:5]
