"""Trees are built from device memory and freed in some threads while others
capture streams (a batch being made captures one of its own): neither fails."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_builds_and_frees_beside_captures():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as vg
    from voxvision_gb300.cameras import HostCamera
    r = np.random.RandomState(1)
    vox = np.unique(r.randint(0, 60, (20000, 3)), axis=0).astype(np.float32)
    dev = torch.from_numpy(vox).cuda()
    still = vg.DeviceTree.build(vox)
    cam = HostCamera(0)
    cam.set_window_size(320, 240)
    cam.set_position((150.0, -90.0, 100.0))
    cam.look_at(np.array([32.0, 32.0, 32.0], np.float32))
    tex = torch.zeros(32768, dtype=torch.uint8, device="cuda")
    out = torch.zeros((240, 320), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    done, wrong = threading.Event(), []

    def run(f):
        def body():
            try:
                f()
            except Exception as e:   # reported by the test's own thread
                wrong.append(repr(e))
            finally:
                done.set()
        return body

    def batches():
        for _ in range(400):
            b = vg.FrameBatch([(still, cam.gpu_struct(), 320, 240, tex, out)])
            b.close()
            if wrong:
                break

    def builds():
        while not done.is_set():
            vg.DeviceTree.build_device(dev).close()

    def host_builds():
        while not done.is_set():
            vg.DeviceTree.build(vox).close()

    threads = [threading.Thread(target=run(f)) for f in (batches, builds, host_builds)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
