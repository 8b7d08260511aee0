"""Trees of more than 2^24 voxels, where the builder's centre sums take maps of
sixteen binades and its largest nodes tiles of more than 2,048 positions: the
image is the host build's byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N = (1 << 24) + 4099


@pytest.fixture(scope="module")
def vg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as m
    before = m.lib().vox_cuda_make_tree_gpu_min(2 ** 63)   # the reference tree is built on the host
    yield m
    m.lib().vox_cuda_make_tree_gpu_min(before)


def _set(kind):
    r = np.random.default_rng(7)
    if kind == "grid":         # cells in raster order, their sums past 2^24
        keep = r.random(323 ** 3) < 0.51
        return np.stack(np.unravel_index(np.flatnonzero(keep)[:N], (323,) * 3), 1).astype(np.float32)
    return (r.random((N, 3), np.float32) * np.float32(10.0) ** r.integers(-3, 5, (N, 1)).astype(np.float32)).astype(np.float32)


@pytest.mark.parametrize("kind", ["grid", "rounding"])
def test_image_is_the_host_builds(vg, kind):
    vox = np.ascontiguousarray(_set(kind))
    assert len(vox) == N
    ht = vg.HostTree.from_voxels(vox)
    up, made = vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)
    (hu, hi), (du, di) = up.image(), made.image()
    assert np.array_equal(hu, du) and np.array_equal(hi, di)
    a, b = up.info(), made.info()
    assert all(a[k] == b[k] for k in ("nodes", "inner", "leaves", "dense_leaves", "dots", "depth"))
