"""Uploads of trees with overflowed leaves: a leaf of a million equal voxels
costs what its bytes cost, and one voxel out of place anywhere in it is seen."""
import ctypes as C
import time

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def vg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as m
    before = m.lib().vox_cuda_make_tree_gpu_min(2 ** 63)
    yield m
    m.lib().vox_cuda_make_tree_gpu_min(before)


def _upload_ms(vg, root):
    best = 1e9
    for _ in range(4):
        a = time.perf_counter()
        dt = vg.DeviceTree(root)
        best = min(best, 1e3 * (time.perf_counter() - a))
        dt.close()
    return best


def test_upload_of_a_long_leaf(vg):
    """Against a tree of ordinary leaves with an image of the same size or less
    (its flattening is the larger part): below 1.0 expected; with one thread to
    a leaf 60."""
    n = 1000000
    equal = np.tile(np.float32([3, 4, 5]), (n, 1))
    equal[0] = 9
    long_leaf = vg.HostTree.from_voxels(equal)
    r = np.random.RandomState(2)
    cells = np.unique(r.randint(0, 160, (400000, 3)), axis=0).astype(np.float32)
    ordinary = vg.HostTree.from_voxels(np.ascontiguousarray(cells))
    assert vg.measure_tree(ordinary.ptr)["device_bytes"] >= 0.8 * vg.measure_tree(long_leaf.ptr)["device_bytes"]
    assert _upload_ms(vg, long_leaf.ptr) < 3 * _upload_ms(vg, ordinary.ptr)


@pytest.mark.parametrize("n", [8, 31, 1024, 1025, 4097, 50000])
@pytest.mark.parametrize("where", ["first", "middle", "last"])
def test_a_voxel_outside_its_long_leaf(vg, n, where):
    """Ball answers over a leaf one of whose voxels lies outside the leaf's box (the box hides it, as in the reference)."""
    vox = np.concatenate([np.tile(np.float32([3, 4, 5]), (n, 1)), np.float32([[20, 20, 20], [21, 20, 20], [40, 4, 5]])])
    ht = vg.HostTree.from_voxels(np.ascontiguousarray(vox))
    stack, leaf = [ht.ptr], None
    while stack:
        p = stack.pop()
        if C.c_uint.from_address(p + 24).value & 1:
            if C.c_uint.from_address(p + 28).value >= n:
                leaf = p
        elif not C.c_uint.from_address(p + 24).value & 2:
            stack += [c for c in (C.c_void_p.from_address(p + 48 + 8 * o).value for o in range(8)) if c]
    assert leaf
    i = {"first": 0, "middle": n // 2, "last": n - 1}[where]
    dots = C.c_void_p.from_address(leaf + 32).value
    for a, x in enumerate((30.0, 30.0, 30.0)):
        C.c_float.from_address(dots + 12 * i + 4 * a).value = x
    r = np.random.RandomState(n)
    c = r.uniform(0, 45, (4096, 3)).astype(np.float32)
    c[::2] = r.uniform(28, 33, (2048, 3))
    rad = r.uniform(0.1, 30, 4096).astype(np.float32)
    want, _ = orc.ball_batch(ht.ptr, c, rad)
    assert np.array_equal(vg.DeviceTree(ht.ptr).balls(c, rad), want)
