"""Trees built on the GPU at the edges of the builder's size classes (voxels in
lanes, by a warp, by a block, tile by tile) and of its centre sums (plain where
no addition rounds, by maps of binades elsewhere), and raw volumes at the edges
of a thread's and a block's samples: the image is the host build's byte for
byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def vg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()
    import voxvision_gb300 as m
    before = m.lib().vox_cuda_make_tree_gpu_min(2 ** 63)   # the reference trees are built on the host
    yield m
    m.lib().vox_cuda_make_tree_gpu_min(before)
    m.set_voxel_size((1, 1, 1))


def _same(vg, vox, made):
    ht = vg.HostTree.from_voxels(vox)
    up = vg.DeviceTree(ht.ptr)
    (hu, hi), (du, di) = up.image(), made.image()
    assert np.array_equal(hu, du) and np.array_equal(hi, di)
    a, b = up.info(), made.info()
    assert all(a[k] == b[k] for k in ("nodes", "inner", "leaves", "dense_leaves", "dots", "depth"))


def _set(kind, n, seed):
    r = np.random.RandomState(seed)
    if kind == "scattered":      # unit cells in no order
        side = max(4, int(round((8 * n) ** (1 / 3))) + 1)
        v = r.choice(side ** 3, n, replace=False)
        v = np.stack([v // side // side, v // side % side, v % side], 1)
    elif kind == "raster":       # a solid region in raster order, one cell missing
        side = int(np.ceil((n + 1) ** (1 / 3)))
        v = np.stack(np.unravel_index(np.arange(n + 1), (side,) * 3), 1)
        v = np.delete(v, n // 2, 0)
    elif kind == "rounding":     # sums that round: coordinates of many magnitudes, off the grid
        v = r.random_sample((n, 3)) * 10.0 ** r.randint(-3, 5, (n, 1))
    else:                        # "duplicates": few distinct voxels, leaves that overflow
        v = r.randint(0, 3, (n, 3)) * 7 - 4
    return np.ascontiguousarray(v.astype(np.float32))


@pytest.mark.parametrize("kind", ["scattered", "raster", "rounding", "duplicates"])
@pytest.mark.parametrize("n", [1, 7, 8, 31, 32, 33, 64, 65, 511, 512, 513, 1024, 1025, 1056, 8191, 8192, 8193, 9216,
                               17409, 32768, 32769, 60000])
def test_sizes_at_class_edges(vg, kind, n):
    vox = _set(kind, n, n)
    _same(vg, vox, vg.DeviceTree.build(vox))


@pytest.mark.parametrize("scale", [1.0, 3.7e4])
def test_large_set_of_rounding_sums(vg, scale):
    vox = _set("rounding", 300000, 3) * np.float32(scale)
    _same(vg, vox, vg.DeviceTree.build(vox))


@pytest.mark.parametrize("dim", [(1, 1, 1), (1, 3, 5), (1, 1, 16), (17, 1, 1), (3, 5, 7), (16, 16, 16), (1, 4095, 1),
                                 (1, 17, 241), (2, 3, 1367), (24, 16, 32)])
@pytest.mark.parametrize("size", [1, 2, 3, 4])
def test_raw_volumes_at_tile_edges(vg, dim, size):
    r = np.random.RandomState(sum(dim) + size)
    n = dim[0] * dim[1] * dim[2]
    x = r.randint(0, 200, n).astype(np.uint32) * np.uint32([0, 1, 300, 70000, 20000000][size])
    raw = x.astype("<u4").view(np.uint8).reshape(n, 4)[:, :size].copy()
    lo, hi = int(x.max() // 4), int(x.max())
    if size == 4:
        hi = 0xFFFFFFFF
    solid = ((x >= lo) & (x <= hi)).reshape(dim)
    made = vg.DeviceTree.from_raw(raw.reshape(-1), dim, size, lo, hi)
    _same(vg, np.ascontiguousarray(np.argwhere(solid).astype(np.float32)), made)
    if size <= 2:
        made = vg.DeviceTree.from_raw(raw.reshape(-1), dim, size, test=lambda s: s % 3 == 1)
        vox = np.argwhere((x % 3 == 1).reshape(dim)).astype(np.float32)
        if len(vox):
            _same(vg, np.ascontiguousarray(vox), made)
        else:
            assert made.info()["nodes"] == 0


@pytest.mark.parametrize("side_stream", [False, True])
def test_voxels_still_on_their_way(vg, side_stream):
    # the set is written by work that is not done when the build is called
    vox = _set("scattered", 40000, 11)
    src, dst = torch.from_numpy(vox).cuda(), torch.zeros(vox.shape, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)   # some 10 ms
        dst.copy_(src)
        made = vg.DeviceTree.build_device(dst)
    _same(vg, vox, made)
