"""What the searches may rely on in an image (ordered boxes, nested boxes): an
uploaded tree that breaks any one part of it takes the searches that do not
rely on it, and rays and balls stay the oracle's.  The route shows in the
kernels launched: sorting takes three, for balls over an image whose boxes
do not nest and for rays over one whose boxes are not ordered."""
import ctypes as C

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
    m.set_voxel_size((1, 1, 1))
    orc.set_voxel((1, 1, 1))
    return m


class Node:
    """A host node's fields in place (struct vox_node)."""

    def __init__(self, p):
        self.p = p
        self.flags = C.c_uint.from_address(p + 24).value
        self.inner = not self.flags & 3
        self.leaf = bool(self.flags & 1) and not self.flags & 2
        self.n = C.c_uint.from_address(p + 28).value

    def f(self, at, value=None):
        x = C.c_float.from_address(self.p + at)
        if value is not None:
            x.value = value
        return x.value

    def lo(self, a, v=None):
        return self.f(4 * a, v)

    def hi(self, a, v=None):
        return self.f(12 + 4 * a, v)

    def centre(self, a, v=None):
        return self.f(32 + 4 * a, v)

    def children(self):
        kids = [C.c_void_p.from_address(self.p + 48 + 8 * o).value for o in range(8)]
        return [(o, Node(c)) for o, c in enumerate(kids) if c]

    def dot(self, i, a, v=None):
        x = C.c_float.from_address(C.c_void_p.from_address(self.p + 32).value + 12 * i + 4 * a)
        if v is not None:
            x.value = v
        return x.value


def _tree(vg, seed=3):
    r = np.random.RandomState(seed)
    cells = np.argwhere(r.random_sample((32, 30, 28)) < 0.08).astype(np.float32)
    return vg.HostTree(vg.lib().vox_make_tree_host(np.ascontiguousarray(cells).ctypes.data_as(C.c_void_p), len(cells)))


def _nodes(root):
    out, stack = [], [(None, None, Node(root))]
    while stack:
        parent, o, x = stack.pop()
        out.append((parent, o, x))
        if x.inner:
            stack += [(x, oc, c) for oc, c in x.children()]
    return out


def _break(what, root, axis, r):
    """Breaks one thing somewhere in the tree; the shape bits it should lose."""
    nodes = _nodes(root)
    pairs = [(p, o, x) for p, o, x in nodes if p is not None]
    r.shuffle(pairs)
    low = [(p, x) for p, o, x in pairs if (o >> axis) & 1]
    high = [(p, x) for p, o, x in pairs if not (o >> axis) & 1]
    leaf = next(x for _, _, x in pairs if x.leaf and 1 < x.n <= 7)
    if what == "nothing":
        return ""
    if what == "child past its parent":
        p, x = high[0]
        x.hi(axis, p.hi(axis) + 3)
    elif what == "child before its parent":
        p, x = low[0]
        x.lo(axis, p.lo(axis) - 3)
    elif what == "upper child below the plane":
        p, x = next((p, x) for p, x in high if p.lo(axis) < p.centre(axis) - 0.5)
        x.lo(axis, p.centre(axis) - 0.5)
    elif what == "lower child past the plane":
        p, x = next((p, x) for p, x in low if p.hi(axis) > p.centre(axis) + 1.5)
        x.hi(axis, p.centre(axis) + 1.5)
    elif what == "voxel past its leaf":
        leaf.dot(leaf.n - 1, axis, leaf.hi(axis) + 2)
    elif what == "voxel before its leaf":
        leaf.dot(0, axis, leaf.lo(axis) - 0.25)
    elif what == "box turned round":
        x = high[0][1]
        a, b = x.lo(axis), x.hi(axis)
        x.lo(axis, b)
        x.hi(axis, a)
        return "ordered"
    elif what == "centre past 2^60":
        next(x for p, x in low if x.inner).centre(axis, 2.0 ** 61)
        return "ordered"
    elif what == "box past 2^60":
        Node(root).hi(axis, 2.0 ** 61)
        return "ordered only"
    elif what == "tiny voxel":
        leaf.dot(0, axis, 1e-30)
        return "ordered"
    elif what == "not a number":
        leaf.dot(0, axis, float("nan"))
        return "ordered"
    return "nested"


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("what", ["nothing", "child past its parent", "child before its parent",
                                  "upper child below the plane", "lower child past the plane", "voxel past its leaf",
                                  "voxel before its leaf", "box turned round", "centre past 2^60", "box past 2^60",
                                  "tiny voxel", "not a number"])
def test_one_thing_broken(vg, what, axis):
    for seed in range(4):
        r = np.random.RandomState(100 * seed + axis)
        ht = _tree(vg, seed)
        lost = _break(what, ht.ptr, axis, r)
        dt = vg.DeviceTree(ht.ptr)
        n = 1 << 18
        c = r.uniform(-6, 38, (n, 3)).astype(np.float32)
        rad = r.uniform(0.1, 5, n).astype(np.float32)
        before = vg.lib().vox_cuda_launch_count()
        hit = dt.balls(c, rad)
        launched = vg.lib().vox_cuda_launch_count() - before
        assert launched == (1 if lost == "" else 4), (what, launched)   # nested: one search; else sorted first
        want, _ = orc.ball_batch(ht.ptr, c, rad)
        assert np.array_equal(hit, want), f"{(hit != want).sum()} balls differ"
        o = r.uniform(-40, 70, (n, 3)).astype(np.float32)
        d = (r.uniform(0, 30, (n, 3)) - o).astype(np.float32)
        before = vg.lib().vox_cuda_launch_count()
        leaf, slot, pts = dt.rays(o, d)
        launched = vg.lib().vox_cuda_launch_count() - before
        assert launched == (4 if lost.startswith("ordered") else 1), (what, launched)
        oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
        assert np.array_equal(leaf, oleaf), f"{(leaf != oleaf).sum()} leaf ids differ"
        assert np.array_equal(slot, oslot)
        ok, bad = same_points(pts, opts, leaf != MISS)
        assert ok, f"{bad} points differ"


@pytest.mark.parametrize("n", [5, 30, 400, 3000, 20000, 40000])
@pytest.mark.parametrize("value,ordinary", [(2.0 ** 57, True), (-2.0 ** 57, True), (np.nextafter(np.float32(2.0 ** 57), np.float32(1e30)), False),
                                            (2.0 ** 60, False), (-2.0 ** 62, False), (1e30, False), (2.0 ** -55, True),
                                            (2.0 ** -56, False), (1e-40, False), (-0.0, True)])
def test_builds_with_a_coordinate_out_of_the_ordinary(vg, n, value, ordinary):
    """Built on the GPU: the host build's image, and its answers."""
    r = np.random.RandomState(n)
    vox = np.unique(r.randint(0, 60, (n, 3)), axis=0).astype(np.float32)
    r.shuffle(vox)
    vox[len(vox) // 2, r.randint(0, 3)] = value
    vox = np.ascontiguousarray(vox)
    copy = vox.copy()
    ht = vg.HostTree(vg.lib().vox_make_tree_host(copy.ctypes.data_as(C.c_void_p), len(copy)))
    up, made = vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)
    (hu, hi), (du, di) = up.image(), made.image()
    assert np.array_equal(hu, du) and np.array_equal(hi, di)
    m = 1 << 18
    c, rad = r.uniform(-10, 70, (m, 3)).astype(np.float32), r.uniform(0.1, 9, m).astype(np.float32)
    o = r.uniform(-90, 150, (m, 3)).astype(np.float32)
    d = (r.uniform(0, 60, (m, 3)) - o).astype(np.float32)
    want, _ = orc.ball_batch(ht.ptr, c, rad)
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    for dt in (up, made):
        assert np.array_equal(dt.balls(c, rad), want)
        before = vg.lib().vox_cuda_launch_count()
        leaf, slot, pts = dt.rays(o, d)
        if ordinary:
            assert vg.lib().vox_cuda_launch_count() - before == 1
        assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
        ok, bad = same_points(pts, opts, leaf != MISS)
        assert ok, f"{bad} points differ"


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("what", ["nothing", "child past its parent", "upper child below the plane", "voxel past its leaf",
                                  "box turned round", "tiny voxel", "not a number"])
def test_one_thing_broken_in_a_small_tree(vg, what, axis):
    """Small images are checked on the host: the routes are the same."""
    r = np.random.RandomState(axis)
    cells = np.argwhere(r.random_sample((8, 8, 8)) < 0.3).astype(np.float32)
    ht = vg.HostTree(vg.lib().vox_make_tree_host(np.ascontiguousarray(cells).ctypes.data_as(C.c_void_p), len(cells)))
    lost = _break(what, ht.ptr, axis, r)
    before = vg.lib().vox_cuda_launch_count()
    dt = vg.DeviceTree(ht.ptr)
    assert vg.lib().vox_cuda_launch_count() == before   # no kernel to check it
    n = 1 << 18
    c, rad = r.uniform(-4, 12, (n, 3)).astype(np.float32), r.uniform(0.1, 3, n).astype(np.float32)
    before = vg.lib().vox_cuda_launch_count()
    hit = dt.balls(c, rad)
    assert vg.lib().vox_cuda_launch_count() - before == (1 if lost == "" else 4)
    assert np.array_equal(hit, orc.ball_batch(ht.ptr, c, rad)[0])
    o = r.uniform(-20, 28, (n, 3)).astype(np.float32)
    d = (r.uniform(0, 8, (n, 3)) - o).astype(np.float32)
    before = vg.lib().vox_cuda_launch_count()
    leaf, slot, pts = dt.rays(o, d)
    assert vg.lib().vox_cuda_launch_count() - before == (4 if lost.startswith("ordered") else 1)
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
    ok, bad = same_points(pts, opts, leaf != MISS)
    assert ok, f"{bad} points differ"
