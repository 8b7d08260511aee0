"""The two forms of the ray search (traverse.cuh): ordinary rays take the
mirrored one, the others the general one.  Every ray's leaf, voxel and point
bits are the oracle's on both sides of each bound that chooses between them,
where crossings tie, and where the mirror cannot tell a zero's sign."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import MISS, same_points

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxvision_gb300.build import build
    build()


def _voxels(seed, voxel, shift):
    """A ragged blob of cells around `shift`, both sides of zero, with flat parts and dense cubes."""
    r = np.random.RandomState(seed)
    g = np.argwhere(r.random_sample((20, 18, 16)) < 0.12)
    cube = np.argwhere(np.ones((5, 5, 5))) + (3, 8, 2)
    flat = np.argwhere(np.ones((12, 1, 9))) + (6, 15, 5)
    cells = np.unique(np.concatenate([g, cube, flat]), axis=0) - (10, 9, 8) + np.asarray(shift)
    return np.ascontiguousarray((cells * np.asarray(voxel)).astype(np.float32))


def _rays(seed, n, box):
    r = np.random.RandomState(seed)
    lo, hi = box
    span = hi - lo
    o = (lo - span + 3 * span * r.random_sample((n, 3))).astype(np.float32)
    to = lo + span * r.random_sample((n, 3))
    d = (to - o).astype(np.float32)
    return r, o, d, to


def _family(kind, seed, box, voxel):
    r, o, d, to = _rays(seed, 4096, box)
    n = len(o)
    a, b = r.randint(0, 3, n), r.randint(0, 3, n)
    i = np.arange(n)
    if kind == "plain":
        pass
    elif kind == "direction bounds":   # one component at, just inside and just outside the accepted range
        edge = np.array([2.0 ** -30, 2.0 ** 20, 1e-40, 0.0], np.float32)[r.randint(0, 4, n)]
        edge = np.nextafter(edge, np.array([0, np.inf], np.float32)[r.randint(0, 2, n)].astype(np.float32))
        d[i, a] = edge * np.sign(d[i, a])
        d[: n // 4] = (d[: n // 4] * np.float32(2.0 ** 14)).astype(np.float32)
    elif kind == "axis and signed zero":
        d[i, a] = np.array([0.0, -0.0], np.float32)[r.randint(0, 2, n)]
        d[i[::2], b[::2]] = np.array([0.0, -0.0], np.float32)[r.randint(0, 2, n // 2)]
    elif kind == "not finite":
        odd = np.array([np.inf, -np.inf, np.nan, 3e38], np.float32)
        d[i[::3], a[::3]] = odd[r.randint(0, 4, len(i[::3]))]
        o[i[1::3], b[1::3]] = odd[r.randint(0, 4, len(i[1::3]))]
    elif kind == "origins on planes":   # on cell faces, a hair off them, and on zero of either sign
        o = (np.rint(o / voxel) * voxel).astype(np.float32)
        o[i[::2], a[::2]] += np.array([0, 1e-30, -1e-30, 1e-12, -1e-12], np.float32)[r.randint(0, 5, n // 2)]
        o[i[::5], b[::5]] = np.array([0.0, -0.0, 1e-30], np.float32)[r.randint(0, 3, len(i[::5]))]
    elif kind == "ties":                # diagonal rays between cell corners: crossings at equal distances
        o = (np.rint(o / voxel) * voxel).astype(np.float32)
        d = (np.sign(d) * np.asarray(voxel) * np.array([1, 1, 2])[r.randint(0, 3, (n, 3))]).astype(np.float32)
    elif kind == "zero coordinates":    # aimed at points with zero coordinates, along both signs
        to = np.rint((box[0] + (box[1] - box[0]) * r.random_sample((n, 3))) / voxel) * voxel
        to[i, a] = 0.0
        step = np.array([1.0, 2.0, 4.0])[r.randint(0, 3, n)][:, None] * np.sign(d) * np.asarray(voxel)
        o, d = (to - 8 * step).astype(np.float32), step.astype(np.float32)
    elif kind == "far origins":
        o[i, a] = (np.float32(2.0) ** r.randint(8, 64, n)).astype(np.float32) * np.sign(o[i, a])
        d = to - o.astype(np.float64)
        d = (d / np.abs(d).max(1, keepdims=True)).astype(np.float32)
    return np.ascontiguousarray(o), np.ascontiguousarray(d)


@pytest.mark.parametrize("voxel,shift", [((1, 1, 1), (0, 0, 0)), ((0.5, 1, 2), (3, -5, 40)), ((1, -1, 1), (0, 0, 0))])
@pytest.mark.parametrize("kind", ["plain", "direction bounds", "axis and signed zero", "not finite",
                                  "origins on planes", "ties", "zero coordinates", "far origins"])
def test_both_forms_of_the_search_match_the_oracle(kind, voxel, shift):
    import voxvision_gb300 as vg
    try:
        vg.set_voxel_size(voxel)   # a negative size gives unordered boxes: every ray takes the general form
        orc.set_voxel(voxel)
        vox = _voxels(5, voxel, shift)
        ht = vg.HostTree.from_voxels(vox)
        up, made = vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)
        box = vox.min(0).astype(np.float64), vox.max(0).astype(np.float64) + np.abs(voxel)
        o, d = _family(kind, 9, box, np.asarray(voxel, np.float64))
        oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
        for dt in (up, made):
            leaf, slot, pts = dt.rays(o, d)
            assert np.array_equal(leaf, oleaf), f"{(leaf != oleaf).sum()} leaf ids differ"
            assert np.array_equal(slot, oslot)
            ok, bad = same_points(pts, opts, leaf != MISS)
            assert ok, f"{bad} points differ"
        if kind == "plain" and voxel[1] > 0:
            assert 0.1 < (leaf != MISS).mean() < 1.0
    finally:
        vg.set_voxel_size((1, 1, 1))
        orc.set_voxel((1, 1, 1))


def _balls(kind, seed, box, voxel):
    r = np.random.RandomState(seed)
    lo, hi = box
    n = 4096
    c = (lo - 3 + (hi - lo + 6) * r.random_sample((n, 3))).astype(np.float32)
    rad = (4 * np.abs(voxel).max() * r.random_sample(n)).astype(np.float32)
    if kind == "touching":   # the radius is the float distance to a cell face, or one step to either side
        face = np.rint(c[np.arange(n), r.randint(0, 3, n)]).astype(np.float32)
        rad = np.abs(face - c[np.arange(n), r.randint(0, 3, n)]).astype(np.float32)
        rad = np.nextafter(rad, np.array([-1e9, 1e9], np.float32)[r.randint(0, 2, n)]).astype(np.float32)
        c[::2] = np.rint(c[::2] / voxel) * voxel
        rad[::2] = (np.rint(rad[::2]) * np.abs(voxel[0])).astype(np.float32)
    elif kind == "odd numbers":
        odd = np.array([np.nan, np.inf, -np.inf, 3e38, -3e38, 1e-40, -0.0, 1e25], np.float32)
        rad[::3] = odd[r.randint(0, 8, len(rad[::3]))]
        c[np.arange(1, n, 3), r.randint(0, 3, len(c[1::3]))] = odd[r.randint(0, 8, len(c[1::3]))]
        rad[2::6] = -rad[2::6]
    return np.ascontiguousarray(c), np.ascontiguousarray(rad)


@pytest.mark.parametrize("voxel,shift", [((1, 1, 1), (0, 0, 0)), ((0.5, 1, 2), (3, -5, 40)), ((1, -1, 1), (0, 0, 0))])
@pytest.mark.parametrize("kind", ["plain", "touching", "odd numbers"])
@pytest.mark.parametrize("off_grid", [False, True])
def test_both_forms_of_the_ball_search_match_the_oracle(kind, voxel, shift, off_grid):
    import voxvision_gb300 as vg
    try:
        vg.set_voxel_size(voxel)   # a negative size gives unordered boxes: the general form
        orc.set_voxel(voxel)
        vox = _voxels(5, voxel, shift)
        if off_grid:               # voxels that reach past the dividing planes
            vox += np.random.RandomState(3).uniform(-0.4, 0.4, vox.shape).astype(np.float32)
        ht = vg.HostTree.from_voxels(vox)
        box = vox.min(0).astype(np.float64), vox.max(0).astype(np.float64) + np.abs(voxel)
        c, rad = _balls(kind, 11, box, np.asarray(voxel, np.float64))
        want, _ = orc.ball_batch(ht.ptr, c, rad)
        if kind == "plain" and voxel[1] > 0:
            assert 0.1 < want.mean() < 0.95
        for dt in (vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)):
            assert np.array_equal(dt.balls(c, rad), want)
        # one voxel, whose record is the root
        one = vg.HostTree.from_voxels(vox[:1])
        assert np.array_equal(vg.DeviceTree(one.ptr).balls(c, rad), orc.ball_batch(one.ptr, c, rad)[0])
    finally:
        vg.set_voxel_size((1, 1, 1))
        orc.set_voxel((1, 1, 1))


@pytest.mark.parametrize("n", [1, 2432, 2433, 4865, 9728, 38913, 38912, 77825])
def test_batches_of_every_lane_count(n):
    """Batches that fill one, two, ... all of a warp's lanes."""
    import voxvision_gb300 as vg
    vox = _voxels(5, (1, 1, 1), (0, 0, 0))
    ht = vg.HostTree.from_voxels(vox)
    dt = vg.DeviceTree(ht.ptr)
    box = vox.min(0).astype(np.float64), vox.max(0).astype(np.float64) + 1
    o, d = (np.resize(x, (n, 3)) for x in _family("plain", 9, box, np.ones(3)))
    c, rad = _balls("plain", 11, box, np.ones(3))
    c, rad = np.resize(c, (n, 3)), np.resize(rad, n)
    leaf, slot, pts = dt.rays(o, d)
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
    assert same_points(pts, opts, leaf != MISS)[0]
    assert np.array_equal(dt.balls(c, rad), orc.ball_batch(ht.ptr, c, rad)[0])
