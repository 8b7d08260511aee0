"""Trees and rays at every scale, down to where quotients lose their last
bits: leaf, voxel and point bits are the oracle's, and balls' answers too."""
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
    yield m
    m.set_voxel_size((1, 1, 1))
    orc.set_voxel((1, 1, 1))


def _cells(seed):
    r = np.random.RandomState(seed)
    g = np.argwhere(r.random_sample((18, 17, 16)) < 0.15)
    cube = np.argwhere(np.ones((5, 5, 5))) + (3, 8, 2)
    return np.unique(np.concatenate([g, cube]), axis=0) - (9, 8, 8)


def _rays(kind, unit, seed, n=30000):
    """Lattice rays (many points on faces and edges), rays between any points, and rays from lattice points."""
    r = np.random.RandomState(seed)
    if kind == "lattice":
        o = r.randint(-10, 11, (n, 3)) * unit
        d = r.randint(1, 8, (n, 3)) * r.choice([-1.0, 1.0], (n, 3)) * 2.0 ** r.randint(-4, 5, (n, 1))
    elif kind == "any":
        o = r.uniform(-14, 14, (n, 3)) * unit
        d = r.standard_normal((n, 3))
    else:   # a lattice point a hair off zero or off a face, long and short directions
        o = r.randint(-10, 11, (n, 3)) * unit
        o += np.where(r.random_sample((n, 3)) < 0.3, r.choice([1e-44, -1e-44, 1e-38, -1e-30, 1e-25], (n, 3)), 0.0)
        d = r.randint(1, 8, (n, 3)) * r.choice([-1.0, 1.0], (n, 3)) * 2.0 ** r.randint(-28, 17, (n, 3))
    return np.ascontiguousarray(o.astype(np.float32)), np.ascontiguousarray(d.astype(np.float32))


@pytest.mark.parametrize("exponent", [-145, -130, -122, -115, -104, -99, -96, -92, -88, -75, -69, -66, -62, -57, -45, -30,
                                      0, 30, 50, 57])
@pytest.mark.parametrize("kind", ["lattice", "any", "hair"])
def test_scales(vg, kind, exponent):
    unit = 2.0 ** exponent
    vg.set_voxel_size((unit,) * 3)
    orc.set_voxel((unit,) * 3)
    vox = np.ascontiguousarray((_cells(5) * unit).astype(np.float32))
    ht = vg.HostTree.from_voxels(vox)
    o, d = _rays(kind, unit, exponent + 200)
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    assert (oleaf != MISS).any()
    for dt in (vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)):
        leaf, slot, pts = dt.rays(o, d)
        assert np.array_equal(leaf, oleaf), f"{(leaf != oleaf).sum()} leaf ids differ"
        assert np.array_equal(slot, oslot)
        ok, bad = same_points(pts, opts, leaf != MISS)
        assert ok, f"{bad} points differ"
        c, rad = o[:8192], np.abs(d[:8192, 0]) * np.float32(unit)
        assert np.array_equal(dt.balls(c, rad), orc.ball_batch(ht.ptr, c, rad)[0])


@pytest.mark.parametrize("unit", [2.0 ** -27, 2.0 ** -26, 1.0])
@pytest.mark.parametrize("kind", ["directions", "origins", "voxels"])
def test_bounds_of_the_mirrored_search(vg, kind, unit):
    """Numbers at, just inside and just outside each bound that sends a ray or an image to the general search."""
    r = np.random.RandomState(17)
    vg.set_voxel_size((unit,) * 3)
    orc.set_voxel((unit,) * 3)
    vox = (_cells(5) * unit).astype(np.float32)
    o, d = _rays("any", unit, 23)
    n = len(o)

    def edges(*values):   # each, and its neighbours on both sides, either sign
        v = np.array(values, np.float32)[r.randint(0, len(values), n)]
        return np.nextafter(v, np.array([0, 1, 1e30], np.float32)[r.randint(0, 3, n)]) * r.choice([-1, 1], n).astype(np.float32)

    at = np.arange(n), r.randint(0, 3, n)
    if kind == "directions":
        d[at] = edges(2.0 ** -22, 2.0 ** 18, 2.0 ** -30, 2.0 ** 20)
    elif kind == "origins":
        o[at] = edges(2.0 ** -79, 2.0 ** -102, 2.0 ** -126, 2.0 ** 60)
    else:
        few = r.choice(len(vox), 40, replace=False)
        vox[few, r.randint(0, 3, 40)] = edges(2.0 ** -79, 2.0 ** -55)[:40]
    vox = np.ascontiguousarray(vox)
    ht = vg.HostTree.from_voxels(vox)
    oleaf, oslot, opts, _ = orc.ray_batch(ht.ptr, o, d)
    for dt in (vg.DeviceTree(ht.ptr), vg.DeviceTree.build(vox)):
        leaf, slot, pts = dt.rays(o, d)
        assert np.array_equal(leaf, oleaf) and np.array_equal(slot, oslot)
        ok, bad = same_points(pts, opts, leaf != MISS)
        assert ok, f"{bad} points differ"
        c, rad = o[:8192], np.abs(d[:8192, 0]) * np.float32(unit)
        assert np.array_equal(dt.balls(c, rad), orc.ball_batch(ht.ptr, c, rad)[0])
