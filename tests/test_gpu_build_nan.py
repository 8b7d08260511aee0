"""Builds of sets with a coordinate that is not a number, in every size class:
the host build's image but for the NaNs' payloads.  (A first voxel that is NaN
stays its node's bound, as in the scan of tree.c:138-155; a later one is never
less or greater than one.)"""
import ctypes as C

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
    m.set_voxel_size((1, 1, 1))
    return m


def _same(a, b):
    if a.shape != b.shape:
        return False
    fa, fb = a.view(np.float32), b.view(np.float32)
    return bool(((a == b) | (np.isnan(fa) & np.isnan(fb))).all())


@pytest.mark.parametrize("n", [2, 7, 8, 9, 32, 33, 100, 128, 129, 1000, 1025, 8000, 8193, 30000, 40000])
@pytest.mark.parametrize("where", [0, 1, "middle", "last", "all"])
@pytest.mark.parametrize("value", [np.nan, -np.inf, np.inf])
def test_not_a_number(vg, n, where, value):
    r = np.random.RandomState(n)
    side = max(3, int(round((4 * n) ** (1 / 3))))
    vox = r.choice(side ** 3, n, replace=False)
    vox = np.stack([vox // side // side, vox // side % side, vox % side], 1).astype(np.float32)
    if where == "all":
        vox[:, 1] = value
    else:
        vox[{"middle": n // 2, "last": n - 1}.get(where, where), 1] = value
    vox = np.ascontiguousarray(vox)
    copy = vox.copy()
    ht = vg.HostTree(vg.lib().vox_make_tree_host(copy.ctypes.data_as(C.c_void_p), len(copy)))
    (hu, hi), (du, di) = vg.DeviceTree(ht.ptr).image(), vg.DeviceTree.build(vox).image()
    assert np.array_equal(hi, di) and _same(hu, du)
