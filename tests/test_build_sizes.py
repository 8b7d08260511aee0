"""What a tree build sets aside (build_sizes.h), on the host: enough for every
way a set can fall into nodes, and in proportion to the set's size."""
import ctypes as C
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxvision_gb300", "csrc")
MOST = 2 ** 31 - 1
HIGH = 32768
SOURCE = r'''
#include "build_sizes.h"
using namespace build_sizes;
extern "C" void sizes(uint64_t n, uint64_t *out)
{
    const Sizes s(n);
    const uint64_t v[] = {s.tiny, s.small, s.low, s.mid, s.high, s.tiled, s.tiles, s.subs, s.chunks, s.window, s.scratch()};
    for (int i = 0; i < 11; i++) out[i] = v[i];
}
extern "C" uint64_t level_bound(uint64_t n, uint64_t m, int subs) { return subs ? Sizes(n).subs_of(m) : Sizes(n).tiles_of(m); }
extern "C" uint32_t shift_of(uint32_t n) { return tile_shift(n); }
extern "C" uint32_t parts_of(uint32_t n, uint32_t shift) { return parts(n, shift); }
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sizes")
    src, so = d / "s.cpp", d / "s.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    m = C.CDLL(str(so))
    m.sizes.argtypes = [C.c_uint64, C.c_void_p]
    m.level_bound.argtypes, m.level_bound.restype = [C.c_uint64, C.c_uint64, C.c_int], C.c_uint64
    m.shift_of.argtypes, m.shift_of.restype = [C.c_uint32], C.c_uint32
    m.parts_of.argtypes, m.parts_of.restype = [C.c_uint32, C.c_uint32], C.c_uint32
    return m


def _sizes(lib, n):
    v = (C.c_uint64 * 11)()
    lib.sizes(n, v)
    return dict(zip(("tiny", "small", "low", "mid", "high", "tiled", "tiles", "subs", "chunks", "window", "scratch"), v))


@pytest.mark.parametrize("n", [1, 1000, HIGH, HIGH + 1, 10 ** 5, 10 ** 6, 2 ** 22 + 1, 2 ** 24 + 1, 2 ** 26 + 1, 10 ** 8,
                               2 ** 29, 2 ** 30, MOST])
def test_memory_is_in_proportion(lib, n):
    # 50 bytes a voxel was a build's scratch when each voxel had its own counts; the voxels' two orders take 24 of them
    s = _sizes(lib, n)
    assert s["scratch"] + 24 * n <= 40 * n + (1 << 20), (s["scratch"] + 24 * n) / n


@pytest.mark.parametrize("n", [HIGH + 1, HIGH + 2, 2 ** 22, 2 ** 22 + 1, 2 ** 23 + 1, 2 ** 26, 2 ** 30 + 5, MOST])
def test_a_nodes_tiles(lib, n):
    shift = lib.shift_of(n)
    assert 11 <= shift and lib.parts_of(n, shift) <= 2048 and lib.parts_of(n, shift) == -(-n // (1 << shift))
    assert shift == 11 or lib.parts_of(n, shift - 1) > 2048   # the smallest that does


@pytest.mark.parametrize("n", [HIGH + 1, 10 ** 5, 10 ** 6, 2 ** 24 + 1, 2 ** 27, 2 ** 30, MOST])
@pytest.mark.parametrize("how", ["one", "least", "halves", "spread"])
def test_every_level_fits(lib, n, how):
    r = random.Random(n)
    if how == "one":
        nodes = [n]
    elif how == "least":
        nodes = [HIGH + 1] * min(n // (HIGH + 1), 70000)
    elif how == "halves":
        nodes, left = [], n
        while left // 2 > HIGH:
            nodes.append(left // 2)
            left -= left // 2
    else:
        nodes, left = [], n
        while left > HIGH and len(nodes) < 3000:
            nodes.append(min(left, r.randint(HIGH + 1, max(HIGH + 1, n // 50))))
            left -= nodes[-1]
    s = _sizes(lib, n)
    tiles = sum(lib.parts_of(k, lib.shift_of(k)) for k in nodes)
    subs = sum(lib.parts_of(k, 11) for k in nodes)
    assert len(nodes) <= s["tiled"] < 1 << 16
    for bound in (s["tiles"], lib.level_bound(n, len(nodes), 0)):
        assert tiles <= bound < 1 << 24
    for bound in (s["subs"], lib.level_bound(n, len(nodes), 1)):
        assert subs <= bound < 1 << 24
    assert s["chunks"] == 2 * s["subs"]
