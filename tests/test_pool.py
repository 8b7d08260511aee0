"""The library's device memory pools (pool.cpp) over a host stand-in for the
CUDA runtime with several devices: one pool to a device, made outside captures,
its memory kept between calls and given back when that device's last tree is
freed, whatever the others hold."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxvision_gb300", "csrc")
FAKE = r'''
#include "pool.h"
#include <cstdlib>
#include <map>
static int blocks[4], waits, broken;
static std::map<void *, int> owner;
static int current = 0, refuse = 0, capturing = 0;
static long made[4], trimmed[4], kept[4], from_pool[4], from_default;
static uint64_t threshold[4];
struct Pool { int dev; };
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c)
{
    *c = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *props)
{
    if (refuse) return cudaErrorNotSupported;
    made[props->location.id]++;
    *p = reinterpret_cast<cudaMemPool_t>(new Pool{props->location.id});
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr, void *v)
{
    threshold[reinterpret_cast<Pool *>(p)->dev] = *static_cast<uint64_t *>(v);
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t)
{
    const int d = reinterpret_cast<Pool *>(pool)->dev;
    from_pool[d]++;
    kept[d] += n;
    *p = std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t, cudaStream_t) { from_default++; *p = std::malloc(1); return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t least)
{
    const int d = reinterpret_cast<Pool *>(pool)->dev;
    trimmed[d]++;
    if (least == 0) kept[d] = 0;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t)
{
    if (broken) return (cudaError_t)broken;
    *p = std::malloc(1);
    blocks[current]++;
    owner[*p] = current;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (p) { blocks[owner[p]]--; waits++; std::free(p); }
    return (cudaError_t)broken;
}
cudaError_t cudaDeviceSynchronize() { return cudaErrorStreamCaptureUnsupported; }   // as while any thread captures
int wait_device(int error)
{
    broken = error;
    waits = 0;
    const int e = (int)wait_for_device();
    broken = 0;
    return e;
}
int n_waits() { return waits; }
int n_blocks(int d) { return blocks[d]; }
void set_device(int d) { current = d; }
void set_refuse(int r) { refuse = r; }
void set_capturing(int c) { capturing = c; }
int alloc(size_t n) { void *p; return (int)pool_alloc(&p, n, nullptr); }
void made_tree(int d) { tree_made(d); }
void gone_tree(int d) { tree_gone(d); }
long pools(int d) { return made[d]; }
long held(int d) { return kept[d]; }
long trims(int d) { return trimmed[d]; }
long pooled(int d) { return from_pool[d]; }
long unpooled() { return from_default; }
uint64_t keeps(int d) { return threshold[d]; }
}
'''


@pytest.fixture
def pool(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    src, so = tmp_path / "fake.cpp", tmp_path / "pool.so"
    src.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", inc, str(src),
                    os.path.join(CSRC, "pool.cpp"), "-o", str(so), "-lpthread"], check=True)
    m = C.CDLL(str(so))
    m.alloc.argtypes, m.keeps.restype = [C.c_size_t], C.c_uint64
    for f in (m.pools, m.held, m.trims, m.pooled, m.unpooled):
        f.restype = C.c_long
    return m


def test_each_device_gives_back_its_own(pool):
    for d in (0, 1):
        pool.set_device(d)
        for _ in range(3):
            assert pool.alloc(1000) == 0
        pool.made_tree(d)
    pool.made_tree(1)
    assert [pool.pools(d) for d in (0, 1)] == [1, 1] and [pool.held(d) for d in (0, 1)] == [3000, 3000]
    assert pool.keeps(0) == 512 << 20
    pool.set_device(2)           # whichever device is current
    pool.gone_tree(0)            # the last of device 0, with trees left on device 1
    assert pool.held(0) == 0 and pool.held(1) == 3000
    pool.gone_tree(1)
    assert pool.held(1) == 3000  # one left
    pool.gone_tree(1)
    assert pool.held(1) == 0


def test_a_device_without_a_pool_is_not_trimmed(pool):
    pool.made_tree(3)            # an uploaded tree
    pool.gone_tree(3)
    assert pool.pools(3) == 0 and pool.trims(3) == 0


def test_no_pool_is_made_in_a_capture_or_where_none_can_be(pool):
    pool.set_capturing(1)
    assert pool.alloc(10) == 0 and pool.pools(0) == 0 and pool.unpooled() == 1
    pool.set_capturing(0)
    pool.set_refuse(1)
    assert pool.alloc(10) == 0 and pool.unpooled() == 2
    pool.set_refuse(0)
    assert pool.alloc(10) == 0 and pool.pools(0) == 1 and pool.pooled(0) == 1
    pool.set_capturing(1)        # a pool there is serves captures too
    assert pool.alloc(10) == 0 and pool.pooled(0) == 2


def test_waiting_for_a_device_in_spite_of_captures(pool):
    pool.set_device(1)
    pool.made_tree(1)
    for _ in range(3):
        assert pool.wait_device(0) == 0 and pool.n_waits() == 1   # a block made and freed
        assert pool.n_blocks(1) == 1                              # beside the one that is kept
    assert pool.wait_device(700) == 700
    pool.set_device(0)
    pool.gone_tree(1)
    assert pool.n_blocks(1) == 0 and pool.n_blocks(0) == 0
    pool.made_tree(0)
    assert pool.wait_device(0) == 0 and (pool.n_blocks(0), pool.n_blocks(1)) == (1, 0)
    pool.gone_tree(0)
    assert pool.n_blocks(0) == 0
