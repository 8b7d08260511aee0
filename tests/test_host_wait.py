"""The host's wait for a kernel's store (host_wait.cpp) over a host stand-in
for the CUDA runtime: blocked, yielding or reading in a loop as the device's
scheduling flag says, and an error where the work ends without the store."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxvision_gb300", "csrc")
AUTO, SPIN, YIELD, BLOCKING = 0, 1, 2, 4
NOT_READY, UNKNOWN, FAULT = 600, 999, 700
FAKE = r'''
#include "host_wait.h"
#include <sched.h>
static uint32_t word;
static unsigned flags;
static int after_queries, after_yields, stores = 1, fault;
static int queries, syncs, yields;
extern "C" {
cudaError_t cudaGetDeviceFlags(unsigned *f) { *f = flags | cudaDeviceMapHost; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    syncs++;
    if (fault) return (cudaError_t)fault;
    if (stores) word = 7;
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t)
{
    if (fault) return (cudaError_t)fault;
    if (++queries < after_queries) return cudaErrorNotReady;
    if (stores) word = 7;
    return cudaSuccess;
}
int sched_yield(void) noexcept
{
    if (++yields == after_yields) word = 7;
    return 0;
}
int wait(unsigned f, int at_query, int at_yield, int store, int error, uint32_t start)
{
    flags = f; after_queries = at_query; after_yields = at_yield; stores = store; fault = error;
    queries = syncs = yields = 0;
    word = start;
    unsigned schedule = 0;
    if (cudaError_t e = wait_schedule(&schedule)) return (int)e;
    return (int)wait_for_word(&word, 7, schedule, nullptr);
}
int n_queries() { return queries; }
int n_syncs() { return syncs; }
int n_yields() { return yields; }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    d = tmp_path_factory.mktemp("wait")
    src, so = d / "fake.cpp", d / "wait.so"
    src.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", inc, str(src),
                    os.path.join(CSRC, "host_wait.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def test_blocking_programs_block(lib):
    assert lib.wait(BLOCKING, 10 ** 6, 0, 1, 0, 0) == 0
    assert (lib.n_syncs(), lib.n_queries(), lib.n_yields()) == (1, 0, 0)
    assert lib.wait(BLOCKING, 1, 0, 0, 0, 0) == UNKNOWN          # the work ended without the store
    assert lib.wait(BLOCKING, 1, 0, 1, FAULT, 0) == FAULT


def test_yielding_programs_yield(lib):
    assert lib.wait(YIELD, 10 ** 6, 5, 1, 0, 0) == 0
    assert (lib.n_syncs(), lib.n_queries(), lib.n_yields()) == (0, 0, 5)


@pytest.mark.parametrize("flag", [AUTO, SPIN])
def test_others_read_in_a_loop(lib, flag):
    assert lib.wait(flag, 3, 0, 1, 0, 0) == 0
    assert (lib.n_syncs(), lib.n_queries(), lib.n_yields()) == (0, 3, 0)
    assert lib.wait(flag, 3, 0, 0, 0, 0) == UNKNOWN
    assert lib.wait(flag, 3, 0, 1, FAULT, 0) == FAULT


def test_a_word_already_there(lib):
    assert lib.wait(BLOCKING, 10 ** 6, 0, 0, FAULT, 7) == 0
    assert (lib.n_syncs(), lib.n_queries(), lib.n_yields()) == (0, 0, 0)
