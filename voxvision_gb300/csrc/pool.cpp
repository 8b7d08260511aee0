/* pool.cpp -- see pool.h. */
#include "pool.h"

#include <atomic>
#include <mutex>

namespace {

constexpr int POOL_DEVICES = 64;
std::mutex g_pool_mu;
std::atomic<cudaMemPool_t> g_pool[POOL_DEVICES];
std::atomic<int> g_trees[POOL_DEVICES];
std::atomic<void *> g_anchor[POOL_DEVICES];   // of wait_for_device

}  // namespace

cudaError_t pool_alloc(void **p, size_t bytes, cudaStream_t s)
{
    *p = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = dev < POOL_DEVICES ? g_pool[dev].load() : nullptr;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!pool && dev < POOL_DEVICES && cudaStreamIsCapturing(s, &cap) == cudaSuccess &&
        cap == cudaStreamCaptureStatusNone) {   // (no pool is made inside a capture)
        std::lock_guard<std::mutex> lock(g_pool_mu);
        pool = g_pool[dev].load();
        if (!pool) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            uint64_t keep = POOL_KEEP;
            if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
                cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
                g_pool[dev].store(pool);
            } else {
                pool = nullptr;
                cudaGetLastError();
            }
        }
    }
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

cudaError_t wait_for_device()
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < POOL_DEVICES && !g_anchor[dev].load()) {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        void *a = nullptr;
        if (!g_anchor[dev].load() && cudaMalloc(&a, 4) == cudaSuccess) g_anchor[dev].store(a);
    }
    void *p = nullptr;
    e = cudaMalloc(&p, 4);
    return e != cudaSuccess ? e : cudaFree(p);
}

void tree_made(int device)
{
    if (device >= 0 && device < POOL_DEVICES) g_trees[device]++;
}

void tree_gone(int device)
{
    if (device < 0 || device >= POOL_DEVICES || --g_trees[device] != 0) return;
    if (cudaMemPool_t pool = g_pool[device].load()) cudaMemPoolTrimTo(pool, 0);
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (void *a = g_anchor[device].exchange(nullptr)) cudaFree(a);
}
