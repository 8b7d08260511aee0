/* host_wait.cpp -- see host_wait.h. */
#include "host_wait.h"

#include <sched.h>

cudaError_t wait_schedule(unsigned *schedule)
{
    unsigned flags = 0;
    const cudaError_t e = cudaGetDeviceFlags(&flags);
    *schedule = flags & cudaDeviceScheduleMask;
    return e;
}

cudaError_t wait_for_word(const uint32_t *word, uint32_t value, unsigned schedule, cudaStream_t s)
{
    const auto there = [&] { return __atomic_load_n(word, __ATOMIC_ACQUIRE) == value; };
    if (there()) return cudaSuccess;
    if (schedule == cudaDeviceScheduleBlockingSync) {
        const cudaError_t e = cudaStreamSynchronize(s);
        return e != cudaSuccess ? e : there() ? cudaSuccess : cudaErrorUnknown;
    }
    for (uint32_t spin = 1;; spin++) {
        if (there()) return cudaSuccess;
        if (spin % 1024 == 0) {
            const cudaError_t e = cudaStreamQuery(s);
            if (e == cudaSuccess) return there() ? cudaSuccess : cudaErrorUnknown;
            if (e != cudaErrorNotReady) return e;
        }
        if (schedule == cudaDeviceScheduleYield) sched_yield();
    }
}
