/* host_wait.h -- the host's wait for a word that a stream's kernel stores into
 * page-locked memory: host code. */
#ifndef VOX_HOST_WAIT_H
#define VOX_HOST_WAIT_H

#include <cuda_runtime_api.h>

#include <cstdint>

/* The current device's scheduling flag (cudaSetDeviceFlags). */
cudaError_t wait_schedule(unsigned *schedule);

/* Waits until *word is `value`, which the work enqueued on s stores; an error
 * when that work ends without it.  Waits as the scheduling flag tells a wait
 * for a stream to: a blocked thread for
 * cudaDeviceScheduleBlockingSync (until all of s's work is done), a thread that
 * yields for cudaDeviceScheduleYield, else one that reads the word in a loop --
 * the store is seen some 8 us before a wait for the stream would return. */
cudaError_t wait_for_word(const uint32_t *word, uint32_t value, unsigned schedule, cudaStream_t s);

#endif
