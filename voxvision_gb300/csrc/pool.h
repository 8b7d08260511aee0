/* pool.h -- stream-ordered device memory of the library's own: host code. */
#ifndef VOX_POOL_H
#define VOX_POOL_H

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>

/* Stream-ordered memory of the current device, freed with cudaFreeAsync (or
 * cudaFree once nothing uses it): the library's scratch and the trees it builds.
 * It comes from a pool of the library's own, one to a device, that keeps up to
 * POOL_KEEP bytes across synchronisations, where the default pool gives
 * everything back and maps it anew: five 16 MB buffers allocated, freed and
 * synchronised cost 20 us against 240-390, a build's 37 MB image and its map and
 * status 10 us against 190.  What a device's pool keeps goes back when the last
 * tree on that device is freed (tree_gone): a program that holds one tree at a
 * time, freed before the next is built, maps its memory anew for each, and one
 * that builds the next first does not. */
constexpr uint64_t POOL_KEEP = 512ull << 20;
cudaError_t pool_alloc(void **p, size_t bytes, cudaStream_t s);

/* Waits until the current device has done all that was enqueued before, in any
 * stream.  By cudaFree, which does, of 4 bytes: where a thread of the program
 * captures a stream (a batch being made is one, in
 * cudaStreamCaptureModeThreadLocal), cudaDeviceSynchronize is an error in every
 * thread and ends the capture.  2 us with cudaMalloc, as the device keeps
 * another 4 bytes until its last tree is gone: without, both map and unmap 2 MB
 * (a 256^3 raw volume that takes another's place 1,530 us instead of 1,345). */
cudaError_t wait_for_device();

/* A tree handle for `device` is made; it is gone, its memory freed. */
void tree_made(int device);
void tree_gone(int device);

#endif
