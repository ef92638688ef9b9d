// dnl_pool.h - device memory of the engines and of the network calls, from one
// stream-ordered pool per device that keeps what they give back.
//
// cudaMalloc and cudaFree cost 0.1 to 1.4 ms each, by the host, and the device
// waits for cudaFree; a small model's life (create, a few thousand increments,
// read, destroy) has six to a dozen of them.  Creating and destroying the
// 800-quad model took 1.5 ms and takes 0.35, an epoch on 400,000 pairs and its
// predictions 4.75 ms and 2.85.  The pool (cudaMemPool) holds at most
// DNL_POOL_KEEP bytes that nobody uses, the driver returns what is above at the
// next synchronisation, and hands blocks from stream to stream in the order of
// the streams' work.  dnl_release_memory (dnl_pool_release) gives back what
// nobody uses, and so does an allocation that fails, before it tries once more.
// Thread-safe, as the driver's pools are.  Blocks above
// DNL_POOL_LARGEST are cudaMalloc's: a pool that has to grow by some 500 MB is
// slower than cudaMalloc (FP64 bar of 153,600 hexahedra, creation 3.0 against
// 4 to 6 ms).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

constexpr size_t DNL_POOL_KEEP = 256u << 20, DNL_POOL_LARGEST = 64u << 20;

// bytes of device memory of the current device for work on `stream` (and, once
// that has been waited for, on any other)
cudaError_t dnl_pool_alloc(void **p, size_t bytes, cudaStream_t stream);
// given back when the work queued on `stream` has completed
void dnl_pool_free(void *p, cudaStream_t stream);
// what the current device's pool keeps, given back to the device (waits for it)
cudaError_t dnl_pool_release(void);
