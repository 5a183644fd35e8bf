// Device memory of the engine, functionals and minimisers: cudaMalloc, or, in a
// thread that has been given one, a stream-ordered pool.
//
// cudaFree waits for the whole device, so a worker of a batch that ended a
// problem stopped for every other worker's kernels (batch.cu has the figures).
// The pool belongs to the caller that made it (one batch call), is told to keep
// what its threads free until then, and never makes a stream wait for another
// one's work (no internal dependencies).  An allocation ends with a
// synchronisation of its stream: some first uses are copies on other streams.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace deft {

struct ThreadPool {
  cudaMemPool_t pool = nullptr;  // null: cudaMalloc and cudaFree
  cudaStream_t stream = nullptr;
};
// The calling thread's; memory is freed by the thread that allocated it, before
// that thread's pool is taken away.
inline thread_local ThreadPool thread_pool;

inline cudaError_t dev_malloc(void **p, size_t n) {
  if (!thread_pool.pool || n == 0) return cudaMalloc(p, n);
  *p = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(p, n, thread_pool.pool, thread_pool.stream);
  if (e == cudaErrorMemoryAllocation) {  // give back what the pool holds unused, once
    cudaGetLastError();
    cudaStreamSynchronize(thread_pool.stream);
    cudaMemPoolTrimTo(thread_pool.pool, 0);
    e = cudaMallocFromPoolAsync(p, n, thread_pool.pool, thread_pool.stream);
  }
  return e == cudaSuccess ? cudaStreamSynchronize(thread_pool.stream) : e;
}
inline cudaError_t dev_free(void *p) {
  if (!p) return cudaSuccess;
  return thread_pool.pool ? cudaFreeAsync(p, thread_pool.stream) : cudaFree(p);
}

// A pool on `device` for one call's threads (null where it cannot be made).
inline cudaMemPool_t make_call_pool(int device) {
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  uint64_t keep = UINT64_MAX;
  int no = 0;
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
  return pool;
}

}  // namespace deft
