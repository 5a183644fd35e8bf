// Device memory of the engine, functionals, minimisers and networks: cudaMalloc, or, in a
// thread that has been given one, a stream-ordered pool.
//
// cudaFree waits for the whole device, so a worker of a batch that ended a
// problem stopped for every other worker's kernels (batch.cu has the figures).
// The pool belongs to the caller that made it (one batch call), keeps what its
// threads free until then, up to a sixteenth of the device's memory, and never
// makes a stream wait for another one's work (no internal dependencies).  What
// the pools of running calls hold unused is given back before any allocation
// here fails, whichever call or thread asks; memory freed on a stream counts
// as unused once that stream has been waited for, so a thread waits for its own
// after each object's life (batch.cu: after each problem).  An allocation ends with
// a synchronisation of its stream: some first uses are copies on other streams.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

namespace deft {

struct ThreadPool {
  cudaMemPool_t pool = nullptr;  // null: cudaMalloc and cudaFree
  cudaStream_t stream = nullptr;
};
// The calling thread's; memory is freed by the thread that allocated it, before
// that thread's pool is taken away.
inline thread_local ThreadPool thread_pool;
// Set when an allocation of the calling thread did not fit.
inline thread_local bool thread_out_of_memory = false;

// The pools of the calls that are running.
struct CallPools {
  std::mutex mu;
  std::vector<cudaMemPool_t> pools;
  // Gives back what they hold unused; false when there are none.
  bool trim() {
    std::lock_guard<std::mutex> lock(mu);
    for (cudaMemPool_t p : pools) cudaMemPoolTrimTo(p, 0);
    return !pools.empty();
  }
};
inline CallPools &call_pools() {
  static CallPools p;
  return p;
}

inline cudaError_t dev_malloc(void **p, size_t n) {
  const ThreadPool &t = thread_pool;
  auto get = [&]() {
    return t.pool && n ? cudaMallocFromPoolAsync(p, n, t.pool, t.stream) : cudaMalloc(p, n);
  };
  *p = nullptr;
  cudaError_t e = get();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (t.pool) cudaStreamSynchronize(t.stream);
    if (call_pools().trim()) e = get();
    if (e == cudaErrorMemoryAllocation) thread_out_of_memory = true;
  }
  if (e != cudaSuccess || !t.pool || n == 0) return e;
  if ((e = cudaStreamSynchronize(t.stream)) != cudaSuccess) {
    cudaFreeAsync(*p, t.stream);  // callers keep no pointer of a failed allocation
    *p = nullptr;
  }
  return e;
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
  size_t unused = 0, total = 0;
  cudaMemGetInfo(&unused, &total);
  uint64_t keep = total / 16;
  int no = 0;
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
  std::lock_guard<std::mutex> lock(call_pools().mu);
  call_pools().pools.push_back(pool);
  return pool;
}
// Ends a pool whose memory has all been freed.
inline void end_call_pool(cudaMemPool_t pool) {
  if (!pool) return;
  {
    std::lock_guard<std::mutex> lock(call_pools().mu);
    std::vector<cudaMemPool_t> &v = call_pools().pools;
    v.erase(std::remove(v.begin(), v.end(), pool), v.end());
  }
  cudaMemPoolDestroy(pool);
}

}  // namespace deft
