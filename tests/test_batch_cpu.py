"""The host side of a batch (csrc/batch.cu, csrc/dev_mem.h) against a model of
the CUDA runtime: which error a batch reports, that the calling thread
keeps its device, and that memory its pool holds unused is there for others.
The sources are compiled with g++ against the few calls they make; no GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# a device of 100 bytes with stream-ordered pools: what has been freed on a
# stream is available once that stream has been waited for
RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdint>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
struct Stream; struct Pool;
typedef Stream *cudaStream_t;
typedef Pool *cudaMemPool_t;
enum { cudaMemAllocationTypePinned = 1, cudaMemHandleTypeNone = 0, cudaMemLocationTypeDevice = 1 };
struct cudaMemPoolProps { int allocType, handleTypes; struct { int type, id; } location; };
enum cudaMemPoolAttr { cudaMemPoolAttrReleaseThreshold, cudaMemPoolReuseAllowInternalDependencies };
cudaError_t cudaGetDeviceCount(int *);
cudaError_t cudaGetDevice(int *);
cudaError_t cudaSetDevice(int);
cudaError_t cudaMalloc(void **, size_t);
cudaError_t cudaFree(void *);
cudaError_t cudaMallocFromPoolAsync(void **, size_t, cudaMemPool_t, cudaStream_t);
cudaError_t cudaFreeAsync(void *, cudaStream_t);
cudaError_t cudaStreamSynchronize(cudaStream_t);
cudaError_t cudaMemPoolCreate(cudaMemPool_t *, const cudaMemPoolProps *);
cudaError_t cudaMemPoolDestroy(cudaMemPool_t);
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *);
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t);
cudaError_t cudaMemGetInfo(size_t *, size_t *);
cudaError_t cudaGetLastError();
"""

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include "BATCH"

struct Stream {};
struct Block { size_t n; Pool *pool; Stream *freed; };  // freed: on which stream, not yet waited for
struct Pool { size_t unused = 0; };
static std::recursive_mutex mu;
static std::map<void *, Block> blocks;
static std::map<Pool *, int> pools;
static size_t used = 0;  // bytes the device has given out (live, being freed, unused in pools)
static const size_t kCapacity = 100;
static uint64_t kept = 0;
static int set_device_calls = 0;
static bool fail_sync = false;
static thread_local bool caller = false;
#define LOCK std::lock_guard<std::recursive_mutex> l(mu)
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { if (caller) set_device_calls++; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { LOCK; *f = kCapacity - used; *t = kCapacity; return cudaSuccess; }
static cudaError_t give(void **p, size_t n, Pool *pool) {
  *p = new char;
  blocks[*p] = {n, pool, nullptr};
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  LOCK;
  if (used + n > kCapacity) return cudaErrorMemoryAllocation;
  used += n;
  return give(p, n, nullptr);
}
cudaError_t cudaFree(void *p) { LOCK; if (p) { used -= blocks[p].n; blocks.erase(p); } return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, Pool *pool, Stream *) {
  LOCK;
  if (pool->unused >= n) { pool->unused -= n; return give(p, n, pool); }
  if (used + n > kCapacity) return cudaErrorMemoryAllocation;
  used += n;
  return give(p, n, pool);
}
cudaError_t cudaFreeAsync(void *p, Stream *s) { LOCK; if (p) blocks[p].freed = s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(Stream *s) {
  LOCK;
  if (fail_sync) return cudaErrorUnknown;
  for (auto it = blocks.begin(); it != blocks.end();)
    if (s && it->second.freed == s) { it->second.pool->unused += it->second.n; it = blocks.erase(it); } else ++it;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(Pool **p, const cudaMemPoolProps *) { LOCK; *p = new Pool; pools[*p] = 1; return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(Pool *p) { LOCK; used -= p->unused; p->unused = 0; pools.erase(p); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(Pool *, cudaMemPoolAttr a, void *v) {
  if (a == cudaMemPoolAttrReleaseThreshold) kept = *(uint64_t *)v;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(Pool *p, size_t) { LOCK; used -= p->unused; p->unused = 0; return cudaSuccess; }

// the C ABI as far as batch.cu uses it; a problem's mu is the status of its
// solve, its kT the device bytes it needs
struct deft_ctx { Stream s; };
struct deft_grid { deft_ctx *c; };
struct deft_fmt { deft_grid *g; void *mem; int status; double R; };
struct deft_cg { deft_fmt *f; };
static std::atomic<bool> waiting(false), done(false);
static void until(std::atomic<bool> &b) {
  for (int i = 0; i < 10000 && !b; i++) std::this_thread::sleep_for(std::chrono::milliseconds(1));
}
static thread_local std::string err;
namespace deft { void set_last_error_message(const std::string &m) { err = m; } }
extern "C" {
const char *deft_last_error(void) { return err.c_str(); }
int deft_ctx_create(int, deft_ctx **o) { *o = new deft_ctx; return 0; }
int deft_ctx_destroy(deft_ctx *c) { delete c; return 0; }
void *deft_ctx_stream(deft_ctx *c) { return &c->s; }
int deft_grid_create(deft_ctx *c, const double *, int, int, int, deft_grid **g) { *g = new deft_grid{c}; return 0; }
int deft_grid_destroy(deft_grid *g) { delete g; return 0; }
int deft_fmt_create(deft_grid *g, const deft_fmt_params *p, deft_fmt **f) {
  void *m = nullptr;
  if (p->R == 2) until(waiting);
  if (p->kT > 0 && deft::dev_malloc(&m, (size_t)p->kT) != cudaSuccess) { err = "memory"; done = true; return DEFT_ERR_NOMEM; }
  if (p->R == 2) done = true;
  *f = new deft_fmt{g, m, (int)p->mu, p->R};
  return 0;
}
int deft_fmt_destroy(deft_fmt *f) { if (f) deft::dev_free(f->mem); delete f; return 0; }
int deft_fmt_set_mask(deft_fmt *, const double *, int) { return 0; }
int deft_fmt_set_vext(deft_fmt *, const double *, int) { return 0; }
int deft_cg_create(deft_fmt *f, const deft_cg_params *, deft_cg **c) { *c = new deft_cg{f}; return 0; }
int deft_cg_destroy(deft_cg *c) { delete c; return 0; }
int deft_cg_set_x(deft_cg *, const double *, int) { return 0; }
int deft_cg_get_x(deft_cg *, double *, int) { return 0; }
int deft_cg_solve(deft_cg *c, deft_cg_status *) {
  if (c->f->R == 1) { waiting = true; until(done); }
  err = "status " + std::to_string(c->f->status); return c->f->status;
}
}

static deft_batch_problem problem(int n, int status, double bytes) {
  deft_batch_problem p{};
  p.N[0] = p.N[1] = p.N[2] = n;
  p.mu = status;
  p.kT = bytes;
  p.R = 0;
  return p;
}
static int batch(std::vector<deft_batch_problem> pr, int workers, std::vector<deft_cg_status> &st, int device = 0) {
  deft_batch_params bp{};
  bp.workers = workers;
  st.resize(pr.size());
  return deft_batch_solve(device, (int)pr.size(), pr.data(), &bp, st.data());
}
#define WANT(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static int errors() {
  std::vector<deft_cg_status> st;
  for (int workers : {1, 4}) {
    // the larger problem runs first; the list's first failure is reported
    WANT(batch({problem(8, 0, 0), problem(8, DEFT_ERR_MAXITER, 0), problem(16, DEFT_ERR_NAN, 0)},
               workers, st) == DEFT_ERR_MAXITER);
    WANT(!strcmp(deft_last_error(), "problem 1: status 5"));
    WANT(st[0].status == 0 && st[1].status == DEFT_ERR_MAXITER && st[2].status == DEFT_ERR_NAN);
    WANT(batch({problem(8, 0, 0), problem(16, 0, 0)}, workers, st) == DEFT_OK);
  }
  return 0;
}
// After a problem of 60 bytes its worker is in another one; 60 bytes are asked
// for by another worker of the call, by another call, and outside any call.
static int memory(const char *who) {
  const std::string w = who;
  std::vector<deft_cg_status> st, st2;
  auto big = problem(16, 0, 60), wait = problem(12, 0, 0), next = problem(8, 0, 60);
  wait.R = 1;  // its solve waits for `done`
  next.R = 2;  // its functional is made once `wait` is being solved
  done = waiting = false;
  int other = -1;
  if (w == "together") {
    // two problems of 60 bytes that the list keeps apart
    next.N[0] = next.N[1] = next.N[2] = 16;
    big.R = 1;
    WANT(batch({big, problem(8, 0, 0), next}, 2, st) == DEFT_OK);
    WANT(st[0].status == 0 && st[1].status == 0 && st[2].status == 0 && used == 0);
    // one that does not fit alone fails, and the others do not
    waiting = done = true;
    WANT(batch({problem(8, 0, 0), problem(16, 0, 160), problem(12, 0, 60)}, 2, st) == DEFT_ERR_NOMEM);
    WANT(!strcmp(deft_last_error(), "problem 1: memory"));
    WANT(st[0].status == 0 && st[1].status == DEFT_ERR_NOMEM && st[2].status == 0);
    return 0;
  }
  if (w == "worker") {
    WANT(batch({big, wait, next}, 2, st) == DEFT_OK);
    return 0;
  }
  std::thread call([&]() { other = batch({big, wait}, 1, st); });
  until(waiting);
  int got;
  if (w == "call") {
    got = batch({next}, 1, st2);
  } else {
    void *p = nullptr;
    got = deft::dev_malloc(&p, 60);
    deft::dev_free(p);
  }
  done = true;
  call.join();
  WANT(got == 0 && other == 0 && used == 0);
  WANT(kept > 0 && kept < kCapacity);  // a bound on what a pool may keep
  return 0;
}
static int failed_wait() {
  // an allocation whose stream fails gives its memory back
  Stream s;
  cudaMemPool_t pool = deft::make_call_pool(0);
  deft::thread_pool = {pool, &s};
  void *p = &s;
  fail_sync = true;
  WANT(deft::dev_malloc(&p, 10) == cudaErrorUnknown && p == nullptr);
  fail_sync = false;
  cudaStreamSynchronize(&s);
  WANT(blocks.empty());
  deft::thread_pool = {};
  deft::end_call_pool(pool);
  return 0;
}
static int caller_device() {
  // a batch on another device than the caller's leaves the caller's thread alone
  std::vector<deft_cg_status> st;
  WANT(batch({problem(8, 0, 10)}, 1, st, 1) == DEFT_OK);
  WANT(set_device_calls == 0);
  return 0;
}
int main(int argc, char **argv) {
  caller = true;
  const std::string s = argv[1];
  return s == "errors" ? errors() : s == "caller_device" ? caller_device()
         : s == "failed_wait" ? failed_wait()
         : s.substr(0, 7) == "memory_" ? memory(argv[1] + 7) : 2;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("batch")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "main.cpp").write_text(PROGRAM.replace(
        "BATCH", os.path.join(ROOT, "deft_gb300", "csrc", "batch.cu")))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(d), str(d / "main.cpp"),
                    "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("scenario", ["errors", "caller_device", "memory_together", "memory_worker", "memory_call",
                                      "memory_alone", "failed_wait"])
def test_batch_host(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
