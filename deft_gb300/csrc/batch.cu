// Batched solves (many independent state points and uneven grids on one
// GPU).  Worker host threads each own a context (one CUDA stream) and pull
// problems from a shared counter; a worker keeps one grid (engine, FFT plans,
// weight tables, work spectra) per grid shape and lattice it has met, so a
// sweep over a few sizes plans each size once per worker.  Kernels of
// different problems run concurrently on the workers' streams; every solve
// is the same minimiser deft_cg_solve runs on its own.
//
// Set-up and clean-up must not stop the other workers: the call's device memory
// comes from a pool of its own (dev_mem.h), and the largest problems are started
// first.  12 solves of 32^3 to 96^3 on 8 workers: 64 ms with cudaMalloc and
// cudaFree in order of the list (49 when nothing was freed), 43 like this; on one
// worker 82 and 73.  Problems that do not fit beside the others run one by one at
// the end.
#include "../../include/deft_gb300.h"
#include "dev_mem.h"

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstring>
#include <functional>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

namespace deft {
void set_last_error_message(const std::string &m);
}

namespace {

struct GridKey {
  int N[3];
  double lat[9];
  bool operator==(const GridKey &o) const {
    return memcmp(N, o.N, sizeof(N)) == 0 && memcmp(lat, o.lat, sizeof(lat)) == 0;
  }
};

struct Worker {
  deft_ctx *ctx = nullptr;
  std::vector<std::pair<GridKey, deft_grid *>> grids;

  deft_grid *grid_for(const deft_batch_problem &p, int *status) {
    GridKey k;
    memcpy(k.N, p.N, sizeof(k.N));
    memcpy(k.lat, p.lat, sizeof(k.lat));
    for (auto &e : grids)
      if (e.first == k) return e.second;
    deft_grid *g = nullptr;
    *status = deft_grid_create(ctx, p.lat, p.N[0], p.N[1], p.N[2], &g);
    if (*status) return nullptr;
    grids.push_back({k, g});
    return g;
  }

  ~Worker() {
    for (auto &e : grids) deft_grid_destroy(e.second);
    if (ctx) deft_ctx_destroy(ctx);
  }
};

int solve_one(Worker &w, const deft_batch_problem &p, const deft_cg_params &cgp,
              deft_cg_status *st) {
  int s = DEFT_OK;
  deft_grid *g = w.grid_for(p, &s);
  if (!g) return s;
  deft_fmt_params fp{};
  fp.functional = p.functional;
  fp.R = p.R;
  fp.kT = p.kT;
  fp.mu = p.mu;
  fp.terms = p.terms;
  fp.precision = p.precision;
  deft_fmt *f = nullptr;
  if ((s = deft_fmt_create(g, &fp, &f))) return s;
  deft_cg *cg = nullptr;
  if (!s && p.mask) s = deft_fmt_set_mask(f, p.mask, 0);
  if (!s && p.V) s = deft_fmt_set_vext(f, p.V, 0);
  if (!s) {
    s = deft_cg_create(f, &cgp, &cg);
    if (s == DEFT_ERR_ARG && cgp.preconditioned == DEFT_PC_STRUCTURE) {
      // a grid or functional the structure preconditioner does not take
      deft_cg_params c2 = cgp;
      c2.preconditioned = DEFT_PC_DENSITY;
      s = deft_cg_create(f, &c2, &cg);
    }
  }
  if (!s) s = deft_cg_set_x(cg, p.n_init, 0);
  if (!s) s = deft_cg_solve(cg, st);
  if (!s && p.n_out) s = deft_cg_get_x(cg, p.n_out, 0);
  deft_cg_destroy(cg);
  deft_fmt_destroy(f);
  return s;
}

}  // namespace

extern "C" int deft_batch_solve(int device, int count, const deft_batch_problem *probs,
                                const deft_batch_params *bp, deft_cg_status *status_out) {
  if (count < 0 || (count && (!probs || !bp || !status_out))) return DEFT_ERR_ARG;
  if (count == 0) return DEFT_OK;
  int workers = bp->workers > 0 ? bp->workers : 8;
  if (workers > count) workers = count > 0 ? count : 1;
  std::atomic<int> next(0);
  // the first failing problem of the list, whatever order they ran in
  std::mutex err_mu;
  int first_index = INT_MAX, first_error = DEFT_OK;
  std::string first_msg;
  auto failed = [&](int index, int status, const std::string &msg) {
    std::lock_guard<std::mutex> lock(err_mu);
    if (index >= first_index) return;
    first_index = index;
    first_error = status;
    first_msg = msg;
  };
  // largest first (a large one started last would run alone at the end)
  std::vector<int> order(count);
  std::iota(order.begin(), order.end(), 0);
  auto points = [&](int i) {
    return (double)probs[i].N[0] * (double)probs[i].N[1] * (double)probs[i].N[2];
  };
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return points(a) > points(b); });
  // made by the first worker: the calling thread keeps its device, and gets no
  // context on another
  std::once_flag pool_made;
  cudaMemPool_t pool = nullptr;
  // problems that did not fit beside the others: largest first puts the large
  // ones side by side, whatever their places in the list
  std::mutex left_mu;
  std::vector<int> left;
  // One worker over the problems next_problem() gives, until it gives -1.
  auto work = [&](const std::function<int()> &next_problem, bool alone) {
    struct PoolScope {  // outlives w: its clean-up frees to the pool
      ~PoolScope() { deft::thread_pool = {}; }
    } scope;
    Worker w;
    if (deft_ctx_create(device, &w.ctx) != DEFT_OK) {
      failed(-1, DEFT_ERR_CUDA, deft_last_error());
      return;
    }
    std::call_once(pool_made, [&]() { pool = deft::make_call_pool(device); });
    deft::thread_pool = {pool, static_cast<cudaStream_t>(deft_ctx_stream(w.ctx))};
    for (int i = next_problem(); i >= 0; i = next_problem()) {
      deft_cg_status &st = status_out[i];
      memset(&st, 0, sizeof(st));
      deft::thread_out_of_memory = false;
      const int s = solve_one(w, probs[i], bp->cg, &st);
      st.status = s;
      // what it freed is there for the other workers from here on
      cudaStreamSynchronize(deft::thread_pool.stream);
      if (s && deft::thread_out_of_memory && !alone) {
        std::lock_guard<std::mutex> lock(left_mu);
        left.push_back(i);
      } else if (s) {
        failed(i, s, "problem " + std::to_string(i) + ": " + deft_last_error());
      }
    }
  };
  std::vector<std::thread> threads;
  for (int t = 0; t < workers; t++)
    threads.emplace_back([&]() {
      work([&]() {
        const int k = next.fetch_add(1);
        return k < count ? order[k] : -1;
      }, false);
    });
  for (auto &th : threads) th.join();
  // one after another, with the memory to themselves
  std::sort(left.begin(), left.end());
  for (int i : left)
    std::thread([&]() {
      bool given = false;
      work([&]() { return given ? -1 : (given = true, i); }, true);
    }).join();
  deft::end_call_pool(pool);
  if (first_error != DEFT_OK) deft::set_last_error_message(first_msg);
  return first_error;
}
