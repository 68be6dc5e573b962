// Slices of a pattern count's long launches: the per-edge kernels (patterns.cu) and
// the pairs and wheels of graphs with hubs (motifs.cu).
#pragma once
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "device_common.cuh"
#include "dgraph.cuh"

namespace mc {

// Long pattern counts run in slices of their task range, each a launch of
// bounded length, so that no kernel runs for minutes and a caller's time
// budget can end the count between two slices.  Slices are sized from the
// previous slice's measured time (first slice: one task per resident warp or
// group, then x(target / measured), clamped to [1/4, 4]).

// Graphs whose largest degree exceeds this run their pattern launches in slices
// (hub edges can take seconds each).
constexpr int64_t kSliceDegree = 4096;

struct Slicer {
  bool on = false;
  double budget_ms = -1.0;  // < 0: no budget
  double target_ms = 250.0;
  bool trace = false;
  double used_ms = 0.0;     // device time of the sliced launches so far
  int64_t tasks_total = 0, tasks_done = 0, slices = 0;
  // With a budget the kernels also stop by themselves at a device deadline
  // (a single hub edge can outlast any slice); stop_flag is the device word
  // they raise, and h_stop its host copy.
  unsigned long long *stop_flag = nullptr;
  unsigned long long *h_stop = nullptr;

  // MERCURY_PATTERN_SLICE=1/0 forces slicing on/off (the tests compare both);
  // MERCURY_PATTERN_SLICE_MS sets the target slice length; MERCURY_TRACE_SLICES
  // prints each slice to stderr.
  Slicer(const mc_dgraph *g, double budget) : budget_ms(budget) {
    on = budget > 0 || g->max_degree > kSliceDegree;
    if (const char *env = std::getenv("MERCURY_PATTERN_SLICE")) on = std::atoi(env) != 0 || budget > 0;
    if (const char *env = std::getenv("MERCURY_PATTERN_SLICE_MS"))
      target_ms = std::max(0.01, std::atof(env));
    trace = std::getenv("MERCURY_TRACE_SLICES") != nullptr;
  }
};

// launch(begin, end) runs tasks [begin, end) of a launch whose queue counter
// is `queue` (null: none); total = the launch's task count, first = first slice size.
template <class Launch>
int run_slices(mc_dgraph *g, Slicer &sl, const char *what, int64_t total, int64_t first,
               unsigned long long *queue, Launch launch) {
  if (!sl.on) return launch(0, -1);
  if (total <= 0) return MC_OK;
  cudaStream_t s = g->stream;
  sl.tasks_total += total;
  int64_t b = 0, size = std::max<int64_t>(first, 1);
  while (b < total) {
    const int64_t e = std::min(total, b + size);
    if (queue) MC_CUDA_TRY(cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s));
    MC_CUDA_TRY(cudaEventRecord(g->ev[4], s));
    const int rc = launch(b, e);
    if (rc != MC_OK) return rc;
    if (sl.stop_flag)
      MC_CUDA_TRY(cudaMemcpyAsync(sl.h_stop, sl.stop_flag, sizeof(unsigned long long),
                                  cudaMemcpyDeviceToHost, s));
    MC_CUDA_TRY(cudaEventRecord(g->ev[5], s));
    MC_CUDA_TRY(cudaEventSynchronize(g->ev[5]));
    float ms = 0.f;
    MC_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev[4], g->ev[5]));
    sl.used_ms += ms;
    sl.tasks_done += e - b;
    sl.slices += 1;
    if (sl.trace)
      std::fprintf(stderr, "mercury: %s slice [%lld, %lld) of %lld: %.3f ms (total %.1f ms)\n",
                   what, (long long)b, (long long)e, (long long)total, ms, sl.used_ms);
    b = e;
    if (sl.h_stop && *sl.h_stop) return MC_ERR_TIMEOUT;  // stopped at the deadline
    if (sl.budget_ms > 0 && sl.used_ms > sl.budget_ms && b < total) return MC_ERR_TIMEOUT;
    // Never below one task per resident warp or group: a smaller slice
    // leaves the GPU idle.
    const double f = ms > 0.01f ? std::min(4.0, std::max(0.25, sl.target_ms / ms)) : 4.0;
    size = std::max<int64_t>(std::max<int64_t>(first, 1), (int64_t)((double)size * f));
  }
  return MC_OK;
}

}  // namespace mc
