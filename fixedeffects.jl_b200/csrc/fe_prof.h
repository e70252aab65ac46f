// fe_prof.h -- per-launch timing of a plan's kernels (FE_OPT_PROFILE).
#pragma once

#include "fe_plan.h"

namespace fe {

// ---------------------------------------------------------------------------
// profiling: CUDA events around launches on the plan's stream
// ---------------------------------------------------------------------------
struct ProfScope {
  fe_plan* pl;
  const char* name;
  double bytes;
  cudaEvent_t a = nullptr, b = nullptr;
  ProfScope(fe_plan* p, const char* n, double by) : pl(p), name(n), bytes(by) {
    if (!pl->prof.on) return;
    a = take();
    b = take();
    cudaEventRecord(a, pl->stream);
  }
  cudaEvent_t take() {
    if (!pl->prof.pool.empty()) {
      cudaEvent_t e = pl->prof.pool.back();
      pl->prof.pool.pop_back();
      return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
  }
  ~ProfScope() {
    if (!pl->prof.on) return;
    cudaEventRecord(b, pl->stream);
    pl->prof.pending.push_back({name, {a, b}});
    pl->prof.bytes_per_launch[name] = bytes;
  }
};

}  // namespace fe
