// One bucket's pre-filled kernel arguments and the launches that use them.  Filled once at set-up by the Python
// side (bindings.cpp); `select` and `apply` are then a handful of kernel launches without any per-call
// marshalling, from Python or from the native step engine (native_engine.cpp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "launchers.h"

namespace st {

struct BucketHandle {
  SelectArgs sel;
  ApplyArgs app;
  GroupArgs grp;
  bool has_group = false;
  uint32_t randomk_seed = 0x5DEECE66u;
  int max_ctas_per_source = 148 * 16;
  // One-pass select: allowed by configuration, and possible once every tensor of the bucket has its threshold
  // (one select through the four-kernel chain, or a restored checkpoint).
  bool fused_enabled = true;
  bool thresholds_ready = false;
  bool last_select_fused = false;

  bool can_fuse() const { return one_pass_possible(sel); }
  bool one_pass_next() const { return fused_enabled && thresholds_ready && can_fuse(); }

  // `before_emit` (or null): what has to be done before entries are stored; the one-pass chain streams beside it.
  cudaError_t select(cudaStream_t stream, cudaEvent_t before_emit = nullptr) {
    const bool fused = one_pass_next();
    if (!fused && before_emit != nullptr) {
      const cudaError_t w = cudaStreamWaitEvent(stream, before_emit, 0);
      if (w != cudaSuccess) return w;
    }
    const cudaError_t e = fused ? launch_select_one_pass(sel, stream, before_emit) : launch_select(sel, randomk_seed, stream);
    thresholds_ready = true;       // the four-kernel chain leaves every tensor with a threshold
    last_select_fused = fused;
    return e;
  }

  // kernels of the last select (telemetry's launch count)
  int select_kernels() const {
    if (sel.compressor == kRandomk) return 2;
    if (!last_select_fused) return 4;
    return sel.compressor == kTopk ? 3 : 2;
  }

  cudaError_t apply(cudaStream_t stream, int phase) { return launch_apply(app, max_ctas_per_source, phase, stream); }

  int apply_kernels() const {
    if (apply_merges_nothing(app)) return 1 + (app.use_flags ? 1 : 0);
    return (app.owner_mode ? 3 : 2) + (app.deterministic ? app.world - 1 : 0) + (app.use_flags ? 1 : 0);
  }

  cudaError_t group_reduce(cudaStream_t stream) {
    if (!has_group) return cudaSuccess;
    grp.segs = sel.segs;
    grp.chunks = sel.chunks;
    grp.n_chunks = sel.n_chunks;
    grp.epoch = sel.epoch;
    grp.status = sel.status;
    grp.timeout_ns = sel.timeout_ns;
    return launch_group_reduce(grp, stream);
  }
};

}  // namespace st
