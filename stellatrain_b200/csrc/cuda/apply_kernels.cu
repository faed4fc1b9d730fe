// Receive side of the sparse exchange fused with the merge and the lazy sparse optimisers.
//
// Replaces the reference's CPU stages
//   wait for W-1 ring messages      backend/src/engine/modules/grad_exchange.cpp:18-81
//   merge (sum over sources, / W, union of indices)
//                                   backend/src/engine/modules/cpu_optimize.cpp:40-72
//   sparse SGD / sparse Adam        backend/src/optim/sgd.cpp:221-262, backend/src/optim/adam.cpp:19-87
//   H2D copy of updated parameters  backend/src/engine/modules/h2d_copy.cpp:31-56  (no longer needed)
// by two kernels per bucket (one when there is a single source, three when the optimiser state is partitioned over the
// ranks):
//   wait     one warp waits (bounded) for the arrival flags of all sources (only when flags are in use)
//   scatter  adds every source's weighted values into a dense accumulator with red.global.add.f32
//   apply    walks the same streams again; the first thread to stamp an index with the current epoch
//            owns it, reads and clears the accumulator and applies the optimiser rule once, which
//            is the "apply once at the union of indices" contract without building the union; the
//            last CTA acknowledges the slot to every source and advances the counters.
//   param    partitioned state only.  A tensor's entries go to one rank, its owner, which keeps the
//   scatter  accumulator and the optimiser state for it (1/W of the memory), applies the update and
//            stores the new values into every rank's write-back area; this kernel waits (bounded) for
//            the owners' flags and copies the values into the local replica, so replicas agree bit for
//            bit.  The reference keeps full optimiser state in every process.
#include "device_utils.cuh"
#include "launch.h"

namespace st {

namespace {
constexpr int kThreads = 256;
constexpr int kSms = 148;
constexpr int kSingleEntries = 4;      // entries that a thread of k_apply_single has under way
}

// One warp waits (bounded) for the arrival flags of all sources, one lane per source, and leaves the outcome
// in the status word.  The wide scatter grid that follows in the stream therefore never sits on the SMs
// spinning while a peer is late, which would keep the backward pass of the lower-priority compute stream out.
__global__ void k_wait_streams(ApplyArgs A) {
  const uint32_t epoch = *A.epoch;
  const uint32_t slot = epoch & 1u;
  // Nothing was selected for this epoch yet (e.g. a captured step replayed right after a flush):
  // the chain of kernels is a no-op and leaves every counter untouched.
  if (epoch >= ld_volatile_u32(A.sel_epoch)) return;
  if (ld_volatile_u32(A.status) == kOk) {
    for (int src = threadIdx.x; src < A.world; src += 32) {
      if (!wait_ge_bounded(A.flag_local + (size_t)slot * A.world + src, (uint64_t)epoch, A.timeout_ns))
        set_status(A.status, kTimeoutFlag);
    }
  }
  __syncwarp();
  next_may_begin();      // not before: the wide grid behind this must not take places while a peer is late
  if (threadIdx.x == 0 && A.stamps != nullptr) A.stamps[2] = global_timer_ns();
}

__global__ void __launch_bounds__(kThreads) k_scatter(ApplyArgs A) {
  const int src = blockIdx.y + A.src_first;
  next_may_begin();
  behind_previous();
  const uint32_t epoch = *A.epoch;
  const uint32_t slot = epoch & 1u;
  if (epoch >= ld_volatile_u32(A.sel_epoch)) return;
  if (ld_volatile_u32(A.status) != kOk) return;   // includes "a stream did not arrive in time"
  if (!A.use_flags && A.stamps != nullptr && blockIdx.x == 0 && src == 0 && threadIdx.x == 0) A.stamps[2] = global_timer_ns();
  const uint2* in = A.recv + (size_t)slot * A.slot_stride + (size_t)src * A.cap;
  const float w = A.weight[(size_t)slot * A.world + src];
  uint32_t sum = 0;
  for (uint32_t i = A.ent_lo + blockIdx.x * kThreads + threadIdx.x; i < A.ent_hi; i += gridDim.x * kThreads) {
    const uint2 e = load_entry(A, in, i);
    if (e.x == kSentinelIdx) continue;
    sum += entry_hash(e.x, e.y);
    const uint32_t s = e.x - A.state_base;   // wraps to a large value below the base
    if (s >= A.state_len) { set_status(A.status, kBadIndex); continue; }
    atomicAdd(&A.rec[s].x, __uint_as_float(e.y) * w);
  }
  if (A.cksum_local != nullptr && sum != 0u) atomicAdd(A.rsum + src, sum);
}

// Store one write-back entry into the same stream position of every rank's write-back area.
__device__ __forceinline__ void emit_writeback(const ApplyArgs& A, uint64_t pos, uint32_t idx, float val) {
  const uint2 e = make_uint2(idx, __float_as_uint(val));
  if (A.wb_mc != nullptr) {
    multimem_st_pair(A.wb_mc + pos, e);
  } else {
#pragma unroll
    for (int p = 0; p < kMaxWorld; ++p) {
      if (p < A.world) A.wb[p][pos] = e;
    }
  }
}

// Last step of a chain: acknowledge the consumed receive slot to every source, advance the counters.
__device__ __forceinline__ void finish_apply(const ApplyArgs& A, uint32_t epoch, uint32_t tick) {
  const uint32_t slot = epoch & 1u;
  if (A.use_acks && ld_volatile_u32(A.status) == kOk) {
    __threadfence_system();
    for (int p = 0; p < A.world; ++p)
      st_release_sys_u64(A.ack[p] + (size_t)slot * A.ack_slot_stride, (uint64_t)epoch);
  }
  A.opt->tick = tick + 1u;
  A.opt->first = 0u;
  *A.epoch = epoch + 1u;
  if (A.stamps != nullptr) {
    A.stamps[3] = global_timer_ns();
    A.stamps[5] = epoch;
  }
}

// What one update needs besides its entry: the bias corrections of this step (Adam) and the host's options.
struct StepConsts {
  float bc1, bc2, lr;
  uint32_t m_iter;
};

// 1 - beta^tick in double, as the reference computes it (adam.cpp:41-42).  Two double-precision powers take about
// 1.5 us: every kernel below sends its own loads off first and computes them, one in each of two warps, while those travel.
__device__ __forceinline__ float bias_correction(const OptState& o, uint32_t moment) {
  return (float)(1.0 - pow((double)(moment == 0u ? o.beta1 : o.beta2), (double)o.tick));
}

// a b + c d, c d rounded by itself.  Which of the products that is the compiler may choose in the plain expression, and kernels
// that share the rule have to agree.
__device__ __forceinline__ float weighted_sum(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }

// The optimiser rule for element `s` of the state range (`rc`: its record with the merged gradient in x, `x`: its
// parameter).  Writes the record back with the accumulator cleared and the stamp of this epoch; returns the new value.
__device__ __forceinline__ float update_element(const ApplyArgs& A, const OptState& o, const StepConsts& c, uint32_t s,
                                                uint32_t epoch, const float4& rc, float x) {
  float g = rc.x, m_new = rc.z, v_new = rc.w, xn;
  if (o.kind == 0) {
    float mu = o.momentum;
    if (o.smart_momentum && A.last != nullptr && c.m_iter != 0u)
      mu = powf(o.momentum, (float)(c.m_iter - A.last[s]));
    if (o.weight_decay != 0.f) g += o.weight_decay * x;
    if (o.momentum != 0.f) {
      const float b = o.first ? g : weighted_sum(1.f - o.dampening, g, rc.z, mu);
      g = o.nesterov ? g + mu * b : b;
      m_new = b;
    }
    xn = x - c.lr * g;
    if (o.smart_momentum && A.last != nullptr) A.last[s] = c.m_iter;
  } else {
    if (o.maximize) g = -g;
    if (o.weight_decay != 0.f) g += o.weight_decay * x;
    const float mt = weighted_sum(o.beta1, rc.z, 1.f - o.beta1, g);
    const float vt = weighted_sum(o.beta2, rc.w, __fmul_rn(1.f - o.beta2, g), g);
    const float mh = mt / c.bc1;
    float vh = vt / c.bc2;
    if (o.amsgrad && A.vmax != nullptr) {
      vh = fmaxf(A.vmax[s], vh);
      A.vmax[s] = vh;
    }
    xn = x - o.lr * mh / (sqrtf(vh) + o.eps);
    m_new = mt;
    v_new = vt;
  }
  // accumulator cleared, stamp kept (a late loser's exchange writes the same epoch again)
  A.rec[s] = make_float4(0.f, __uint_as_float(epoch), m_new, v_new);
  return xn;
}

__global__ void __launch_bounds__(kThreads) k_apply(ApplyArgs A) {
  __shared__ float s_bc[2];
  const int src = blockIdx.y;
  // nothing but the previous update writes what these need, and that was done in front of the first kernel of this chain
  const OptState o = *A.opt;
  if ((threadIdx.x & 31u) == 0u && threadIdx.x < 64u && o.kind != 0) s_bc[threadIdx.x >> 5] = bias_correction(o, threadIdx.x >> 5);
  behind_previous();
  const uint32_t epoch = *A.epoch;
  const uint32_t slot = epoch & 1u;
  if (epoch >= ld_volatile_u32(A.sel_epoch)) return;
  const bool ok = ld_volatile_u32(A.status) == kOk;

  if (ok) {
    const uint64_t src_off = (size_t)slot * A.slot_stride + (size_t)src * A.cap;
    uint2* in = A.recv + src_off;
    const uint32_t step = gridDim.x * kThreads;
    uint32_t i = A.ent_lo + blockIdx.x * kThreads + threadIdx.x;
    // The exchange that decides whether this thread owns the element comes first, and only a winner reads record and parameter.
    // A load of the record next to the exchange in flight on it makes L2 serve them one after the other: 300,000 random entries
    // of two sources took 540 us a bucket instead of 15, 900,000 of eight sources 750 us instead of 62.
    uint32_t idx = kSentinelIdx, s = 0u, old = 0u;
    bool in_range = false;
    auto claim = [&]() {
      idx = load_entry(A, in, i).x;
      s = idx - A.state_base;        // sentinel or invalid indices (already reported) fall outside
      in_range = s < A.state_len;
      // the first thread to stamp an index with this epoch owns it
      if (in_range) old = atomicExch(reinterpret_cast<uint32_t*>(&A.rec[s].y), epoch);
    };
    if (i < A.ent_hi) claim();
    if (A.cksum_local != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
      // the scatter kernel has read the whole stream of this source: does it add up to what was sent?
      const uint32_t got = atomicExch(A.rsum + src, 0u);
      const uint32_t want = __ldcg(A.cksum_local + (size_t)slot * A.world + src);
      if (got != want) set_status(A.status, kBadChecksum);
    }
    __syncthreads();
    const StepConsts c = {s_bc[0], s_bc[1], o.maximize ? -o.lr : o.lr, o.tick - 1u};
    while (i < A.ent_hi) {
      const bool won = in_range && old != epoch;
      float xn = 0.f;
      if (won) {
        const float4 rc = __ldcg(A.rec + s);      // accumulator, stamp, m, v in one 16-byte load
        xn = update_element(A, o, c, s, epoch, rc, A.param[idx]);
        A.param[idx] = xn;
      }
      // every consumed position is rewritten each epoch, so a stale value can never be read back
      if (A.owner_mode) emit_writeback(A, src_off + i, won ? idx : kSentinelIdx, xn);
      if (A.poison && !A.narrow) in[i] = make_uint2(kSentinelIdx, 0u);
      i += step;
      if (i < A.ent_hi) claim();
    }
  }

  __syncthreads();
  if (threadIdx.x == 0) {
    if (A.owner_mode) __threadfence_system();   // this CTA's stores into the peers before the count below
    else __threadfence();
    const uint32_t prev = atomicAdd(A.done_ctr, 1u);
    if (prev == gridDim.x * gridDim.y - 1) {
      *A.done_ctr = 0;
      if (!A.owner_mode) {
        finish_apply(A, epoch, o.tick);
      } else if (ld_volatile_u32(A.status) == kOk) {
        // the new values are on their way to every replica: tell them; the copy kernel finishes the chain
        __threadfence_system();
        for (int p = 0; p < A.world; ++p)
          st_release_sys_u64(A.pflag[p] + (size_t)slot * A.pflag_slot_stride, (uint64_t)epoch);
      }
    }
  }
}

// One source: its stream names every element at most once (each select emits an element once, also where the narrow wire
// format's rounding leaves something of it in the residual; random-k strides through the tensor with a step coprime to its
// size), so there is nothing to merge: no accumulator, no stamp to compete for, one kernel instead of two.
//
// Bound by a chain of trips (counters, entry, record and parameter) and, with scattered entries, by DRAM accesses to single
// records.  A thread has N entries under way: a CTA's life is the chain, so fewer and fuller CTAs leave the SMs to the streaming
// kernels of other buckets.  One entry a thread and four, us: blocks of 16 neighbours (threshold-v16) 168,000 entries of a 64 MB
// bucket 11.0 and 6.9, 670,000 28.7 and 13.5; scattered ones (top-k) 168,000 17.2 and 14.7, but 670,000 58 and 67 (every entry
// opens DRAM rows of its own, and the more of them compete the fewer stay open).  Up to one entry a thread on every SM there is
// nothing to gather.  So: four entries a thread for blocks, for scattered entries as long as that is at most two CTAs per SM.
template <int N>
__global__ void __launch_bounds__(kThreads) k_apply_single(ApplyArgs A) {
  __shared__ float s_bc[2];
  const uint32_t epoch = *A.epoch;
  const uint32_t slot = epoch & 1u;
  if (epoch >= ld_volatile_u32(A.sel_epoch)) return;
  const bool ok = ld_volatile_u32(A.status) == kOk;
  const OptState o = *A.opt;
  if (A.stamps != nullptr && !A.use_flags && blockIdx.x == 0 && threadIdx.x == 0) A.stamps[2] = global_timer_ns();
  if (ok) {
    const uint2* in = A.recv + (size_t)slot * A.slot_stride;
    const float w = A.weight[slot];
    const uint32_t step = gridDim.x * kThreads * N;
    uint32_t i = blockIdx.x * kThreads * N + threadIdx.x;
    uint2 e[N];
    float4 rc[N];
    float x[N];
    auto fetch = [&]() {
#pragma unroll
      for (int u = 0; u < N; ++u)
        e[u] = i + u * kThreads < A.ent_hi ? load_entry(A, in, i + u * kThreads) : make_uint2(kSentinelIdx, 0u);
#pragma unroll
      for (int u = 0; u < N; ++u) {
        if (e[u].x < A.n_total) {
          rc[u] = __ldcg(A.rec + e[u].x);
          x[u] = __ldcg(A.param + e[u].x);
        } else if (e[u].x != kSentinelIdx) {
          set_status(A.status, kBadIndex);
        }
      }
    };
    fetch();
    if ((threadIdx.x & 31u) == 0u && threadIdx.x < 64u && o.kind != 0) s_bc[threadIdx.x >> 5] = bias_correction(o, threadIdx.x >> 5);
    __syncthreads();
    const StepConsts c = {s_bc[0], s_bc[1], o.maximize ? -o.lr : o.lr, o.tick - 1u};
    while (true) {
#pragma unroll
      for (int u = 0; u < N; ++u) {
        if (e[u].x < A.n_total) {
          rc[u].x += __uint_as_float(e[u].y) * w;      // what the merge would have left in the accumulator
          A.param[e[u].x] = update_element(A, o, c, e[u].x, epoch, rc[u], x[u]);
        }
      }
      i += step;
      if (i >= A.ent_hi) break;
      fetch();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t prev = atomicAdd(A.done_ctr, 1u);
    if (prev == gridDim.x - 1) {
      *A.done_ctr = 0;
      finish_apply(A, epoch, o.tick);
    }
  }
}

// Partitioned state, every rank: wait (bounded) for each owner's values, copy them into the replica.
// CTAs with blockIdx.y == o serve the positions owner o consumed.
__global__ void __launch_bounds__(kThreads) k_param_scatter(ApplyArgs A) {
  __shared__ int s_ok;
  const int owner = blockIdx.y;
  const uint32_t epoch = *A.epoch;
  const uint32_t slot = epoch & 1u;
  if (epoch >= ld_volatile_u32(A.sel_epoch)) return;
  if (threadIdx.x == 0) {
    int ok = ld_volatile_u32(A.status) == kOk;
    if (ok) {
      ok = wait_ge_bounded(A.pflag_local + (size_t)slot * A.world + owner, (uint64_t)epoch, A.timeout_ns);
      if (!ok) set_status(A.status, kTimeoutFlag);
    }
    s_ok = ok;
  }
  __syncthreads();
  const uint32_t lo = A.own_lo[owner], len = A.own_lo[owner + 1] - lo;
  if (s_ok && owner != A.rank && len != 0u) {   // the owner has already written its own replica
    const uint64_t total = (uint64_t)len * (uint64_t)A.world;
    const uint2* in = A.wb_local + (size_t)slot * A.slot_stride;
    for (uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x; t < total; t += (uint64_t)gridDim.x * kThreads) {
      const uint32_t src = (uint32_t)(t / len), i = lo + (uint32_t)(t % len);
      const uint2 e = __ldcg(in + (size_t)src * A.cap + i);
      if (e.x < A.n_total) A.param[e.x] = __uint_as_float(e.y);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t prev = atomicAdd(A.done_ctr, 1u);
    if (prev == gridDim.x * gridDim.y - 1) {
      *A.done_ctr = 0;
      finish_apply(A, epoch, A.opt->tick);
    }
  }
}

// One source has nothing to merge.  The debug checks keep the two kernels: the stream's checksum has to be known
// before its first entry is applied.
bool apply_merges_nothing(const ApplyArgs& A) { return A.world == 1 && !A.owner_mode && A.cksum_local == nullptr && !A.poison; }

// phase 0: the whole chain; 1: scatter + apply only; 2: the parameter copy of partitioned state only
// (split launches let a test run several emulated ranks on one GPU without a kernel waiting for a later one).
cudaError_t launch_apply(const ApplyArgs& A, int max_ctas_per_source, int phase, cudaStream_t stream) {
  if (A.cap == 0 || A.world <= 0) return cudaSuccess;
  if (A.world > kMaxWorld) return cudaErrorInvalidValue;
  if (A.ent_hi < A.ent_lo || A.ent_hi > A.cap) return cudaErrorInvalidValue;
  // The update of an entry is a chain of dependent random accesses: its latency is hidden by many entries in flight at once.  One
  // entry per thread where streams are merged; the update of a single source may have four, see k_apply_single.
  if (phase == 0 || phase == 1) {
    int parts = (int)((A.ent_hi - A.ent_lo + kThreads - 1) / kThreads);
    if (parts < 1) parts = 1;
    if (parts > max_ctas_per_source) parts = max_ctas_per_source;
    dim3 grid(parts, A.world);
    cudaError_t e = cudaSuccess;
    if (A.use_flags) e = launch_first(k_wait_streams, dim3(1), 32, stream, A);
    if (e != cudaSuccess) return e;
    if (apply_merges_nothing(A)) {
      const uint32_t n = A.ent_hi - A.ent_lo;
      const int wide = (int)((n + kThreads * kSingleEntries - 1) / (kThreads * kSingleEntries));
      if (n > (uint32_t)(kSms * kThreads) && (A.blocks || wide <= 2 * kSms))
        k_apply_single<kSingleEntries><<<wide < max_ctas_per_source ? wide : max_ctas_per_source, kThreads, 0, stream>>>(A);
      else
        k_apply_single<1><<<parts, kThreads, 0, stream>>>(A);
      return cudaGetLastError();
    }
    if (A.deterministic) {
      ApplyArgs one = A;
      for (int src = 0; src < A.world; ++src) {   // one launch per source: a fixed order of additions
        one.src_first = (uint32_t)src;
        e = src == 0 && !A.use_flags ? launch_first(k_scatter, dim3(parts, 1), kThreads, stream, one)
                                     : launch_behind(k_scatter, dim3(parts, 1), kThreads, stream, one);
        if (e != cudaSuccess) return e;
      }
    } else {
      e = A.use_flags ? launch_behind(k_scatter, grid, kThreads, stream, A) : launch_first(k_scatter, grid, kThreads, stream, A);
    }
    if (e == cudaSuccess) e = launch_behind(k_apply, grid, kThreads, stream, A);
    if (e != cudaSuccess) return e;
  }
  if (A.owner_mode && (phase == 0 || phase == 2)) {
    uint32_t longest = 0;
    for (int o = 0; o < A.world; ++o) {
      if (A.own_lo[o + 1] < A.own_lo[o] || A.own_lo[o + 1] > A.cap) return cudaErrorInvalidValue;
      longest = A.own_lo[o + 1] - A.own_lo[o] > longest ? A.own_lo[o + 1] - A.own_lo[o] : longest;
    }
    uint64_t parts = ((uint64_t)longest * (uint64_t)A.world + kThreads - 1) / kThreads;
    if (parts < 1) parts = 1;
    if (parts > (uint64_t)max_ctas_per_source) parts = (uint64_t)max_ctas_per_source;
    dim3 grid((unsigned)parts, A.world);
    k_param_scatter<<<grid, kThreads, 0, stream>>>(A);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Single-tensor compression: the pairs of a wide stream as two arrays, in stream order.  Entries without an element ("no
// entry" of a short stream, zero padding behind the tensor) are counted; the caller drops them when there are any.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_unpack(UnpackArgs A) {
  const uint32_t epoch = A.epoch[0];      // the select has advanced it
  const uint2* in = A.recv + (size_t)((epoch - 1u) & 1u) * A.slot_stride;
  uint32_t none = 0;
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < A.k; i += gridDim.x * kThreads) {
    const uint2 e = __ldcg(in + i);
    const bool there = e.x < A.n;
    A.idx[i] = there ? (int32_t)e.x : -1;
    A.val[i] = __uint_as_float(e.y);
    none += there ? 0u : 1u;
  }
  none = __reduce_add_sync(0xffffffffu, none);
  if ((threadIdx.x & 31) == 0 && none) atomicAdd(A.left_out, none);
  if (blockIdx.x == 0 && threadIdx.x == 0) A.epoch[1] = epoch;      // both advance together, as in the engine
}

cudaError_t launch_unpack(const UnpackArgs& A, cudaStream_t stream) {
  if (A.k == 0) return cudaSuccess;
  int grid = (int)((A.k + kThreads * 2 - 1) / (kThreads * 2));
  if (grid > 148 * 8) grid = 148 * 8;
  k_unpack<<<grid, kThreads, 0, stream>>>(A);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Replica parity: max |mine - peer| over a flat range, read through a peer pointer.  The
// reference checks cross-node divergence by shipping whole tensors to the broker
// (backend/src/engine/core.cpp:843-847, 874-878); here one kernel reads the peer over NVLink.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_max_abs_diff(const float* a, const float* b, uint64_t n,
                                                          uint32_t* out_bits) {
  __shared__ uint32_t s_tmp[kThreads / 32 + 1];
  float mx = 0.f;
  for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kThreads) {
    const float d = fabsf(a[i] - b[i]);
    mx = (d == d) ? fmaxf(mx, d) : __uint_as_float(0x7f800000u);   // NaN counts as infinite drift
  }
  const uint32_t r = block_max_u32(__float_as_uint(mx), s_tmp);
  if (threadIdx.x == 0 && r) atomicMax(out_bits, r);
}

cudaError_t launch_max_abs_diff(const float* a, const float* b, uint64_t n, uint32_t* out_bits,
                                cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  int grid = (int)((n + kThreads * 8 - 1) / (kThreads * 8));
  if (grid > 148 * 8) grid = 148 * 8;
  k_max_abs_diff<<<grid, kThreads, 0, stream>>>(a, b, n, out_bits);
  return cudaGetLastError();
}

// Copy a flat range from a peer (initial parameter broadcast from rank 0; the reference relays
// every tensor through its broker: backend/src/engine/comm_manager.cpp:1022-1077).
__global__ void __launch_bounds__(kThreads) k_copy_f4(float4* dst, const float4* src, uint64_t n4) {
  for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < n4; i += (uint64_t)gridDim.x * kThreads)
    dst[i] = src[i];
}

cudaError_t launch_peer_copy(float* dst, const float* src, uint64_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if ((n & 3u) || ((uintptr_t)dst & 15u) || ((uintptr_t)src & 15u)) return cudaErrorInvalidValue;
  const uint64_t n4 = n / 4;
  int grid = (int)((n4 + kThreads * 4 - 1) / (kThreads * 4));
  if (grid > 148 * 8) grid = 148 * 8;
  k_copy_f4<<<grid, kThreads, 0, stream>>>(reinterpret_cast<float4*>(dst), reinterpret_cast<const float4*>(src), n4);
  return cudaGetLastError();
}

}  // namespace st
