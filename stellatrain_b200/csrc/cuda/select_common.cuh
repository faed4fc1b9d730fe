// What the select chains share: guarded float4 accesses, block keys, the histogram window, and the completion of a stream.
#pragma once
#include "device_utils.cuh"

namespace st {

constexpr float kWindowDefault = 0.05f;        // threshold-v16's near misses: keys in [tau * (1 - window), tau)

__device__ __forceinline__ uint32_t key_bits(float a) { return __float_as_uint(a) & 0x7fffffffu; }

// Gradients are read once: streaming loads and stores (evict-first) keep them from pushing the
// residual, which pass 2 reads again, out of L2.
__device__ __forceinline__ float4 load4_guarded(const float* p, uint32_t i, uint32_t valid) {
  if (i + 4 <= valid) return __ldcs(reinterpret_cast<const float4*>(p + i));
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i + 0 < valid) v.x = p[i + 0];
  if (i + 1 < valid) v.y = p[i + 1];
  if (i + 2 < valid) v.z = p[i + 2];
  return v;
}

__device__ __forceinline__ void store4_guarded(float* p, uint32_t i, uint32_t valid, float4 v) {
  if (i + 4 <= valid) {
    __stcs(reinterpret_cast<float4*>(p + i), v);
    return;
  }
  if (i + 0 < valid) p[i + 0] = v.x;
  if (i + 1 < valid) p[i + 1] = v.y;
  if (i + 2 < valid) p[i + 2] = v.z;
}

// L1 norm of the 16-element block held by four consecutive lanes (one float4 each).  The
// reduction tree is fixed, so the value is identical in all four lanes and reproducible.
__device__ __forceinline__ float quad_l1(const float4& a) {
  float s = (fabsf(a.x) + fabsf(a.y)) + (fabsf(a.z) + fabsf(a.w));
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s;
}

// ------------------------------------------------------------------------------------------------
// histogram window
// ------------------------------------------------------------------------------------------------
struct HistWindow {
  uint32_t base, shift;
};

__device__ __forceinline__ HistWindow window_of(const SegState& ss) {
  HistWindow w;
  w.base = ss.hist_shift ? ss.hist_base : 0u;
  w.shift = ss.hist_shift ? ss.hist_shift : (uint32_t)kHistShift;
  return w;
}

// Monotone in key, so "bin > b" implies "key above every key of bin b".
__device__ __forceinline__ uint32_t bin_of(uint32_t key, const HistWindow& w) {
  if (key < w.base) return 0u;
  const uint32_t b = (key - w.base) >> w.shift;
  return b < (uint32_t)(kHistBins - 1) ? b : (uint32_t)(kHistBins - 1);
}

// Window for the next select: 2048 bins of 2^13 key units (2^-10 relative) centred on `key`,
// i.e. one octave to either side; keys outside fall into the two end bins.
__device__ __forceinline__ void centre_window(SegState& ss, uint32_t key) {
  const uint32_t half = (uint32_t)(kHistBins / 2) << kFineShift;
  ss.hist_shift = kFineShift;
  ss.hist_base = key > half ? key - half : 0u;
}

// Debug checks: hand every destination the sum over the entries this select stored into it, and clear
// the accumulators for the next select.  Called by the one thread that publishes the arrival flags, before
// them (their release orders these stores too).
__device__ __forceinline__ void publish_checksums(const SelectArgs& A, uint32_t epoch) {
  if (A.stamps != nullptr) {
    A.stamps[1] = global_timer_ns();
    A.stamps[4] = epoch;
  }
  if (A.cksum_acc == nullptr) return;
  for (int p = 0; p < A.world; ++p) {
    const uint32_t sum = atomicAdd(A.cksum_acc + (A.owner_mode ? p : 0), 0u);
    if (A.cksum[p] != nullptr) A.cksum[p][(size_t)(epoch & 1u) * A.cksum_slot_stride] = sum;
  }
  for (int p = 0; p < kMaxWorld; ++p) A.cksum_acc[p] = 0u;
  __threadfence_system();
}

// The receive slot about to be overwritten was last used two epochs ago; every destination must have consumed
// it.  One thread calls this right before its CTA stores into the destinations.  Inlined: as a function of its own, which reads the
// kernel's arguments through memory between loads that acquire, it made a select with eight destinations 3 us longer.
__device__ __forceinline__ bool acks_arrived(const SelectArgs& A, uint32_t epoch) {
  if (!A.use_acks || epoch <= 2u) return true;
  const uint64_t want = (uint64_t)epoch - 2u;
  for (int p = 0; p < A.world; ++p) {
    if (!wait_ge_bounded(A.ack_local + (size_t)(epoch & 1u) * A.world + p, want, A.timeout_ns)) {
      set_status(A.status, kTimeoutAck);
      return false;
    }
  }
  return true;
}

// Completion of a select chain, called by thread 0 of every CTA of its last kernel after a CTA barrier: the last
// CTA publishes the arrival flags and advances the epoch.  The CTA barrier orders the CTA's stores before this
// thread's system-scope fence, the counter orders the CTAs.  `refills`: when the word is not zero the stream is not
// complete yet and the chain's next kernel finishes it, unless `is_refill` says that this is that kernel.
__device__ __forceinline__ void finish_select(const SelectArgs& A, uint32_t epoch, uint32_t* refills = nullptr,
                                              bool is_refill = false) {
  if (A.publish) __threadfence_system();   // stores into peers' memory; without peers the counter's own order is enough
  const uint32_t prev = atom_add_acq_rel_gpu(A.done_ctr, 1u);
  if (prev == gridDim.x - 1) {
    *A.done_ctr = 0;
    if (A.publish) __threadfence_system();     // without peers the end of the kernel is enough, and sooner
    if (refills != nullptr) {
      if (is_refill) *refills = 0;
      else if (ld_volatile_u32(refills) != 0u) return;
    }
    publish_checksums(A, epoch);
    if (A.publish && ld_volatile_u32(A.status) == kOk) {
      for (int p = 0; p < A.world; ++p)
        st_release_sys_u64(A.flag[p] + (size_t)(epoch & 1u) * A.flag_slot_stride, (uint64_t)epoch);
    }
    *A.epoch = epoch + 1;
  }
}

}  // namespace st
