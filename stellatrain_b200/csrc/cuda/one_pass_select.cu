// One-pass select: the steady state of top-k, threshold-v and threshold-v16.
//
// Every tensor remembers the threshold of its previous select, so one pass over gradient and residual can already tell
// the few items that matter from the rest:
//   scan    a = g + r, r <- a; every warp walks one run of 1024 consecutive elements and lists the run's items at or over
//           a cut, without a word to any other warp.  The cut is the persistent threshold (threshold-v and threshold-v16,
//           backend/src/compress/thresholdv.cpp:44-52, backend/src/compress/thresholdv16.cpp:81-97; the latter also lists
//           near-miss blocks just under it) or a little less than the previous k-th largest value (top-k, which also
//           counts its candidates in a histogram around that value).
//   emit    one CTA per piece (8 to 128 runs) of a tensor turns the lists into stream entries, stores them into the
//           destinations' receive areas and clears them in r.  The CTA that finishes a tensor last settles what is left:
//           the exact cut inside the threshold's bin (top-k), the best of the near misses when the blocks over the
//           threshold fall short of the budget (the reference's heap, backend/src/compress/thresholdv16.cpp:261-293),
//           the step of the threshold (AIMD).  Threshold-v pads a short stream instead
//           (backend/src/compress/thresholdv.cpp:82).
//   refill  top-k only: tensors whose candidates fell short of k (the distribution dropped below the cut) are selected
//           from r itself.  Their histogram was taken by `emit`; with no such tensor this kernel returns at once.
// 12 bytes per element cross HBM (read g, read r, write r) against 16 to 20 of the four-kernel chain, which remains for a
// tensor's first select.  The entries are those of the four-kernel chain, with one exception: a threshold-v16 block that holds
// nothing is never sent, and a tensor with fewer blocks that hold something than its budget says "no entry" for the rest.  The
// order differs: top-k's entries come as its pieces get to them, and a threshold-v16 stream that is short of blocks over the
// threshold has those first, in index order, and the fill behind them.
//
// What bounds it, 64 MB bucket (16.8 M elements, 201 MB of traffic, 31 us at the 6.5 TB/s of a plain copy), one B200:
//   scan    memory: 35.5 us for threshold-v16 (29 where L2 holds part of a single bucket), 36 us for top-k at 0.1 %, 39 us at 1 %
//           (list and histogram).  Runs of one warp need no barrier and no shared state, so a late load holds up nothing else;
//           with one CTA per 8192 elements that scanned, chained counts over CTAs and emitted by itself the same traffic took
//           54 us.
//   emit    latency, a chain of about ten trips to L2, and its own instructions (see send_staged): 9.6 us for threshold-v16, 16 us
//           for top-k at 1 %; the slowest sections of the latter are the sum of the histograms (3 us) and the last CTA's
//           search (3 us).
//   refill  1.4 to 2.5 us when there is nothing to do; one tensor of 16.8 M normal values (3 M), residual empty, that fell to a
//           third takes 104 us (22) here and 65 us (15) in `emit`, where a CTA counts a piece of 131,072 elements (16,384); where they
//           fell to a hundredth, so that the cut lies in a wide bin, 729 us (112), most of them for the ranking by the last CTA.
#include "launch.h"
#include "launchers.h"
#include "select_common.cuh"

namespace st {

namespace {

enum ScanMode : int { kScanTop = 0, kScanElem = 1, kScanBlock = 2 };

constexpr int kScanThreads = 256;
constexpr int kScanWarps = kScanThreads / 32;
constexpr uint32_t kHalf = kRunElems / 2;      // a run is read in two halves: four float4 of r and of g per lane in flight
constexpr uint32_t kRunBlocks = kRunElems / 16;
constexpr uint32_t kMaxPieceElems = kMaxPieceRuns * kRunElems;

constexpr int kEmitThreads = 256;
constexpr uint32_t kStageItems = 2048;         // entries staged at a time
constexpr uint32_t kPickMax = 2048;            // candidates that a CTA holds in shared memory to pick the best from

// Top-k of a tensor this small is picked from shared memory by its one CTA of `emit`: its k-th largest value moves too much from
// step to step to be worth predicting, and no list, histogram or cut is needed.
constexpr uint32_t kTopDirect = 4096;
constexpr float kTopWindowDefault = 0.1f;
constexpr float kTopWindowMin = 1e-3f;
constexpr float kTopWindowMax = 0.45f;         // the histogram reaches down to half the previous threshold

__device__ __forceinline__ float window_or(uint32_t bits, float fallback) {
  const float w = __uint_as_float(bits);
  return (w > 0.f && w <= 1.f) ? w : fallback;
}

// Lowest key top-k lists: a little under the previous k-th largest value, and never zero.
__device__ __forceinline__ uint32_t top_cut(const SegState& ss, uint32_t n_pad) {
  if (n_pad <= kTopDirect) return 0xFFFFFFFFu;     // lists nothing
  const float t = __uint_as_float(ss.reserved[1]);
  const float w = fminf(window_or(ss.reserved[0], kTopWindowDefault), kTopWindowMax);
  const uint32_t cut = t < __uint_as_float(0x7f800000u) ? __float_as_uint(t * (1.f - w)) : ss.reserved[1];
  return cut ? cut : 1u;
}

// Histogram of top-k's candidates around the previous threshold c (float bits), widths of bins that grow with the distance, on
// either side 256 of 2^-16 (relative) as far as 0.4 %, 128 of 2^-12 as far as 3 %, 512 of 2^-9 as far as an octave, 128 of an
// eighth of an octave each beyond (gradients that jump up), the rest in the end bins.  Error feedback piles items up at the
// threshold: with bins of 2^-10 throughout a few of them took most of the counts (L2 adds to one address one after the other:
// 239 us for a scan of 38.6 M elements, of which the traffic needs 75) and the threshold's bin held thousands of undecided
// items.  A batch whose norm differs puts the threshold far from c: with bins of 2^-7 there, 25,000 of a 64 MB bucket's items
// were undecided at 10 % kept.
// c = 0 stands for "no usable threshold": 2048 even bins over all keys.
// A tensor of several pieces spreads its counts over up to eight such histograms (one per piece modulo their number): 500,000
// adds into the 64 cache lines of a single one still took 60 us longer than the traffic.
constexpr int kNearShift = 7, kMidShift = 11, kFarShift = 14, kBeyondShift = 20;
constexpr uint32_t kNearBins = 256u, kMidBins = 128u, kFarBins = 512u;
constexpr uint32_t kMidFrom = kNearBins, kFarFrom = kMidFrom + kMidBins, kBeyondFrom = kFarFrom + kFarBins;      // of 1024 bins a side
constexpr uint32_t kNear = kNearBins << kNearShift, kMid = kNear + (kMidBins << kMidShift);     // distances where the widths change
constexpr uint32_t kFar = kMid + (kFarBins << kFarShift);

__device__ __forceinline__ uint32_t top_centre(const SegState& ss) {
  return ss.reserved[1] >= (1u << 24) ? ss.reserved[1] : 0u;      // all bins under it fit
}

// Histogram of what lies under the cut, for a tensor whose candidates fell short: bins of 2^15 key units for the four octaves
// under the cut (2^-8 relative; coarser ones would put most elements on a few shared-memory addresses), four bins per octave
// below, bin 0 for zeros alone.  Monotone in key; key < cut.
__device__ __forceinline__ uint32_t rest_bin(uint32_t key, uint32_t cut) {
  const uint32_t d = cut - 1u - key;
  if (d < 1u << 25) return key ? 2047u - (d >> 15) : 0u;
  return key ? max(1u, min(1023u, key >> 21)) : 0u;
}

__device__ __forceinline__ void rest_bin_range(uint32_t bin, uint32_t cut, uint32_t& lo, uint32_t& hi) {
  if (bin == 0u) { lo = 0u; hi = 1u; return; }
  if (bin >= 1024u) {
    const uint32_t from = (2047u - bin) << 15;         // distances [from, from + 2^15)
    hi = cut - from;
    lo = hi > 1u << 15 ? hi - (1u << 15) : 1u;
  } else {
    lo = bin == 1u ? 1u : bin << 21;
    hi = (bin + 1u) << 21;
  }
  if (cut > 1u << 25) {                                // the four octaves end where the coarse bins begin
    const uint32_t edge = cut - (1u << 25);
    if (bin >= 1024u) lo = max(lo, edge); else hi = min(hi, edge);
  }
}

// By the tensor's size and not its number of pieces, which is never smaller: every CTA of `emit` reads them all.
__device__ __forceinline__ uint32_t hist_copies(uint32_t n_pad) {
  const uint32_t full = (n_pad + kMaxPieceElems - 1u) / kMaxPieceElems;
  return full >= 8u ? 8u : full >= 4u ? 4u : full >= 2u ? 2u : 1u;
}

// Monotone in key.
__device__ __forceinline__ uint32_t top_bin(uint32_t key, uint32_t c) {
  if (c == 0u) return key >> kHistShift;
  const bool above = key >= c;
  const uint32_t d = above ? key - c : c - key - 1u;
  const uint32_t b = d < kNear  ? d >> kNearShift
                     : d < kMid ? kMidFrom + ((d - kNear) >> kMidShift)
                     : d < kFar ? kFarFrom + ((d - kMid) >> kFarShift)
                                : min(1023u, kBeyondFrom + ((d - kFar) >> kBeyondShift));
  return above ? 1024u + b : 1023u - b;
}

// Key range [lo, hi) of a bin; keys are below 2^31, so 2^31 stands for "none above".
__device__ __forceinline__ void top_bin_range(uint32_t bin, uint32_t c, uint32_t& lo, uint32_t& hi) {
  if (c == 0u) {
    lo = bin << kHistShift;
    hi = (bin + 1u) << kHistShift;
    return;
  }
  const bool above = bin >= 1024u;
  const uint32_t b = above ? bin - 1024u : 1023u - bin;
  const int shift = b < kMidFrom ? kNearShift : b < kFarFrom ? kMidShift : b < kBeyondFrom ? kFarShift : kBeyondShift;
  const uint32_t from = b < kMidFrom      ? b << kNearShift
                        : b < kFarFrom    ? kNear + ((b - kMidFrom) << kMidShift)
                        : b < kBeyondFrom ? kMid + ((b - kFarFrom) << kFarShift)
                                          : kFar + ((b - kBeyondFrom) << kBeyondShift);
  const uint32_t to = from + (1u << shift);          // distances [from, to)
  if (above) {
    lo = min(c + from, 0x80000000u);
    hi = b == 1023u ? 0x80000000u : min(c + to, 0x80000000u);
  } else {
    lo = b == 1023u || to >= c ? 0u : c - to;
    hi = from >= c ? 0u : c - from;
  }
}
static_assert(kHistBins == 2048 && kHistShift == 20 && kFar < 1u << 24, "bins of top_bin");

}  // namespace

// ------------------------------------------------------------------------------------------------
// the residual
// ------------------------------------------------------------------------------------------------
namespace {

__device__ __forceinline__ float number_or_zero(float x) { return x == x ? x : 0.f; }

// Elements of the residual.  A tensor compressed by itself has none: A.resid is the caller's tensor then, which is read where it
// lies, up to its last element, with NaN as zero (scan's policy), and never written.  Half of the traffic of scan: with a copy of
// the tensor as its residual, 38.6 M elements took 63 us.
// FRESH: A.fresh is not 0.
//
// Four elements are read in two parts, so that a thread's loads travel together: `load4` for all of them, without a branch, then
// `resid4` for each, which adds what the tensor's end cut off.  With a branch around every load they went one after the other: a
// `compress` of 16.8 M elements (top-k, 1 %) whose values had fallen to a thirtieth took 778 us and now 551, fallen to a third 338
// and 256, grown thirtyfold 1497 and 1206; `emit` of threshold-v16, values fallen to a third, 185 and 106.
template <bool FRESH>
__device__ __forceinline__ float4 load4(const SelectArgs& A, uint32_t i) {
  return !FRESH || i + 4u <= A.fresh ? __ldcg(reinterpret_cast<const float4*>(A.resid + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
}

template <bool FRESH>
__device__ __forceinline__ float4 resid4(const SelectArgs& A, uint32_t i, float4 a) {
  if (!FRESH) return a;
  if (i < A.fresh && i + 4u > A.fresh) a = load4_guarded(A.resid, i, A.fresh);
  return make_float4(number_or_zero(a.x), number_or_zero(a.y), number_or_zero(a.z), number_or_zero(a.w));
}

template <bool FRESH>
__device__ __forceinline__ float resid1(const SelectArgs& A, uint32_t i) {
  if (!FRESH) return __ldcg(A.resid + i);
  const float a = __ldcg(A.resid + min(i, A.fresh - 1u));
  return i < A.fresh ? number_or_zero(a) : 0.f;
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// scan
// ------------------------------------------------------------------------------------------------
// FRESH: A.fresh is not 0 (a tensor compressed by itself).  Known when the kernel is compiled, as the tests for it cost 2 % of a
// captured step otherwise.
template <int MODE, bool FRESH>
__global__ void __launch_bounds__(kScanThreads, 4) k_scan(SelectArgs A) {
  // The run's place is all the first loads of r need: they are on their way while the tensor's descriptor, threshold and
  // gradient pointer (a second level of dependent loads) are fetched.
  const Chunk ch = A.chunks[blockIdx.x];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  // Half a run that has listed elements, and their places in it: all lanes take part in storing (and, top-k, counting) them.  The
  // lists of top-k are instructions before they are traffic: with the listed values stored from registers, one predicated store
  // for each of a lane's sixteen, this kernel issued 157 warp instructions per 128 elements at 1 % and took 37 us where
  // threshold-v16 takes 29 (64 MB bucket).
  __shared__ float4 s_half[MODE == kScanBlock ? 1 : kScanWarps][MODE == kScanBlock ? 1 : kHalf / 4];
  __shared__ uint16_t s_place[MODE == kScanBlock ? 1 : kScanWarps][MODE == kScanBlock ? 1 : kHalf];
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.stamps != nullptr) A.stamps[0] = global_timer_ns();
  next_may_begin();

  const uint32_t piece_shift = A.piece_shift + kRunShift;      // of elements
  for (uint32_t rel = warp * kRunElems; rel < ch.len; rel += kScanWarps * kRunElems) {
    const uint32_t start = ch.start + rel;
    const uint32_t len = min(kRunElems, ch.len - rel);     // multiple of 16
    float* r = A.resid + start;
    float4 rv[4], gv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t i = j * 128u + lane * 4u;
      rv[j] = i < len && !FRESH ? *reinterpret_cast<const float4*>(r + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const SegDesc sd = A.segs[ch.seg];
    const bool tab = A.grad_tab != nullptr;
    const uint32_t seg_rel = start - sd.off;
    float* g = tab ? A.grad_tab[ch.seg] + seg_rel : A.grad + start;
    const SegState ss = A.state[ch.seg];
    if (sd.reserved & kSegSkip) {
      // a tensor another rank of the group is responsible for: only clear the consumed gradient
      if (A.zero_grad && !tab)
        for (uint32_t i = lane * 4u; i < len; i += 128u) *reinterpret_cast<float4*>(g + i) = make_float4(0.f, 0.f, 0.f, 0.f);
      continue;
    }
    const uint32_t n_valid = sd.n > seg_rel ? min(len, sd.n - seg_rel) : 0u;
    const uint32_t g_valid = tab || FRESH ? n_valid : len;   // gradients handed over per tensor are not padded
    const bool add = !A.skip_ef;
    // a tensor without a threshold yet lists nothing: `emit` then takes the exact top items from the residual
    const uint32_t tau_bits = ss.inited ? __float_as_uint(ss.tau) : 0xFFFFFFFFu;
    uint32_t cut = tau_bits, near_lo = 0xFFFFFFFFu;
    if (MODE == kScanTop) cut = top_cut(ss, sd.n_pad);
    if (MODE == kScanBlock && ss.inited)
      near_lo = __float_as_uint(fmaxf(ss.tau * (1.f - window_or(ss.reserved[0], kWindowDefault)), 0.f));

    // Magnitudes compare as their bits do; nothing reaches a cut over the bits of infinity, also with the sign bit set (a restored
    // threshold may be anything): all of those become one that is no number.
    const float cut_value = __uint_as_float(min(cut, 0x7fc00000u));
    uint32_t n_list = 0;                // entries listed so far
    float mx = 0.f;                     // largest magnitude of this lane
    uint32_t own[2] = {0u, 0u};         // block mode: keys of two of the run's blocks, numbers h * 32 + (lane & 3) * 8 + lane / 4
    uint2* list = A.cand + (MODE == kScanBlock ? start >> 4 : start);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t h0 = h * kHalf + lane * 4u;
      if (h == 1) {
        if (len <= kHalf) break;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t i = h0 + j * 128u;
          rv[j] = i < len && !FRESH ? *reinterpret_cast<const float4*>(r + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (add) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t i = h0 + j * 128u;
          gv[j] = i < len ? load4_guarded(g, i, g_valid) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      uint32_t mask = 0;                // bit 4 j + e: element e of float4 j is listed
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t i = h0 + j * 128u;
        float4 a = rv[j];
        if (add) {
          a.x += gv[j].x; a.y += gv[j].y; a.z += gv[j].z; a.w += gv[j].w;
          // NaN policy: a NaN is dropped (neither sent nor kept), so it cannot poison the residual.  The sum of the
          // magnitudes is NaN exactly when one of them is.
          const float s = (fabsf(a.x) + fabsf(a.y)) + (fabsf(a.z) + fabsf(a.w));
          if (!(s == s)) {
            if (!(a.x == a.x)) a.x = 0.f;
            if (!(a.y == a.y)) a.y = 0.f;
            if (!(a.z == a.z)) a.z = 0.f;
            if (!(a.w == a.w)) a.w = 0.f;
          }
          if (i < len && !FRESH) {
            *reinterpret_cast<float4*>(r + i) = a;
            if (A.zero_grad) store4_guarded(g, i, g_valid, make_float4(0.f, 0.f, 0.f, 0.f));
          }
          rv[j] = a;
        }
        if (MODE == kScanBlock) {
          const uint32_t key = __float_as_uint(quad_l1(a));   // the same value in the four lanes of a block
          if ((lane & 3u) == (uint32_t)j) own[h] = key;
        } else {
          if (fabsf(a.x) >= cut_value) mask |= 1u << (4 * j);
          if (fabsf(a.y) >= cut_value) mask |= 2u << (4 * j);
          if (fabsf(a.z) >= cut_value) mask |= 4u << (4 * j);
          if (fabsf(a.w) >= cut_value) mask |= 8u << (4 * j);
          if (MODE == kScanElem) mx = fmaxf(mx, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))));
        }
      }
      if (MODE == kScanElem && n_valid < (h + 1) * kHalf) {
        // the padding behind the tensor never counts, whatever the threshold
#pragma unroll
        for (int b = 0; b < 16; ++b)
          if (h0 + (b >> 2) * 128u + (b & 3) >= n_valid) mask &= ~(1u << b);
      }
      if (MODE != kScanBlock && __any_sync(0xffffffffu, mask != 0u)) {
        // places in index order: one scan carries the counts of the four float4 in its four bytes (at most 128 each)
        uint32_t n4 = mask - ((mask >> 1) & 0x5555u);
        n4 = (n4 & 0x3333u) + ((n4 >> 2) & 0x3333u);
        n4 = (n4 & 0xFu) | (n4 & 0xF0u) << 4 | (n4 & 0xF00u) << 8 | (n4 & 0xF000u) << 12;
        const uint32_t incl = warp_incl_scan(n4), ex = incl - n4;
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t c0 = all & 0xFFu, c1 = c0 + ((all >> 8) & 0xFFu), c2 = c1 + ((all >> 16) & 0xFFu), n_half = c2 + (all >> 24);
        // the lane's next place for an element of each float4, 16 bits each
        uint32_t at01 = (ex & 0xFFu) | (c0 + ((ex >> 8) & 0xFFu)) << 16;
        uint32_t at23 = (c1 + ((ex >> 16) & 0xFFu)) | (c2 + (ex >> 24)) << 16;
        float4* const half = s_half[warp];
        uint16_t* const place = s_place[warp];
#pragma unroll
        for (int j = 0; j < 4; ++j) half[j * 32 + lane] = rv[j];
        for (uint32_t left = mask; left != 0u; left &= left - 1u) {
          const uint32_t bit = __ffs(left) - 1u, shift = (bit & 4u) << 2;
          const uint32_t at = bit & 8u ? at23 : at01;
          place[(at >> shift) & 0xFFFFu] = (uint16_t)((bit >> 2) * 128u + lane * 4u + (bit & 3u));
          if (bit & 8u) at23 += 1u << shift; else at01 += 1u << shift;
        }
        __syncwarp();
        const float* const value = reinterpret_cast<const float*>(half);
        uint2* const dst = list + n_list;
        // Histogram of top-k's candidates.  The top bin, which holds many of them, is not counted: `emit` knows their number.
        uint32_t* gh = nullptr;
        uint32_t centre = 0;
        if (MODE == kScanTop) {
          centre = top_centre(ss);
          const uint32_t piece = seg_rel >> piece_shift;      // of the tensor
          const uint32_t first_piece = ((ch.run0 + rel / kRunElems) >> A.piece_shift) - piece;
          gh = A.hist_top + (size_t)(first_piece + (piece & (hist_copies(sd.n_pad) - 1u))) * kHistBins;
        }
        for (uint32_t q = lane; q < n_half; q += 32u) {
          const uint32_t i = place[q], bits = __float_as_uint(value[i]);
          dst[q] = make_uint2(start + h * kHalf + i, bits);
          if (MODE == kScanTop) {
            const uint32_t b = top_bin(bits & 0x7fffffffu, centre);
            if (b != (uint32_t)(kHistBins - 1)) atomicAdd(gh + b, 1u);
          }
        }
        __syncwarp();
        n_list += n_half;
      }
    }
    uint32_t n_near = 0;
    if (MODE == kScanBlock) {
      // selected blocks fill the run's area from the front, near misses from the back: together they are at most all
      const uint32_t n_blk = len >> 4;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t b = h * 32u + lane;    // block of the run this lane answers for now: lanes in index order
        const uint32_t key = __shfl_sync(0xffffffffu, own[h], (lane & 7u) * 4u + (lane >> 3));
        const bool sel = b < n_blk && key >= tau_bits;
        const bool near = b < n_blk && !sel && key >= near_lo && key != 0u;
        const uint32_t bs = __ballot_sync(0xffffffffu, sel), bn = __ballot_sync(0xffffffffu, near);
        const uint32_t below = (1u << lane) - 1u;
        const uint2 e = make_uint2((start >> 4) + b, key);
        if (sel) list[n_list + __popc(bs & below)] = e;
        if (near) list[n_blk - 1u - n_near - __popc(bn & below)] = e;
        n_list += __popc(bs);
        n_near += __popc(bn);
      }
    }
    if (MODE == kScanElem) {
      const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
      // runs that do not raise the maximum leave its one address alone
      if (lane == 0 && top > ld_volatile_u32(&A.work[ch.seg].max_bits)) atomicMax(&A.work[ch.seg].max_bits, top);
    }
    if (lane == 0) {
      const uint32_t run = ch.run0 + rel / kRunElems;
      A.run_cnt[run] = n_list | n_near << 16;
      // tensors of several pieces: every piece's total, so that each CTA of `emit` can place itself
      if (sd.n_pad > 1u << piece_shift && (n_list | n_near))
        atomicAdd(reinterpret_cast<unsigned long long*>(A.piece_cnt + (run >> A.piece_shift)),
                  (unsigned long long)n_near << 32 | n_list);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// emit
// ------------------------------------------------------------------------------------------------
namespace {

struct EmitShared {
  alignas(16) uint2 stage[kStageItems];      // also read and written four words at a time
  uint32_t hist[2048];
  uint32_t pre[kMaxPieceRuns + 1];     // listed items in front of each run of the piece
  uint32_t near[kMaxPieceRuns + 1];    // near misses in front of each run of the piece
  uint32_t tmp[kEmitThreads / 32 + 1];
  uint32_t res[4];
  uint32_t word[4];                 // [0] may emit, [1] last CTA of the tensor, [2], [3] bases of a batch
  unsigned long long sum;           // listed items | near misses << 32 of the tensor
  uint32_t at[2];                   // piece of the tensor that holds a position, positions in front of it
  // where the tensor's entries go
  uint2* out[kMaxWorld];            // its region in each destination, when entries are plain pairs
  uint32_t n_out;                   // 0: they are not (narrow wire format, multicast, checksums)
  uint32_t off;                     // the tensor's first element
  uint32_t nb;
  int dest;
  uint64_t slot_off;
};
static_assert(alignof(EmitShared) % alignof(uint4) == 0 && offsetof(EmitShared, stage) % alignof(uint4) == 0,
              "16-byte accesses to EmitShared::stage");

// Run (of the piece) that holds item j: the last one that starts at or in front of it and is not empty.
__device__ __forceinline__ uint32_t run_of(const uint32_t* pre, uint32_t j) {
  uint32_t lo = 0, hi = kMaxPieceRuns;
#pragma unroll
  for (int s = 0; s < 7; ++s) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= j) lo = mid; else hi = mid;
  }
  return lo;
}
static_assert(kMaxPieceRuns == 128, "run_of halves 128 runs seven times");

// What a CTA of `emit` / `refill` works on.
struct Job {
  Piece pc;
  SegDesc sd;
  SegWork* wp;
  uint32_t epoch, kk;
  uint64_t slot_off;
  int dest;
  uint32_t nb;
  uint32_t piece_elems;       // of a full piece
  uint32_t len;               // elements of this one
};

__device__ __forceinline__ Job job_of(const SelectArgs& A, bool block) {
  Job J;
  J.pc = A.pieces[blockIdx.x];
  J.sd = A.segs[J.pc.seg];
  J.wp = &A.work[J.pc.seg];
  J.epoch = *A.epoch;
  J.kk = block ? (J.sd.k + 15u) / 16u : J.sd.k;
  J.slot_off = (uint64_t)(J.epoch & 1u) * A.slot_stride + J.sd.out_off;
  J.dest = dest_of(A, J.sd);
  J.nb = narrow_base_of(J.sd);
  J.piece_elems = kRunElems << A.piece_shift;
  J.len = min(J.piece_elems, J.sd.off + J.sd.n_pad - J.pc.start);
  return J;
}

// Where the tensor's entries go.  A CTA barrier follows before anybody reads it.
__device__ __forceinline__ void note_destinations(const SelectArgs& A, const Job& J, EmitShared& S) {
  const bool plain = J.nb == kNotNarrow && A.cksum_acc == nullptr && (J.dest >= 0 || A.out_mc == nullptr);
  const uint32_t n = J.dest >= 0 ? 1u : (uint32_t)A.world;
  if (threadIdx.x < n) S.out[threadIdx.x] = A.out[J.dest >= 0 ? (uint32_t)J.dest : threadIdx.x] + J.slot_off;
  if (threadIdx.x == 0) {
    S.n_out = plain ? n : 0u;
    S.off = J.sd.off;
    S.nb = J.nb;
    S.dest = J.dest;
    S.slot_off = J.slot_off;
  }
}

template <bool FRESH>
__device__ __forceinline__ void emit_and_keep(const SelectArgs& A, const EmitShared& S, uint32_t pos, uint32_t gi, float a) {
  const float sv = wire_value(S.nb, a);
  emit_entry(A, S.dest, S.nb, S.slot_off, pos, gi, sv);
  if (!FRESH) A.resid[gi] = a - sv;     // exactly zero unless the wire format rounds
}

// True in every thread of the CTA that finishes its tensor last; orders the other CTAs' stores in front of what follows.
// The CTA barrier orders a CTA's stores before its thread 0, whose release and acquire on the counter order the CTAs.
__device__ __forceinline__ bool last_of_tensor(const Job& J, EmitShared& S) {
  __syncthreads();
  if (J.pc.count == 1u) return true;
  if (threadIdx.x == 0) {
    const bool last = atom_add_acq_rel_gpu(&J.wp->pieces_done, 1u) == J.pc.count - 1u;
    if (last) J.wp->pieces_done = 0u;
    S.word[1] = last ? 1u : 0u;
  }
  __syncthreads();
  return S.word[1] != 0u;
}

// Picks the bin of `gh` that holds the kk-th largest of n_items keys: S.res = {bin, items still to be taken from it, items
// in it}.  One end bin is not counted and holds what the others do not: the top one or, for the histogram of the rest, bin 0.
__device__ __forceinline__ void plan_top(const uint32_t* gh, uint32_t copies, uint32_t n_items, uint32_t kk, bool rest_hist,
                                         EmitShared& S) {
  constexpr int kPer = kHistBins / kEmitThreads;
  const uint32_t tid = threadIdx.x;
  static_assert(kPer == 8, "two 16-byte loads per thread");
  // thread t owns the bins 2047 - 8 t ... 2040 - 8 t, highest first
  uint32_t h[kPer] = {};
#pragma unroll
  for (uint32_t r = 0; r < 8u; ++r) {
    if (r < copies) {
      const uint4* row = reinterpret_cast<const uint4*>(gh + (size_t)r * kHistBins + kHistBins - kPer * (tid + 1));
      const uint4 lo = __ldcg(row), hi = __ldcg(row + 1);
      h[0] += hi.w; h[1] += hi.z; h[2] += hi.y; h[3] += hi.x;
      h[4] += lo.w; h[5] += lo.z; h[6] += lo.y; h[7] += lo.x;
    }
  }
  if (tid == 0 && !rest_hist) h[0] = 0u;
  if (tid == kEmitThreads - 1 && rest_hist) h[kPer - 1] = 0u;
  uint32_t local = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) local += h[j];
  uint32_t total;
  uint32_t running = block_excl_scan(local, S.tmp, total);
  const uint32_t rest = n_items > total ? n_items - total : 0u;
  if (rest_hist) {
    if (tid == kEmitThreads - 1) h[kPer - 1] = rest;
  } else {
    if (tid == 0) h[0] = rest;
    else running += rest;
  }
  if (tid == 0) { S.res[0] = 0u; S.res[1] = 0u; S.res[2] = 0u; }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (running < kk && running + h[j] >= kk) {
      S.res[0] = kHistBins - 1 - (tid * kPer + j);
      S.res[1] = kk - running;
      S.res[2] = h[j];
    }
    running += h[j];
  }
  __syncthreads();
}

// Which pairs a CTA sends: S.stage in order; those that S.hist names; of a tensor whose values are the words of S.stage, those.
enum Staged : uint32_t { kInOrder = 0, kNamed = 1, kWords = 2 };

// Sends m of the CTA's pairs at positions pos, pos + 1, ... and takes them out of the residual.
//
// The kernels of this part run once per CTA and step from one section to the next: what they wait for, besides L2, is their own
// instructions.  With the stores to the destinations inlined wherever pairs are sent, and the searches below unrolled over
// registers, `emit` had 166 KB of code for top-k, and a section took microseconds of fetches the first time an SM came to it (the
// last CTA's search in a tensor 7 us for 100 items).  So sections that are used twice are functions, loops are loops, and items
// lie in shared memory: a 64 MB bucket takes 16 us instead of 23 (top-k, 1 %) and 9.6 instead of 12.9 (threshold-v16).  Without a
// residual the code that takes pairs out of it is left out as well (top-k, one tensor of 38.6 M elements: 28.9 us, now 27.6).
template <bool FRESH>
__device__ __noinline__ void send_staged(const SelectArgs& A, EmitShared& S, Staged how, uint32_t m, uint32_t pos) {
  const uint32_t* const words = reinterpret_cast<const uint32_t*>(S.stage);
  const uint32_t n_out = S.n_out, off = S.off;
  auto pair = [&](uint32_t q) {
    const uint32_t i = how == kInOrder ? q : S.hist[q];
    return how == kWords ? make_uint2(off + i, words[i]) : S.stage[i];
  };
  if (n_out == 0u) {
#pragma unroll 1
    for (uint32_t q = threadIdx.x; q < m; q += kEmitThreads) {
      const uint2 e = pair(q);
      emit_and_keep<FRESH>(A, S, pos + q, e.x, __uint_as_float(e.y));
    }
    return;
  }
  float* const resid = A.resid;
  auto take_out = [&](const uint2& e) {
    if (!FRESH) resid[e.x] = __uint_as_float(e.y) - __uint_as_float(e.y);      // zero, or what the next select drops
  };
  if (n_out == 1u) {
    uint2* const out = S.out[0] + pos;
#pragma unroll 4
    for (uint32_t q = threadIdx.x; q < m; q += kEmitThreads) {
      const uint2 e = pair(q);
      out[q] = e;
      take_out(e);
    }
    return;
  }
  // a pair is read once and goes to all of them: with a pass over the pairs per destination, one rank of eight (ResNet-152) took
  // 3 to 8 us of 365 longer
#pragma unroll 1
  for (uint32_t q = threadIdx.x; q < m; q += kEmitThreads) {
    const uint2 e = pair(q);
#pragma unroll 4
    for (uint32_t p = 0; p < n_out; ++p) S.out[p][pos + q] = e;
    take_out(e);
  }
}

// Sends the `n` marked items of a CTA's batch at positions base, base + 1, ...: bit u of `sel` marks the thread's item u, `ex`
// is the number of marked items in front of the thread's first.  They go through shared memory, so that the stores into the
// destinations are consecutive.
template <bool FRESH, int N>
__device__ __forceinline__ void send_marked(const SelectArgs& A, EmitShared& S, const uint32_t (&idx)[N], const uint32_t (&bits)[N],
                                            uint32_t sel, uint32_t ex, uint32_t n, uint32_t base) {
  uint2* const stage = S.stage;
#pragma unroll 1
  for (uint32_t w = 0; w < n; w += kStageItems) {
    uint32_t p = ex - w;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      if (sel >> u & 1u) {
        if (p < kStageItems) stage[p] = make_uint2(idx[u], bits[u]);
        ++p;
      }
    }
    __syncthreads();
    send_staged<FRESH>(A, S, kInOrder, min(kStageItems, n - w), base + w);
    __syncthreads();
  }
}

// Sends the items over the threshold's bin and notes those inside it.  `emitted` / `noted`: counts so far when one CTA
// has the whole tensor; several CTAs draw theirs from the tensor's counters, once per batch.
template <bool FRESH, int N>
__device__ __forceinline__ void emit_top_batch(const SelectArgs& A, const Job& J, EmitShared& S, uint2* undecided,
                                               const uint32_t (&idx)[N], const uint32_t (&bits)[N], uint32_t key_lo,
                                               uint32_t key_hi, uint32_t& emitted, uint32_t& noted) {
  uint32_t sel = 0, und = 0;
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const uint32_t key = bits[u] & 0x7fffffffu;
    const bool there = idx[u] != kSentinelIdx;
    sel |= (uint32_t)(there && key >= key_hi) << u;
    und |= (uint32_t)(there && key >= key_lo && key < key_hi) << u;
  }
  uint32_t total;
  const uint32_t ex = block_excl_scan(__popc(sel) | __popc(und) << 16, S.tmp, total);
  const uint32_t t_sel = total & 0xffffu, t_und = total >> 16;
  uint32_t b_sel = emitted, b_und = noted;
  if (J.pc.count > 1u) {
    if (threadIdx.x == 0) {
      S.word[2] = t_sel ? atomicAdd(&J.wp->out_cursor, t_sel) : 0u;
      S.word[3] = t_und ? atomicAdd(&J.wp->cand_cnt, t_und) : 0u;
    }
    __syncthreads();
    b_sel = S.word[2];
    b_und = S.word[3];
  }
  emitted += t_sel;
  noted += t_und;
  uint32_t q = b_und + (ex >> 16);
#pragma unroll
  for (int u = 0; u < N; ++u)
    if (und >> u & 1u) undecided[q++] = make_uint2(idx[u], bits[u]);
  send_marked<FRESH, N>(A, S, idx, bits, sel, ex & 0xffffu, t_sel, b_sel);
}

// Keys of the last two octaves under the largest differ from it in these bits: where the best of a distribution are looked for
// first.
constexpr uint32_t kTwoOctaves = 24u;
constexpr uint32_t kNoCut = 0xFFFFFFFFu;       // a search that found none; no key

// Where the best `take` of n items in S.stage end (larger key first, equal keys by lower id): {key, id - id_lo} of the
// lowest-ranked one taken; 1 <= take <= n.  The items are pairs (id, key or signed value), or the words (keys or signed values) of
// one tensor, whose ids count from 0.  No key lies above `top`; ids lie in [id_lo, id_lo + n_ids).
// A radix search, 8 bits at a time with a bin per thread.  Its digits are those of the distance to `top`, so that they differ
// where the cut is: of the `open` lowest bits first, which is a guess; a cut further away is found in all 31.  Keys have no more
// than those, so a search that covers them fails only where the items are not what the caller says (a key over `top`, fewer than
// `take` of them): it then reports kBadCandidate and returns kNoCut.  At most twelve digits in all.
__device__ __noinline__ uint2 find_cut(EmitShared& S, uint32_t* status, bool words, uint32_t n, uint32_t take, uint32_t top,
                                       uint32_t open, uint32_t id_lo, uint32_t n_ids) {
  static_assert(kEmitThreads == 256, "a bin per thread");
  const uint32_t tid = threadIdx.x, lane = tid & 31u, n_up = (n + kEmitThreads - 1u) & ~(kEmitThreads - 1u);
  const uint32_t* const word = reinterpret_cast<const uint32_t*>(S.stage);
  auto distance = [&](uint32_t i) { return top - ((words ? word[i] : S.stage[i].y) & 0x7fffffffu); };
  auto id_of = [&](uint32_t i) { return words ? i : S.stage[i].x - id_lo; };
  uint32_t prefix = 0, rem = take, ties = 0, d = 0;
  bool by_id = false, all_bits = open >= 31u;
  top = min(top, 0x7fffffffu);      // a threshold with its sign bit set lies over every key
#pragma unroll 1
  for (;;) {
    // among the values whose bits from `open` upwards are `prefix`: the digit of the rem-th smallest
    const uint32_t w = min(open, 8u), shift = open - w;
    S.hist[tid] = 0u;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = tid; i < n_up; i += kEmitThreads) {
      uint32_t bin = 256u;
      if (i < n) {
        uint32_t v = distance(i);
        const bool counts = !by_id || v == d;
        if (by_id) v = id_of(i);
        if (counts && v >> open == prefix) bin = v >> shift & ((1u << w) - 1u);
      }
      int same;
      __match_all_sync(0xffffffffu, bin, &same);      // equal values would queue up at one counter
      if (bin < 256u && (!same || lane == 0u)) atomicAdd(&S.hist[bin], same ? 32u : 1u);
    }
    __syncthreads();
    const uint32_t h = S.hist[tid];
    if (tid == 0) S.res[2] = 0u;
    uint32_t total;
    const uint32_t ex = block_excl_scan(h, S.tmp, total);
    if (ex < rem && ex + h >= rem) { S.res[0] = tid; S.res[1] = rem - ex; S.res[2] = h; }
    __syncthreads();
    ties = S.res[2];
    if (ties == 0u) {
      if (all_bits || by_id) {
        if (tid == 0) set_status(status, kBadCandidate);
        return make_uint2(kNoCut, 0u);
      }
      open = 31u;      // the guess was wrong
      prefix = 0u;
      all_bits = true;
      continue;
    }
    prefix = prefix << w | S.res[0];
    rem = S.res[1];
    open = shift;
    if (by_id) {
      if (open == 0u) break;
      continue;
    }
    if (rem == ties) break;
    if (open == 0u) {      // more items share the key than are wanted: the rem-th smallest id
      d = prefix;
      by_id = true;
      open = 32u - __clz(n_ids);
      prefix = 0u;
    }
  }
  uint32_t last = prefix;
  if (!by_id) {
    // all items that share these bits: the furthest of them, and the highest id there
    uint32_t mx = 0;
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += kEmitThreads)
      if (distance(i) >> open == prefix) mx = max(mx, distance(i));
    d = block_max_u32(mx, S.tmp);
    mx = 0;
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += kEmitThreads)
      if (distance(i) == d) mx = max(mx, id_of(i));
    last = block_max_u32(mx, S.tmp);
  }
  return make_uint2(top - d, last);
}

// The best `take` of c <= kPickMax candidates (id, key or signed value): they come to S.stage, and S.hist names those taken, the
// lowest-ranked one last.  Returns its key, or kNoCut (S.hist then names none).  `top`, `open`: see find_cut.
__device__ __forceinline__ uint32_t pick_few(const SelectArgs& A, const uint2* cand, uint32_t c, uint32_t take, uint32_t top,
                                             uint32_t open, uint32_t id_lo, uint32_t n_ids, EmitShared& S) {
  static_assert(kPickMax <= kStageItems && kPickMax <= 2048, "the candidates fit EmitShared::stage, their numbers EmitShared::hist");
  constexpr int kPer = kPickMax / kEmitThreads;
  const uint32_t tid = threadIdx.x;
  uint2 e[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u)
    if (u * kEmitThreads + tid < c) e[u] = __ldcg(cand + u * kEmitThreads + tid);
#pragma unroll
  for (int u = 0; u < kPer; ++u)
    if (u * kEmitThreads + tid < c) S.stage[u * kEmitThreads + tid] = e[u];
  if (tid == 0) S.word[2] = 0u;
  __syncthreads();
  const uint2 cut = find_cut(S, A.status, false, c, take, top, open, id_lo, n_ids);
  __syncthreads();      // the search is through with S.hist
  if (cut.x == kNoCut) return kNoCut;
#pragma unroll 1
  for (uint32_t i = tid; i < c; i += kEmitThreads) {
    const uint32_t key = S.stage[i].y & 0x7fffffffu, id = S.stage[i].x - id_lo;
    if (key > cut.x || (key == cut.x && id <= cut.y))
      S.hist[key == cut.x && id == cut.y ? take - 1u : atomicAdd(&S.word[2], 1u)] = i;
  }
  __syncthreads();
  return cut.x;
}

// Top-k of a small tensor: its values lie in shared memory.  Returns the k-th largest key, or kNoCut.
template <bool FRESH>
__device__ __forceinline__ uint32_t top_direct(const SelectArgs& A, const Job& J, EmitShared& S) {
  static_assert(kTopDirect == 2u * kStageItems && kTopDirect == 16u * kEmitThreads, "the values are the words of EmitShared::stage");
  const uint32_t tid = threadIdx.x;
  uint4* const words = reinterpret_cast<uint4*>(S.stage);
  uint32_t top = 0;
  float4 v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t i = (u * kEmitThreads + tid) * 4u;
    v[u] = i < J.sd.n_pad ? load4<FRESH>(A, J.sd.off + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float4 e = resid4<FRESH>(A, J.sd.off + (u * kEmitThreads + tid) * 4u, v[u]);
    const uint4 a = make_uint4(__float_as_uint(e.x), __float_as_uint(e.y), __float_as_uint(e.z), __float_as_uint(e.w));
    words[u * kEmitThreads + tid] = a;
    top = max(max(max(top, a.x & 0x7fffffffu), max(a.y & 0x7fffffffu, a.z & 0x7fffffffu)), a.w & 0x7fffffffu);
  }
  top = block_max_u32(top, S.tmp);
  const uint2 cut = find_cut(S, A.status, true, J.sd.n_pad, J.kk, top, kTwoOctaves, 0u, J.sd.n_pad);
  if (cut.x == kNoCut) return kNoCut;
  uint32_t take = 0;      // bit 4 u + e: element e of the thread's u-th four
#pragma unroll 1
  for (uint32_t u = 0; u < 4u; ++u) {
    const uint32_t i = (u * kEmitThreads + tid) * 4u;
    const uint4 v = words[u * kEmitThreads + tid];
    const uint32_t key[4] = {v.x & 0x7fffffffu, v.y & 0x7fffffffu, v.z & 0x7fffffffu, v.w & 0x7fffffffu};
#pragma unroll
    for (uint32_t e = 0; e < 4u; ++e)
      take |= (uint32_t)(i < J.sd.n_pad && (key[e] > cut.x || (key[e] == cut.x && i + e <= cut.y))) << (4u * u + e);
  }
  uint32_t total;
  const uint32_t ex = block_excl_scan(__popc(take), S.tmp, total);
#pragma unroll 1
  for (uint32_t w = 0; w < total; w += 2048u) {
    uint32_t p = ex - w;
#pragma unroll 1
    for (uint32_t left = take; left != 0u; left &= left - 1u, ++p) {
      const uint32_t b = __ffs(left) - 1u;
      if (p < 2048u) S.hist[p] = ((b >> 2) * kEmitThreads + tid) * 4u + (b & 3u);
    }
    __syncthreads();
    send_staged<FRESH>(A, S, kWords, min(2048u, total - w), w);
    __syncthreads();
  }
  return cut.x;
}

// The same for more items than shared memory holds: a radix search over the bits that the keys of `cand` leave open, 11 at a time.
// Fixed digits of the whole key put nearly all pairs, which lie close together, on one counter: 25,000 adds to one address of
// shared memory took longer than all passes over the pairs.  Ids lie in [id_lo, id_lo + n_ids).
__device__ __forceinline__ uint2 cut_of_many(const uint2* cand, uint32_t c, uint32_t take, uint32_t id_lo, uint32_t n_ids,
                                             EmitShared& S) {
  constexpr int kIlp = 8;              // independent loads in flight per thread
  constexpr uint32_t kDigit = 11u;
  const uint32_t tid = threadIdx.x;
  auto each = [&](auto f) {
    for (uint32_t i0 = tid; i0 < c; i0 += kEmitThreads * kIlp) {
      uint2 e[kIlp];
#pragma unroll
      for (int u = 0; u < kIlp; ++u) e[u] = i0 + u * kEmitThreads < c ? __ldcg(cand + i0 + u * kEmitThreads) : make_uint2(0u, 0u);
#pragma unroll
      for (int u = 0; u < kIlp; ++u)
        if (i0 + u * kEmitThreads < c) f(make_uint2(e[u].x, e[u].y & 0x7fffffffu));
    }
  };
  // The digit of the rem-th value, counted from the largest (`down`) or the smallest one: S.res = {digit, values still to be
  // taken among those that have it, their number}.
  auto pick_digit = [&](uint32_t n_bins, uint32_t rem, bool down) {
    constexpr int kPer = (1 << kDigit) / kEmitThreads;
    uint32_t h[kPer], local = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t d = kPer * tid + j;
      h[j] = d < n_bins ? S.hist[down ? n_bins - 1u - d : d] : 0u;
      local += h[j];
    }
    uint32_t total;
    uint32_t ex = block_excl_scan(local, S.tmp, total);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t d = kPer * tid + j;
      if (ex < rem && ex + h[j] >= rem) { S.res[0] = down ? n_bins - 1u - d : d; S.res[1] = rem - ex; S.res[2] = h[j]; }
      ex += h[j];
    }
    __syncthreads();
  };
  uint32_t mn = 0xFFFFFFFFu, mx = 0;
  each([&](const uint2& e) { mn = min(mn, e.y); mx = max(mx, e.y); });
  mn = ~block_max_u32(~mn, S.tmp);
  mx = block_max_u32(mx, S.tmp);
  uint32_t t = 0, rem = take, ties = c;
  for (uint32_t open = 32u - __clz(mx - mn); open != 0u;) {
    const uint32_t w = min(open, kDigit), shift = open - w, n_bins = 1u << w;
    for (uint32_t b = tid; b < n_bins; b += kEmitThreads) S.hist[b] = 0u;
    __syncthreads();
    each([&](const uint2& e) {
      const uint32_t v = e.y - mn;
      if (v >> open == t) atomicAdd(&S.hist[v >> shift & (n_bins - 1u)], 1u);
    });
    __syncthreads();
    pick_digit(n_bins, rem, true);
    t = t << w | S.res[0];
    rem = S.res[1];
    ties = S.res[2];
    open = shift;
    __syncthreads();
  }
  const uint32_t key = mn + t;
  if (rem == ties) {      // all pairs of this key: the highest id among them
    uint32_t last = 0;
    each([&](const uint2& e) { if (e.y == key) last = max(last, e.x); });
    return make_uint2(key, block_max_u32(last, S.tmp));
  }
  uint32_t id = 0;        // the rem-th smallest id
  for (uint32_t open = 32u - __clz(n_ids); open != 0u;) {
    const uint32_t w = min(open, kDigit), shift = open - w, n_bins = 1u << w;
    for (uint32_t b = tid; b < n_bins; b += kEmitThreads) S.hist[b] = 0u;
    __syncthreads();
    each([&](const uint2& e) {
      const uint32_t v = e.x - id_lo;
      if (e.y == key && v >> open == id) atomicAdd(&S.hist[v >> shift & (n_bins - 1u)], 1u);
    });
    __syncthreads();
    pick_digit(n_bins, rem, false);
    id = id << w | S.res[0];
    rem = S.res[1];
    open = shift;
    __syncthreads();
  }
  return make_uint2(key, id_lo + id);
}

// Last CTA of a tensor, c > kPickMax candidates: sends the best `take` of them behind the `done` items that are in the stream,
// the lowest-ranked one last.  Returns its key.  `list` is the area of the tensor's lists, which nobody reads any more.  Ranked
// by one CTA of 1024 threads, which drew a stream position per item from one address and copied a block with one thread,
// this took up to 0.1 ms for the 25,000 undecided items of a 64 MB bucket whose gradients had changed in scale.
// Rare, but inline: as a function of its own the loops over the candidates took a quarter longer (a threshold-v16 tensor of 16.8 M
// elements whose threshold is far too high, 10 % kept: 5.4 to 6.3 ms against 3.5; 1 %: 2.8 against 2.4).
template <bool kBlock, bool FRESH>
__device__ __forceinline__ uint32_t send_best(const SelectArgs& A, const Job& J, EmitShared& S, const uint2* cand, uint32_t c,
                                              uint32_t take, uint32_t done, uint2* list) {
  constexpr uint32_t kPerItem = kBlock ? 16u : 1u;
  constexpr int kIlp = kStageItems / kEmitThreads;
  const uint32_t tid = threadIdx.x;
  const uint2 cut = cut_of_many(cand, c, take, kBlock ? J.sd.off >> 4 : J.sd.off, kBlock ? J.sd.n_pad >> 4 : J.sd.n_pad, S);
  uint32_t base = 0;
  for (uint32_t i0 = 0; i0 < c; i0 += kStageItems) {
    uint32_t id[kIlp], taken = 0;
#pragma unroll
    for (int u = 0; u < kIlp; ++u) {
      const uint32_t i = i0 + u * kEmitThreads + tid;
      uint2 e = i < c ? __ldcg(cand + i) : make_uint2(0xFFFFFFFFu, 0u);
      e.y &= 0x7fffffffu;
      id[u] = e.x;
      const bool is_last = e.y == cut.x && e.x == cut.y;
      if (is_last) list[take - 1u].x = e.x;
      taken |= (uint32_t)(i < c && !is_last && (e.y > cut.x || (e.y == cut.x && e.x < cut.y))) << u;
    }
    uint32_t n;
    uint32_t at = base + block_excl_scan(__popc(taken), S.tmp, n);
#pragma unroll
    for (int u = 0; u < kIlp; ++u)
      if (taken >> u & 1u) list[at++].x = id[u];
    base += n;
  }
  __syncthreads();
  uint2* const stage = S.stage;
  for (uint32_t t0 = 0; t0 < take * kPerItem; t0 += kStageItems) {
#pragma unroll
    for (int u = 0; u < kIlp; ++u) {
      const uint32_t t = t0 + u * kEmitThreads + tid;
      uint2 e = make_uint2(0u, 0u);
      if (t < take * kPerItem) {
        e.x = __ldcg(&list[t / kPerItem].x) * kPerItem + t % kPerItem;
        e.y = __float_as_uint(resid1<FRESH>(A, e.x));
      }
      stage[u * kEmitThreads + tid] = e;
    }
    __syncthreads();
    const uint32_t p0 = done * kPerItem + t0;      // the last block may be cut off at k
    send_staged<FRESH>(A, S, kInOrder, min(min(kStageItems, take * kPerItem - t0), J.sd.k > p0 ? J.sd.k - p0 : 0u), p0);
    __syncthreads();
  }
  return cut.x;
}

// Top-k, last CTA of a tensor: the best `rem` of the `c` undecided items complete the stream.  Returns the k-th largest key, or
// kNoCut.
template <bool FRESH>
__device__ __forceinline__ uint32_t settle_top(const SelectArgs& A, const Job& J, EmitShared& S, const uint2* undecided,
                                               uint32_t c, uint32_t rem, uint32_t key_lo, uint32_t key_hi) {
  const uint32_t done = J.kk - rem;
  if (c <= kPickMax) {
    const uint32_t t_key = pick_few(A, undecided, c, rem, key_hi - 1u, 32u - __clz(key_hi - 1u - key_lo), J.sd.off, J.sd.n_pad, S);
    if (t_key != kNoCut) send_staged<FRESH>(A, S, kNamed, rem, done);
    return t_key;
  }
  return send_best<false, FRESH>(A, J, S, undecided, c, rem, done, A.cand + J.sd.off);
}

// Sends the items [j0, j1) of one piece at positions base + j; items and positions are in index order.  The dependent loads
// (list, residual) of a thread travel together; the entries then pass through shared memory as above.
template <bool kBlock, bool FRESH>
__device__ __forceinline__ void send_range(const SelectArgs& A, const Job& J, EmitShared& S, const uint2* lists,
                                           uint32_t base, uint32_t j0, uint32_t j1) {
  constexpr uint32_t kPerItem = kBlock ? 16u : 1u, kArea = kBlock ? kRunBlocks : kRunElems;
  const uint32_t end = j1 * kPerItem;
#pragma unroll 1
  for (uint32_t t0 = j0 * kPerItem; t0 < end; t0 += kStageItems) {
    if (kBlock) {
      // four lanes to a block
      constexpr int kPer = kStageItems / 4 / kEmitThreads;
      uint32_t gi[kPer];
      float4 a[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const uint32_t t = t0 + (u * kEmitThreads + threadIdx.x) * 4u, j = t / 16u, run = run_of(S.pre, j);
        if (t < end) gi[u] = lists[run * kArea + (j - S.pre[run])].x * 16u + (t & 15u);
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u)
        if (t0 + (u * kEmitThreads + threadIdx.x) * 4u < end) a[u] = load4<FRESH>(A, gi[u]);
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const uint32_t q = (u * kEmitThreads + threadIdx.x) * 4u;
        if (t0 + q < end) {
          const float4 v = resid4<FRESH>(A, gi[u], a[u]);
          uint4* const to = reinterpret_cast<uint4*>(&S.stage[q]);
          to[0] = make_uint4(gi[u], __float_as_uint(v.x), gi[u] + 1u, __float_as_uint(v.y));
          to[1] = make_uint4(gi[u] + 2u, __float_as_uint(v.z), gi[u] + 3u, __float_as_uint(v.w));
        }
      }
    } else {
      // 256 consecutive items to a warp: a lane's items are 32 apart, and its run moves on with them
      constexpr int kPer = kStageItems / kEmitThreads;
      const uint32_t q0 = (threadIdx.x & ~31u) * kPer + (threadIdx.x & 31u);
      uint32_t run = run_of(S.pre, t0 + q0);
      uint2 e[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const uint32_t j = t0 + q0 + u * 32u;
        if (j < end) {
          while (S.pre[run + 1u] <= j) ++run;
          e[u] = lists[run * kArea + (j - S.pre[run])];
        }
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u)
        if (t0 + q0 + u * 32u < end) S.stage[q0 + u * 32u] = e[u];
    }
    __syncthreads();
    // a truncated last block leaves the residual exact: only emitted elements are cleared
    const uint32_t p0 = base * kPerItem + t0;
    send_staged<FRESH>(A, S, kInOrder, min(min(kStageItems, end - t0), J.sd.k > p0 ? J.sd.k - p0 : 0u), p0);
    __syncthreads();
  }
}

// Threshold-v16: the blocks of a piece that hold something and are not on its lists (`total` listed blocks), as candidates of
// the fill.  A listed block is sent whenever the stream is short; what the narrow wire format's rounding leaves of it in the
// residual waits for the next select, so that a stream names an element once.  The lists, and not the residual, say which
// blocks these are: other CTAs of the tensor may be sending them now.  Returns the number collected by this CTA.  Inline: as a
// function of its own it made the select of a tensor of 3 M elements whose threshold is twice too high 476 us instead of 461.
template <bool FRESH>
__device__ __forceinline__ uint32_t collect_unlisted(const SelectArgs& A, const Job& J, EmitShared& S, const uint2* area,
                                                     uint32_t total, uint2* cand) {
  constexpr uint32_t kQuads = kEmitThreads / 4, kKeys = 8;      // blocks side by side; keys a lane keeps per round
  static_assert(kMaxPieceElems / 16u / 32u <= 2048u, "a bit per block of a piece fits EmitShared::hist");
  const uint32_t tid = threadIdx.x, first = J.pc.start >> 4;
  const uint32_t n_blk = J.len >> 4;
  for (uint32_t w = tid; w < kMaxPieceElems / 16u / 32u; w += kEmitThreads) S.hist[w] = 0u;
  __syncthreads();
  for (uint32_t j = tid; j < total; j += kEmitThreads) {
    const uint32_t run = run_of(S.pre, j), b = area[run * kRunBlocks + (j - S.pre[run])].x - first;
    atomicOr(&S.hist[b >> 5], 1u << (b & 31u));
  }
  __syncthreads();
  const uint32_t src = J.pc.start + (tid & 3u) * 4u;
  uint32_t done = 0;
  for (uint32_t b0 = 0; b0 < n_blk; b0 += kQuads * kKeys * 4u) {
    uint32_t key[kKeys], there = 0;
#pragma unroll
    for (uint32_t s = 0; s < kKeys; ++s) {
      float4 a[4];
      uint32_t left_out = 0;
#pragma unroll
      for (uint32_t q = 0; q < 4u; ++q) {   // independent loads in flight
        const uint32_t b = b0 + (s * 4u + q) * kQuads + (tid >> 2);
        const bool take = b < n_blk && !(S.hist[b >> 5] >> (b & 31u) & 1u);
        a[q] = take ? load4<FRESH>(A, src + b * 16u) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (FRESH && !take) left_out |= 1u << q;
      }
#pragma unroll
      for (uint32_t q = 0; q < 4u; ++q) {
        // a block left out stays zero: no end of the tensor lies behind ~0
        const uint32_t at = left_out >> q & 1u ? kSentinelIdx : src + (b0 + (s * 4u + q) * kQuads + (tid >> 2)) * 16u;
        const uint32_t k = __float_as_uint(quad_l1(resid4<FRESH>(A, at, a[q])));
        if ((tid & 3u) == q) key[s] = k;
      }
      there |= (key[s] != 0u ? 1u : 0u) << s;
    }
    uint32_t n;
    const uint32_t ex = block_excl_scan(__popc(there), S.tmp, n);
    uint32_t base = done;
    if (J.pc.count > 1u) {
      if (tid == 0) S.word[2] = n ? atomicAdd(&J.wp->cand_cnt, n) : 0u;
      __syncthreads();
      base = S.word[2];
    }
    uint32_t at = base + ex;
#pragma unroll
    for (uint32_t s = 0; s < kKeys; ++s)
      if (there >> s & 1u) cand[at++] = make_uint2(first + b0 + (s * 4u + (tid & 3u)) * kQuads + (tid >> 2), key[s]);
    done += n;
  }
  return done;
}

// The candidates do not reach down to the k-th largest value: a histogram of the rest.
template <bool FRESH>
__device__ __noinline__ void count_rest(const SelectArgs& A, EmitShared& S) {
  const uint32_t tid = threadIdx.x;
  const Job J = job_of(A, false);
  const uint32_t cut = top_cut(A.state[J.pc.seg], J.sd.n_pad);
  for (uint32_t b = tid; b < (uint32_t)kHistBins; b += kEmitThreads) S.hist[b] = 0u;
  __syncthreads();
  uint32_t zeros = 0;
  auto count = [&](const float4& a) {
    const uint32_t key[4] = {key_bits(a.x), key_bits(a.y), key_bits(a.z), key_bits(a.w)};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (key[e] == 0u) ++zeros;
      else if (key[e] < cut) atomicAdd(&S.hist[rest_bin(key[e], cut)], 1u);
    }
  };
  constexpr int kQuads = 4;
  uint32_t i = tid * 4u;
#pragma unroll 1
  for (; i + (kQuads - 1) * kEmitThreads * 4u < J.len; i += kQuads * kEmitThreads * 4u) {
    float4 a[kQuads];
#pragma unroll
    for (int u = 0; u < kQuads; ++u) a[u] = load4<FRESH>(A, J.pc.start + i + u * kEmitThreads * 4u);
#pragma unroll
    for (int u = 0; u < kQuads; ++u) count(resid4<FRESH>(A, J.pc.start + i + u * kEmitThreads * 4u, a[u]));
  }
#pragma unroll 1
  for (; i < J.len; i += kEmitThreads * 4u) count(resid4<FRESH>(A, J.pc.start + i, load4<FRESH>(A, J.pc.start + i)));
  block_excl_scan(zeros, S.tmp, zeros);
  uint32_t* gh = A.hist_rest + (size_t)J.pc.seg * kHistBins;
  for (uint32_t b = tid; b < (uint32_t)kHistBins; b += kEmitThreads)
    if (S.hist[b]) atomicAdd(gh + b, S.hist[b]);
  if (tid == 0) A.run_cnt[blockIdx.x << A.piece_shift] = zeros;     // this CTA has read its own counts
}

// Thread 0 of the last CTA of a top-k tensor: what the next select starts from.  Every candidate costs a list entry and a
// histogram count; candidates that fall short cost two more passes over the tensor by the emitting kernels (a step of 16 M
// elements takes up to 125 us more, one of 3 M 60) and hold up the whole bucket.  How many more
// candidates there were than entries says how near the cut came to falling short.  The threshold of one batch differs from
// that of the next, so the window grows at once when few were spare and shrinks by a few per cent a step when many were.
__device__ __forceinline__ void step_top(const SelectArgs& A, const Job& J, SegState ss, uint32_t t_key, uint32_t listed) {
  float w = fminf(window_or(ss.reserved[0], kTopWindowDefault), kTopWindowMax);
  const float k = (float)J.kk, spare = (float)listed - k, noise = 4.f * sqrtf(k);
  if (spare < 0.f) w *= 2.f;
  else if (spare < noise + 0.15f * k) w *= 1.3f;
  else if (spare > 2.f * noise + 0.3f * k) w *= 0.97f;
  if (J.sd.n_pad > kTopDirect) ss.reserved[0] = __float_as_uint(fminf(fmaxf(w, kTopWindowMin), kTopWindowMax));
  ss.reserved[1] = t_key;
  if (t_key < (uint32_t)(kHistBins / 2) << (kFineShift + 1)) { ss.hist_shift = 0; ss.hist_base = 0; }
  else centre_window(ss, t_key);
  A.state[J.pc.seg] = ss;
}

}  // namespace

template <int MODE, bool FRESH>
__global__ void __launch_bounds__(kEmitThreads, 4) k_emit(const __grid_constant__ SelectArgs A) {
  __shared__ EmitShared S;
  constexpr bool kBlock = MODE == kScanBlock;
  const uint32_t tid = threadIdx.x;
  const Job J = job_of(A, kBlock);
  // all of this was written in front of `scan`
  const SegState ss = A.state[J.pc.seg];
  note_destinations(A, J, S);
  behind_previous();
  const uint32_t cnt = tid < J.pc.n_runs ? A.run_cnt[(blockIdx.x << A.piece_shift) + tid] : 0u;
  const bool ok = ld_volatile_u32(A.status) == kOk;

  if (!(J.sd.reserved & kSegSkip)) {
    // listed items and near misses of this piece and of the tensor; listed items in front of this piece, and of the fullest one
    unsigned long long all = 0ull;
    uint32_t ahead = 0, most = 0;
    if (J.pc.count > 1u)
      for (uint32_t t = tid; t < J.pc.count; t += kEmitThreads) {
        const unsigned long long n = A.piece_cnt[J.pc.first + t];
        all += n;
        if (MODE != kScanTop) {
          if (t < J.pc.index) ahead += (uint32_t)n;
          most = max(most, (uint32_t)n);
        }
      }
    if (tid == 0) { S.sum = 0ull; S.at[0] = 0u; S.at[1] = 0u; }
    uint32_t total, near_total = 0;
    uint32_t ex = block_excl_scan(cnt & 0xffffu, S.tmp, total);
    if (tid <= kMaxPieceRuns) S.pre[tid] = ex;
    if (kBlock) {
      const uint32_t nex = block_excl_scan(cnt >> 16, S.tmp, near_total);
      if (tid <= kMaxPieceRuns) S.near[tid] = nex;
    }
    uint32_t found = total, c_near = near_total;
    bool even = true;       // no CTA gets much more than its share when each sends the items of its own piece
    if (J.pc.count > 1u) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) all += __shfl_xor_sync(0xffffffffu, all, d);
      if (MODE != kScanTop) {
        ahead = __reduce_add_sync(0xffffffffu, ahead);
        most = __reduce_max_sync(0xffffffffu, most);
      }
      if ((tid & 31u) == 0u && all) {
        atomicAdd(&S.sum, all);
        if (MODE != kScanTop) {
          atomicAdd(&S.at[0], ahead);
          atomicMax(&S.at[1], most);
        }
      }
      __syncthreads();
      found = (uint32_t)S.sum;
      c_near = (uint32_t)(S.sum >> 32);
      ahead = S.at[0];
      constexpr uint32_t kPerItem = kBlock ? 16u : 1u;
      even = S.at[1] * kPerItem <= 2u * max(kStageItems, min(found, J.kk) / J.pc.count * kPerItem);
    }
    const bool short_of = found < J.kk;
    // will this CTA store into the destinations?  Then they must have consumed the slot.
    if (tid == 0) S.word[0] = ok && acks_arrived(A, J.epoch) ? 1u : 0u;
    __syncthreads();
    const bool may = S.word[0] != 0u;
    uint2* const area = A.cand + (kBlock ? J.pc.start >> 4 : J.pc.start);
    constexpr uint32_t kArea = kBlock ? kRunBlocks : kRunElems;      // list slots per run

    if (MODE == kScanTop) {
      uint2* const undecided = A.cand + A.n_total + J.sd.off;
      uint32_t emitted = 0, noted = 0, key_lo = 0, key_hi = 0;
      const bool direct = J.sd.n_pad <= kTopDirect;
      if (direct) {
        if (may) {
          const uint32_t t_key = top_direct<FRESH>(A, J, S);
          if (tid == 0 && t_key != kNoCut) step_top(A, J, ss, t_key, 0u);
        }
      } else if (short_of && ok) {
        count_rest<FRESH>(A, S);      // for `refill`
      } else if (!short_of) {
        plan_top(A.hist_top + (size_t)J.pc.first * kHistBins, hist_copies(J.sd.n_pad), found, J.kk, false, S);
        top_bin_range(S.res[0], top_centre(ss), key_lo, key_hi);
        if (may) {
          constexpr int kItems = 8;
#pragma unroll 1
          for (uint32_t j0 = 0; j0 < total; j0 += kEmitThreads * kItems) {
            uint32_t idx[kItems], bits[kItems];
            uint32_t j = j0 + tid * kItems, run = run_of(S.pre, j);      // the stream keeps the lists' order: the update reads it faster
#pragma unroll
            for (int u = 0; u < kItems; ++u, ++j) {
              idx[u] = kSentinelIdx;
              bits[u] = 0u;
              if (j < total) {
                while (S.pre[run + 1u] <= j) ++run;
                const uint2 e = area[run * kArea + (j - S.pre[run])];
                idx[u] = e.x;
                bits[u] = e.y;
              }
            }
            emit_top_batch<FRESH, kItems>(A, J, S, undecided, idx, bits, key_lo, key_hi, emitted, noted);
          }
        }
      }
      const uint32_t rem = S.res[1];     // read before the helpers below reuse the words
      if (!direct && last_of_tensor(J, S)) {
        if (!short_of) {
          const uint32_t c = J.pc.count == 1u ? noted : __ldcg(&J.wp->cand_cnt);
          if (may && rem != 0u && rem <= c) {
            const uint32_t t_key = settle_top<FRESH>(A, J, S, undecided, c, rem, key_lo, key_hi);
            if (tid == 0 && t_key != kNoCut) step_top(A, J, ss, t_key, found);
          } else if (may && tid == 0) {
            set_status(A.status, kBadCandidate);   // cannot happen: the histogram counted these very items
          }
        } else if (tid == 0 && ok) {
          J.wp->refill = 1u;                       // `refill` selects this tensor
          J.wp->found = found;
          atomicAdd(A.refills, 1u);
        }
        __syncthreads();
        if (tid == 0) { J.wp->out_cursor = 0u; J.wp->cand_cnt = 0u; }
        for (uint32_t t = tid; t < J.pc.count; t += kEmitThreads) A.piece_cnt[J.pc.first + t] = 0ull;
        uint4* gh = reinterpret_cast<uint4*>(A.hist_top + (size_t)J.pc.first * kHistBins);
        for (uint32_t b = tid; b < hist_copies(J.sd.n_pad) * (kHistBins / 4); b += kEmitThreads) gh[b] = make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
      uint2* const nears = A.cand + (A.n_total >> 4) + (J.sd.off >> 4);     // block mode: one slot per block of the tensor
      // Do the near misses not suffice (or is there no threshold yet), then every block that holds something and is not over
      // the threshold is a candidate.  Each CTA collects those of its own piece.
      const bool rescan = kBlock && short_of && (!ss.inited || c_near < J.kk - found);
      uint32_t collected = 0;
      if (rescan) {
        collected = collect_unlisted<FRESH>(A, J, S, area, total, nears);
      } else if (kBlock && short_of && near_total) {
        // the fill needs the tensor's near misses in one place
        if (tid == 0) S.word[2] = J.pc.count == 1u ? 0u : atomicAdd(&J.wp->cand_cnt, near_total);
        __syncthreads();
        const uint32_t nb0 = S.word[2];
        for (uint32_t j = tid; j < near_total; j += kEmitThreads) {
          const uint32_t run = run_of(S.near, j);
          const uint32_t in_seg = J.pc.start - J.sd.off + run * kRunElems;
          const uint32_t n_blk = min(kRunElems, J.sd.n_pad - in_seg) >> 4;
          nears[nb0 + j] = area[run * kArea + n_blk - 1u - (j - S.near[run])];
        }
      }
      // The first kk items in index order are sent, as a rule by the CTA of their piece.  A threshold that lags behind lets nearly
      // everything pass, and the budget then ends within the tensor's first piece; items may also lie in a few places only: then
      // the positions, not the pieces, are shared out among the CTAs, which costs two more trips to find the piece of a position
      // and its runs.
      const uint32_t n_send = min(found, J.kk);
      const uint32_t lo = (uint32_t)((uint64_t)n_send * J.pc.index / J.pc.count);
      const uint32_t hi = (uint32_t)((uint64_t)n_send * (J.pc.index + 1u) / J.pc.count);
      if (may && even) {
        if (ahead < n_send) send_range<kBlock, FRESH>(A, J, S, area, ahead, 0u, min(total, n_send - ahead));
      } else if (may && lo < hi) {
        uint32_t piece = 0, base = 0;
        {
          uint32_t carry = 0;
          for (uint32_t t0 = 0; t0 < J.pc.count && carry <= lo; t0 += kEmitThreads) {
            const uint32_t t = t0 + tid;
            const uint32_t v = t < J.pc.count ? (uint32_t)A.piece_cnt[J.pc.first + t] : 0u;
            uint32_t sum;
            const uint32_t at = carry + block_excl_scan(v, S.tmp, sum);
            if (at <= lo && lo < at + v) { S.at[0] = t; S.at[1] = at; }
            carry += sum;
          }
          __syncthreads();
          piece = S.at[0];
          base = S.at[1];
        }
        for (;;) {
          {
            const uint32_t n_runs = (min(J.piece_elems, J.sd.n_pad - piece * J.piece_elems) + kRunElems - 1u) / kRunElems;
            const uint32_t v = tid < n_runs ? A.run_cnt[((J.pc.first + piece) << A.piece_shift) + tid] & 0xffffu : 0u;
            ex = block_excl_scan(v, S.tmp, total);
            if (tid <= kMaxPieceRuns) S.pre[tid] = ex;
            __syncthreads();
          }
          const uint2* const lists = A.cand + (kBlock ? J.sd.off >> 4 : J.sd.off) + (size_t)piece * (kArea << A.piece_shift);
          send_range<kBlock, FRESH>(A, J, S, lists, base, lo > base ? lo - base : 0u, min(hi - base, total));
          base += total;
          ++piece;
          if (base >= hi || piece >= J.pc.count) break;
          __syncthreads();     // S.pre is rewritten
        }
      }
      if (!kBlock && short_of && may) {
        // pad the fixed-size stream, every CTA its share
#pragma unroll 1
        for (uint32_t p = found + J.pc.index * kEmitThreads + tid; p < J.sd.k; p += J.pc.count * kEmitThreads)
          emit_entry(A, J.dest, J.nb, J.slot_off, p, kSentinelIdx, 0.f);
      }
      if (last_of_tensor(J, S)) {
        uint32_t t_key = 0;
        if (kBlock && short_of && may) {
          const uint32_t need = J.kk - found;
          const uint32_t c = !rescan ? c_near : J.pc.count == 1u ? collected : __ldcg(&J.wp->cand_cnt);
          const uint32_t take = min(need, c);
          if (take && c <= kPickMax) {
            // none reaches the threshold, and the best lie in the two octaves under it
            const uint32_t top = ss.inited ? max(__float_as_uint(ss.tau), 1u) - 1u : 0x7fffffffu;
            t_key = pick_few(A, nears, c, take, top, ss.inited ? kTwoOctaves : 31u, J.sd.off >> 4, J.sd.n_pad >> 4, S);
#pragma unroll 1
            for (uint32_t e = tid; t_key != kNoCut && e < take * 16u; e += kEmitThreads) {
              const uint32_t q = e >> 4, p = (found + q) * 16u + (e & 15u);
              if (p < J.sd.k) {   // only the lowest-ranked block can be cut off
                const uint32_t gi = S.stage[S.hist[q]].x * 16u + (e & 15u);
                emit_and_keep<FRESH>(A, S, p, gi, resid1<FRESH>(A, gi));
              }
            }
          } else if (take) {
            t_key = send_best<true, FRESH>(A, J, S, nears, c, take, found, A.cand + (J.sd.off >> 4));
          }
          // fewer blocks with anything in them than the budget: the rest of the stream says "no entry"
#pragma unroll 1
          for (uint32_t p = (found + take) * 16u + tid; p < J.sd.k; p += kEmitThreads)
            emit_entry(A, J.dest, J.nb, J.slot_off, p, kSentinelIdx, 0.f);
        }
        __syncthreads();
        if (tid == 0 && ok) {
          SegState st = ss;
          if (!kBlock) {
            const float max_abs = __uint_as_float(__ldcg(&J.wp->max_bits));
            if (st.inited) {   // AIMD of thresholdv.cpp:70-76
              if (J.sd.k > found) st.tau *= 0.99f;
              else if (J.sd.k < found) st.tau = st.tau + 0.01f * ((float)found / (float)J.sd.k) * max_abs;
            }
          } else if (!st.inited) {
            if (short_of && may && t_key != kNoCut) {   // first threshold: the smallest selected key plus the first additive step
              const float t0 = __uint_as_float(t_key);
              st.tau_inc = 0.01f * t0;
              st.tau = t0 + st.tau_inc;
              st.inited = 1;
            }
          } else {
            if (short_of) st.tau *= 0.99f;      // "must drop less" (thresholdv16.cpp:245-248)
            else st.tau += st.tau_inc;          // thresholdv16.cpp:249-252
            // Keep a sixteenth to a quarter of the budget in near-miss blocks, and at least twice what this fill took:
            // the additive and multiplicative steps of the threshold move the count of blocks over it by a few per
            // cent, which is all a fill ever needs, and ranking the candidates costs time in proportion to their number.
            float w = window_or(st.reserved[0], kWindowDefault);
            const uint32_t needed = short_of ? J.kk - found : 0u;
            if (rescan) w *= 2.f;
            else if (c_near < J.kk / 16u + 8u || c_near < 2u * needed) w *= 1.5f;
            else if (c_near > J.kk / 4u + 32u) w *= 0.75f;
            st.reserved[0] = __float_as_uint(fminf(fmaxf(w, 1e-3f), 1.f));
          }
          A.state[J.pc.seg] = st;
        }
        if (tid == 0) { J.wp->cand_cnt = 0u; J.wp->out_cursor = 0u; J.wp->max_bits = 0u; }
        for (uint32_t t = tid; t < J.pc.count; t += kEmitThreads) A.piece_cnt[J.pc.first + t] = 0ull;
      }
    }
  }

  __syncthreads();
  next_may_begin();
  if (tid == 0) finish_select(A, J.epoch, MODE == kScanTop ? A.refills : nullptr);
}

// Top-k tensors whose candidates fell short: the exact selection from the residual, with the histogram that `emit` took.
template <bool FRESH>
__global__ void __launch_bounds__(kEmitThreads, 2) k_refill(const __grid_constant__ SelectArgs A) {
  __shared__ EmitShared S;
  behind_previous();
  if (ld_volatile_u32(A.refills) == 0u) return;     // the same for every CTA: it is cleared behind the last one
  const uint32_t tid = threadIdx.x;
  const Job J = job_of(A, false);
  const bool ok = ld_volatile_u32(A.status) == kOk;
  if (!(J.sd.reserved & kSegSkip) && J.wp->refill != 0u) {
    if (tid == 0) S.word[0] = ok && acks_arrived(A, J.epoch) ? 1u : 0u;
    note_destinations(A, J, S);
    const SegState ss = A.state[J.pc.seg];
    const uint32_t cut = top_cut(ss, J.sd.n_pad), found = J.wp->found;      // found < kk items reach the cut
    uint32_t* gh = A.hist_rest + (size_t)J.pc.seg * kHistBins;
    plan_top(gh, 1u, J.sd.n_pad - found, J.kk - found, true, S);
    const bool may = S.word[0] != 0u, zero_fill = S.res[0] == 0u;
    uint32_t key_lo, key_hi, emitted = 0, noted = 0;
    rest_bin_range(S.res[0], cut, key_lo, key_hi);
    const uint32_t rem = S.res[1];
    uint2* const undecided = A.cand + A.n_total + J.sd.off;
    const uint32_t len = J.len;
    if (may && zero_fill) {
      // fewer non-zero elements than the budget: zeros complete it, lowest index first; `emit` left their number per piece.
      // This comes first, because what is sent below becomes zero in the residual.
      uint32_t before = 0, base;
      for (uint32_t t = tid; t < J.pc.index; t += kEmitThreads) before += A.run_cnt[(J.pc.first + t) << A.piece_shift];
      block_excl_scan(before, S.tmp, base);
      for (uint32_t i0 = 0; i0 < len && base < rem; i0 += kEmitThreads * 4u) {
        const uint32_t i = i0 + tid * 4u;
        const bool act = i < len;
        const float4 a = act ? resid4<FRESH>(A, J.pc.start + i, load4<FRESH>(A, J.pc.start + i)) : make_float4(1.f, 1.f, 1.f, 1.f);
        const uint32_t at = J.pc.start + i, idx[4] = {at, at + 1u, at + 2u, at + 3u};
        const uint32_t bits[4] = {__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z), __float_as_uint(a.w)};
        uint32_t zero = 0, total;
#pragma unroll
        for (int e = 0; e < 4; ++e) zero |= (uint32_t)((bits[e] & 0x7fffffffu) == 0u) << e;
        const uint32_t ex = block_excl_scan(__popc(zero), S.tmp, total);
        while (zero && base + ex + __popc(zero) > rem) zero &= ~(0x80000000u >> __clz(zero));      // the budget ends here
        send_marked<FRESH, 4>(A, S, idx, bits, zero, ex, min(total, rem - base), J.kk - rem + base);
        base += total;
      }
    }
    if (may) {
      constexpr int kItems = 16;
      for (uint32_t i0 = 0; i0 < len; i0 += kEmitThreads * kItems) {
        uint32_t idx[kItems], bits[kItems];
        float4 raw[kItems / 4];
#pragma unroll
        for (int u = 0; u < kItems / 4; ++u) {
          const uint32_t i = i0 + (u * kEmitThreads + tid) * 4u;
          raw[u] = i < len ? load4<FRESH>(A, J.pc.start + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kItems / 4; ++u) {
          const uint32_t i = i0 + (u * kEmitThreads + tid) * 4u;
          const bool act = i < len;
          const float4 a = resid4<FRESH>(A, J.pc.start + i, raw[u]);
          const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            bits[4 * u + e] = __float_as_uint(v[e]);
            idx[4 * u + e] = act && (bits[4 * u + e] & 0x7fffffffu) ? J.pc.start + i + e : kSentinelIdx;
          }
        }
        emit_top_batch<FRESH, kItems>(A, J, S, undecided, idx, bits, key_lo, key_hi, emitted, noted);
      }
    }
    if (last_of_tensor(J, S)) {
      const uint32_t c = J.pc.count == 1u ? noted : __ldcg(&J.wp->cand_cnt);
      if (may && rem != 0u && (zero_fill || rem <= c)) {
        const uint32_t t_key = zero_fill ? 0u : settle_top<FRESH>(A, J, S, undecided, c, rem, key_lo, key_hi);
        if (tid == 0 && t_key != kNoCut) step_top(A, J, ss, t_key, 0u);
      } else if (may && tid == 0) {
        set_status(A.status, kBadCandidate);
      }
      __syncthreads();
      if (tid == 0) { J.wp->out_cursor = 0u; J.wp->cand_cnt = 0u; J.wp->refill = 0u; J.wp->found = 0u; }
      for (uint32_t b = tid; b < (uint32_t)kHistBins; b += kEmitThreads) gh[b] = 0u;
    }
  }
  __syncthreads();
  if (tid == 0) finish_select(A, J.epoch, A.refills, true);
}

// ------------------------------------------------------------------------------------------------
// host launchers
// ------------------------------------------------------------------------------------------------
bool one_pass_possible(const SelectArgs& A) {
  // list positions and counts are 32-bit; behind the lists, of one slot per item, lie as many slots for top-k's undecided
  // items and for the candidates of threshold-v16's fill
  const uint64_t slots = A.compressor == kTopk ? 2ull * A.n_total : A.compressor == kThresholdv16 ? A.n_total / 8u : A.n_total;
  return A.compressor != kRandomk && A.pieces != nullptr && A.n_total < (1u << 30) && A.cand_cap >= slots;
}

cudaError_t launch_select_one_pass(const SelectArgs& A, cudaStream_t stream, cudaEvent_t before_emit) {
  if (A.n_chunks == 0 || A.n_segs == 0) return cudaSuccess;
  if (A.world > kMaxWorld || !one_pass_possible(A) || (1u << A.piece_shift) > kMaxPieceRuns) return cudaErrorInvalidValue;
  using Kernel = void (*)(SelectArgs);
  const Kernel scan[2][3] = {{k_scan<kScanTop, false>, k_scan<kScanElem, false>, k_scan<kScanBlock, false>},
                             {k_scan<kScanTop, true>, k_scan<kScanElem, true>, k_scan<kScanBlock, true>}};
  const Kernel emit[2][3] = {{k_emit<kScanTop, false>, k_emit<kScanElem, false>, k_emit<kScanBlock, false>},
                             {k_emit<kScanTop, true>, k_emit<kScanElem, true>, k_emit<kScanBlock, true>}};
  const int fresh = A.fresh ? 1 : 0, mode = A.compressor == kThresholdv16 ? kScanBlock : A.compressor == kThresholdv ? kScanElem : kScanTop;
  cudaError_t e = launch_streaming(scan[fresh][mode], A.n_chunks, kScanThreads, stream, A);
  if (e == cudaSuccess && before_emit != nullptr) e = cudaStreamWaitEvent(stream, before_emit, 0);
  if (e != cudaSuccess) return e;
  // With peers every CTA of the emission ends in a system-wide fence; begun beside the scan it took 40 us on one of two boxes, 23
  // behind it (64 MB bucket, eight destinations; 20 since entries are read once for all of them).
  e = before_emit == nullptr && !A.publish ? launch_behind(emit[fresh][mode], A.n_pieces, kEmitThreads, stream, A)
                                           : launch_first(emit[fresh][mode], A.n_pieces, kEmitThreads, stream, A);
  if (e == cudaSuccess && A.compressor == kTopk)
    e = launch_behind(A.fresh ? k_refill<true> : k_refill<false>, A.n_pieces, kEmitThreads, stream, A);
  return e;
}

}  // namespace st
