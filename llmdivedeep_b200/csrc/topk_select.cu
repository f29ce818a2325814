// Per-row top-k by radix select (sm_100a).  Stands in for the torch.topk calls at
// sparse_attn/DSA.py:361, 567 and 675-676 of the reference.
//
// One CTA per row.  fp32 values are mapped to order-preserving 32-bit keys.  Three ways to the same set (ties: lower column):
//   * direct (rows of at most 8188 columns): the row stays in registers.  One histogram of 2048 equal bins over its range of
//     VALUES -- they spread, where the leading bits of the keys pile up on a few exponents -- gives the bin of the k-th value;
//     what lies above it leaves in column order, the bin's own few elements are ranked against one another.
//   * sampled (longer rows): a sample of the row (one 128-float block in every 16, more of a row below 32768 columns) is ranked by the
//     same kind of histogram, a threshold a few standard deviations below the sample's estimate of the k-th value is taken
//     from it, one ordered pass stages every element at or above it (at most 4096) and counts it by bins as it does, and the
//     select reads the candidates once.  Values far from the others, which would leave a histogram of equal bins
//     blind, cost a second look at the sample and no more: the rank's bin is cut into bins in turn, and the candidates are binned
//     by their keys.
//   * two passes, for what the others give up (a staged count that misses [k, 4096], infinities or NaN in the range, more than 256
//     elements in the threshold bin, long unaligned rows): the k-th key digit by digit (12 + 12 + 8 bits):
//       1. histogram the top 12 key bits of the row (shared-memory atomics), suffix-
//          scan the bins to find the bin holding the k-th largest element;
//       2. if that bin holds more than 2048 elements, repeat on the next digit over
//          the row (only rows with tightly clustered values need this);
//       3. one ordered pass over the row writes every element above the threshold
//          bin straight to the output and stages the threshold bin's elements
//          ("candidates") in shared memory, in column order;
//       4. the remaining digits are resolved on the staged candidates, and a final
//          ordered compaction emits candidates above the exact k-th key plus the
//          first `need` candidates equal to it.
// Compaction uses block prefix sums, never atomics, and no order depends on the number of threads, so a row's output is
// the same from run to run and whatever the number of rows of the call.
// What bounds it: latency, of the barriers between a row's steps.  us, against the form before (digit passes behind the sample, two
// passes below 16384 columns), k = 2048: 7 rows of up to 33000 columns 13.5 -> 8.7, 64 x 131072 21.2 -> 12.3, 160 x 9000 15.0 -> 10.4, 2048 x 16384
// causal 104 -> 71, 4096 x 32768 213 -> 166, 4096 x 131072 453 -> 383, 3000 x 3000 30 -> 19; 2048 x 2048, k = 256 42 -> 21.
// With 64 values of a row at 300 sigma (before; equal bins alone, which give up and pay for two passes as well; now): 64 x 131072 23.2, 56.2,
// 16.2, 7 x 33000 15.8, 22.7, 10.3, 1024 x 32768 68, 126, 53, 160 x 9000 15.7, 21.8, 14.0; rows in registers, 1024 x 3000 27.8, 49.9, 32.1, 1024 x
// 8000 35.5, 44.4, 45.6.  Rows in registers have no second look: bins of the bin, from the registers, made ordinary rows 10 % slower.
#include <math_constants.h>

#include <cstdlib>

#include "dsa_common.cuh"
#include "dsa_host.h"

namespace dsa {

constexpr int kDigitBits = 12;
constexpr int kBins = 1 << kDigitBits;                 // digit passes
constexpr int kLinBins = 2048;                         // one-pass histograms over a range of values
constexpr int kCand = 2048;                            // two-pass path: largest threshold bin staged
constexpr int kCandS = 4096;                           // candidates that the sampled path may stage
constexpr int kDirectChunk = 4096;
constexpr int kDirectRow = 2 * kDirectChunk - 4;       // longest row without sample and staging (it may start three columns into a float4)
constexpr int kTieCap = 256;                           // elements of the threshold bin that are ranked by counting
constexpr int kMaxLevels = 3;                          // a crowded bin of the sample is cut into bins at most that often
constexpr int kSampleBlock = 128;                      // floats per sampled block (one float4 per lane)
constexpr int kSampleMaxBlocks = 64;                   // at most 8192 sampled values
constexpr int kSampleWant = 16;                        // blocks wanted where a block in 16 gives fewer
constexpr int kRun = 32;                               // sampled path: columns per thread per chunk
constexpr int kVec = 4;
constexpr int kEltPerThread = 16;                      // two-pass path, final pass: 4 x float4, contiguous

__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return u ^ (static_cast<uint32_t>(static_cast<int32_t>(u) >> 31) | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float(key ^ (static_cast<uint32_t>(static_cast<int32_t>(~key) >> 31) | 0x80000000u));
}

// A range of values cut into kLinBins equal bins, counted from the top.  (hi - x) and its product with a positive factor are
// monotone in floating point, so the bins order elements as their keys do; what lies above hi falls into bin 0, what lies below
// the range into the last.  A NaN with the sign bit clear has the largest key and falls into bin 0, one with the sign bit set
// must not come here.
struct LinBins {
  float hi, scale;
  uint32_t base = 0;                                    // not 0: the elements' coordinate is how far their key lies above this one
  __device__ __forceinline__ int of_key(uint32_t key) const { return of(base ? __uint2float_rz(key - base) : key_value(key)); }
  __device__ __forceinline__ bool set(float top, float bottom) {       // false: no usable range (all equal, infinite, NaN)
    hi = top;
    scale = static_cast<float>(kLinBins) / (top - bottom);
    return top > bottom && scale > 0.f && scale < CUDART_INF_F;
  }
  __device__ __forceinline__ int of(float x) const { return max(0, min(kLinBins - 1, __float2int_rz((hi - x) * scale))); }
};

// hist and cand_key share storage: candidate keys are copied to registers (followed by a block
// barrier) before the histogram is next cleared, and the histogram is dead while candidates are staged.
struct alignas(16) TopkSmem {
  union {
    uint32_t hist[kBins];
    uint32_t cand_key[kCandS];
  };
  int32_t cand_idx[kCandS];
  union {
    uint32_t lin[kLinBins];
    struct { uint32_t key[kTieCap]; int32_t col[kTieCap]; } tie;       // the threshold bin's elements
  };
  uint32_t warp_tot[2][32];
  uint32_t bin, need, cnt;
};
static_assert(kBins == kCandS, "hist and cand_key are one array");

template <int TH, int BINS>
__device__ __forceinline__ void zero_bins(uint32_t* hist) {
  uint4* h4 = reinterpret_cast<uint4*>(hist);
#pragma unroll
  for (int b = threadIdx.x; b < BINS / 4; b += TH) h4[b] = make_uint4(0u, 0u, 0u, 0u);
}

// Block-wide: given hist[], find the bin b with  sum(hist[b+1..]) < need <= sum(hist[b..]), or with FROM_TOP counting from bin 0:
// sum(hist[..b-1]) < need <= sum(hist[..b]).  Leaves bin / need (remaining within the bin) / cnt (= hist[b]) in shared memory.
template <int TH, int BINS, bool FROM_TOP>
__device__ __forceinline__ void find_threshold_bin(TopkSmem& sm, const uint32_t* hist, uint32_t need) {
  constexpr int PER = BINS / TH;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = (FROM_TOP ? tid : TH - 1 - tid) * PER;  // threads in the order of the count
  uint32_t h[PER];
  uint32_t mine = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    h[j] = hist[FROM_TOP ? b0 + j : b0 + PER - 1 - j];
    mine += h[j];
  }
  uint32_t v = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t nb = __shfl_up_sync(0xffffffffu, v, off);
    if (lane >= off) v += nb;
  }
  if (lane == 31) sm.warp_tot[0][warp] = v;
  __syncthreads();
  uint32_t wt = lane < warp ? sm.warp_tot[0][lane] : 0u;               // warps before this one
  wt = __reduce_add_sync(0xffffffffu, wt);
  const uint32_t incl = v + wt;
  uint32_t cum = incl - mine;
  if (cum < need && need <= incl) {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (cum < need && cum + h[j] >= need) {
        sm.bin = FROM_TOP ? b0 + j : b0 + PER - 1 - j;
        sm.need = need - cum;
        sm.cnt = h[j];
      }
      cum += h[j];
    }
  }
  __syncthreads();
}

// Exclusive block prefix of a packed (lo16, hi16) counter pair; also returns the block total.
// `buf` alternates between calls so one __syncthreads per call is enough.
template <int TH>
__device__ __forceinline__ uint32_t block_exclusive_scan(TopkSmem& sm, uint32_t packed, int buf, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = packed;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t nb = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += nb;
  }
  if (lane == 31) sm.warp_tot[buf][warp] = incl;
  __syncthreads();
  const uint32_t wt = lane < TH / 32 ? sm.warp_tot[buf][lane] : 0u;
  total = __reduce_add_sync(0xffffffffu, wt);          // the halves do not carry into each other: counts stay below 2^16
  return incl - packed + __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
}

// Digit passes over keys held in registers (bit j of `valid` says whether ck[j] counts): refines
// (prefix, pbits, need) 12 bits at a time until `stop_bits` key bits are decided.  Ends on a block barrier.
template <int TH, int NPT>
__device__ __forceinline__ void digit_passes(TopkSmem& sm, const uint32_t (&ck)[NPT], uint32_t valid, uint32_t& prefix,
                                             int& pbits, uint32_t& need, int stop_bits) {
  while (pbits < stop_bits) {
    const int dbits = min(kDigitBits, 32 - pbits);
    const int shift = 32 - pbits - dbits;
    const uint32_t dmask = (1u << dbits) - 1u;
    zero_bins<TH, kBins>(sm.hist);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
      const bool match = pbits == 0 || (ck[j] >> (32 - pbits)) == prefix;
      if (((valid >> j) & 1u) && match) atomicAdd(&sm.hist[(ck[j] >> shift) & dmask], 1u);
    }
    __syncthreads();
    find_threshold_bin<TH, kBins, false>(sm, sm.hist, need);
    prefix = (pbits == 0 ? 0u : (prefix << dbits)) | sm.bin;
    need = sm.need;
    pbits += dbits;
    __syncthreads();
  }
}

// Ordered emission of staged candidates (thread t holds candidates [t*NPT, t*NPT+NPT) in column order):
// those above the exact k-th key `kth` go to o[n_above...], the first `need` equal to it fill the tail.
template <int TH, int NPT>
__device__ __forceinline__ void emit_candidates(TopkSmem& sm, const uint32_t (&ck)[NPT], uint32_t valid, uint32_t kth,
                                                uint32_t need, uint32_t n_above, int k, int32_t* __restrict__ o) {
  const int tid = threadIdx.x;
  uint32_t fgt = 0, feq = 0;
#pragma unroll
  for (int j = 0; j < NPT; ++j) {
    if ((valid >> j) & 1u) {
      fgt |= (uint32_t)(ck[j] > kth) << j;
      feq |= (uint32_t)(ck[j] == kth) << j;
    }
  }
  uint32_t total;
  const uint32_t excl = block_exclusive_scan<TH>(sm, __popc(fgt) | (__popc(feq) << 16), 0, total);
  uint32_t pg = n_above + (excl & 0xffffu);
  uint32_t pe = excl >> 16;
#pragma unroll
  for (int j = 0; j < NPT; ++j) {
    const uint32_t a = tid * NPT + j;
    if (fgt & (1u << j)) {
      o[pg++] = sm.cand_idx[a];
    } else if (feq & (1u << j)) {
      if (pe < need) o[k - need + pe] = sm.cand_idx[a];
      ++pe;
    }
  }
}

// Staging test of the sampled pass on the raw float bits u, exact for every bit pattern:
// key(u) >= thr.  tfb holds the float bits whose key is thr.  For a threshold that is a non-negative
// float a signed compare does it (negative floats are negative integers, a positive NaN is the largest);
// for a negative threshold an unsigned one does (every non-negative float lies below the sign bit).
template <bool NEG>
__device__ __forceinline__ bool at_or_above(float v, uint32_t tfb) {
  const uint32_t u = __float_as_uint(v);
  return NEG ? (u <= tfb) : (static_cast<int32_t>(u) >= static_cast<int32_t>(tfb));
}

// One chunk (32 columns a thread) of the sampled pass: warp w owns columns [w*1024, w*1024+1024) of the chunk and
// reads them as 8 coalesced float4 rows.  Returns the hit flags of this lane, bit q*4+e for column
// wbase + q*128 + lane*4 + e.
template <bool NEG>
__device__ __forceinline__ uint32_t chunk_flags(const float* x, int wbase, int lane, int lo, int hi,
                                                uint32_t tfb) {
  uint32_t fc = 0;
  if (wbase >= lo && wbase + kRun * 32 <= hi) {
#pragma unroll
    for (int q = 0; q < kRun / kVec; ++q) {
      const float4 f = *reinterpret_cast<const float4*>(x + wbase + q * 128 + lane * kVec);
      if (at_or_above<NEG>(f.x, tfb)) fc |= 1u << (q * 4 + 0);
      if (at_or_above<NEG>(f.y, tfb)) fc |= 1u << (q * 4 + 1);
      if (at_or_above<NEG>(f.z, tfb)) fc |= 1u << (q * 4 + 2);
      if (at_or_above<NEG>(f.w, tfb)) fc |= 1u << (q * 4 + 3);
    }
  } else if (wbase < hi && wbase + kRun * 32 > lo) {
    for (int q = 0; q < kRun / kVec; ++q) {
      const int i = wbase + q * 128 + lane * kVec;
      if (i < hi && i + kVec > lo) {         // a float4 that starts below hi lies inside the row's allocation
        const float4 f = *reinterpret_cast<const float4*>(x + i);
        const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int e2 = 0; e2 < kVec; ++e2)
          if (i + e2 >= lo && i + e2 < hi && at_or_above<NEG>(v[e2], tfb)) fc |= 1u << (q * 4 + e2);
      }
    }
  }
  return fc;
}

// Stages a lane's hits of a chunk: their columns first, then their values, by the lanes of the warp alike and while the L1 still has
// them.  (All values at the end of the row, by all threads: 4096 x 131072 478 us instead of 383, the rows in flight do not fit the L2.  A
// lane's own values in its own loop: 406, and 64 x 131072 13.1 instead of 12.4, or 17.7 where the compiler lets the lanes drift apart.)
__device__ __forceinline__ void stage_hits(TopkSmem& sm, const float* x, int wbase, int lane, uint32_t fc, uint32_t pc,
                                           const LinBins& bins) {
  const uint32_t begin = __shfl_sync(0xffffffffu, pc, 0);
  while (fc) {                               // few bits set
    const int j = __ffs(fc) - 1;
    fc &= fc - 1;
    sm.cand_idx[pc++] = wbase + (j >> 2) * 128 + lane * kVec + (j & 3);
  }
  const uint32_t end = __shfl_sync(0xffffffffu, pc, 31);
  __syncwarp();
  // the warp's hits, dealt to its lanes: read again (from the L1) rather than kept
  for (uint32_t a = begin + lane; a < end; a += 32) {
    const uint32_t key = order_key(x[sm.cand_idx[a]]);
    sm.cand_key[a] = key;
    atomicAdd(&sm.lin[bins.of_key(key)], 1u);
  }
  __syncwarp();
}

// The ordered pass of the sampled path: stages every element with key >= thr, two chunks per block scan, and counts them by
// bins.  Candidates end up in a fixed order (1024 columns, lane, column) that does not depend on timing or on TH.
// Returns the staged count, or 0xffffffff once it would exceed the capacity (uniform over the block).
template <int TH, bool NEG>
__device__ __forceinline__ uint32_t stage_row(TopkSmem& sm, const float* x, int lo, int hi, uint32_t tfb,
                                              const LinBins& bins) {
  constexpr int CHUNK = TH * kRun;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int base = lo & ~(kVec - 1);
  const int n_pairs = (hi - base + 2 * CHUNK - 1) / (2 * CHUNK);
  uint32_t staged = 0;
  for (int c = 0; c < n_pairs; ++c) {
    const int wb0 = base + (2 * c) * CHUNK + warp * (kRun * 32);
    const int wb1 = wb0 + CHUNK;
    const uint32_t f0 = chunk_flags<NEG>(x, wb0, lane, lo, hi, tfb);
    const uint32_t f1 = chunk_flags<NEG>(x, wb1, lane, lo, hi, tfb);
    uint32_t total;
    const uint32_t excl = block_exclusive_scan<TH>(sm, __popc(f0) | (__popc(f1) << 16), c & 1, total);
    const uint32_t t0 = total & 0xffffu, t1 = total >> 16;
    if (staged + t0 + t1 > (uint32_t)kCandS) return 0xffffffffu;   // every thread sees the same totals
    stage_hits(sm, x, wb0, lane, f0, staged + (excl & 0xffffu), bins);
    stage_hits(sm, x, wb1, lane, f1, staged + t0 + (excl >> 16), bins);
    staged += t0 + t1;
  }
  __syncthreads();
  return staged;
}

// Block-wide largest and smallest key (threads without one give 0 and 0xffffffff); clears sm.lin on the way, which is clear and may
// be counted into when this returns.
template <int TH>
__device__ __forceinline__ void key_range(TopkSmem& sm, uint32_t& kmax, uint32_t& kmin) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  if (lane == 0) {
    sm.warp_tot[0][warp] = kmax;
    sm.warp_tot[1][warp] = kmin;
  }
  zero_bins<TH, kLinBins>(sm.lin);
  __syncthreads();
  kmax = __reduce_max_sync(0xffffffffu, lane < TH / 32 ? sm.warp_tot[0][lane] : 0u);
  kmin = __reduce_min_sync(0xffffffffu, lane < TH / 32 ? sm.warp_tot[1][lane] : 0xffffffffu);
}

// The k largest of a set of elements that sm.lin counts by `bins` (complete, a barrier behind it), in CHUNKS chunks: each(c, ck,
// col) gives thread t's elements of a chunk (keys and columns; returns which of them count), in a fixed order over chunks,
// threads and elements.  One look for the threshold bin; what lies above it leaves in that order, the bin's own few elements are
// ranked against one another (ties: lower column first).  Returns false, for all threads alike and with nothing written, when
// the bin holds too many.
template <int TH, int NPT, int CHUNKS, typename Each>
__device__ __forceinline__ bool select_by_bins(TopkSmem& sm, const LinBins& bins, int k, int32_t* __restrict__ o, const Each& each) {
  find_threshold_bin<TH, kLinBins, true>(sm, sm.lin, (uint32_t)k);
  const int b = sm.bin;
  const uint32_t need = sm.need, cnt = sm.cnt, n_above = k - need;
  if (cnt > (uint32_t)kTieCap) return false;
  uint32_t pg = 0, pe = 0;                                // emitted and ranked elements of the chunks before
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    uint32_t ck[NPT];
    int32_t col[NPT];
    const uint32_t valid = each(c, ck, col);
    uint32_t fgt = 0, feq = 0;
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
      if ((valid >> j) & 1u) {
        const int bj = bins.of_key(ck[j]);
        fgt |= (uint32_t)(bj < b) << j;
        feq |= (uint32_t)(bj == b) << j;
      }
    }
    uint32_t total;
    const uint32_t excl = block_exclusive_scan<TH>(sm, __popc(fgt) | (__popc(feq) << 16), (c & 1) ^ 1, total);
    uint32_t p = pg + (excl & 0xffffu), q = pe + (excl >> 16);
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
      if (fgt & (1u << j)) o[p++] = col[j];
      if (feq & (1u << j)) {
        sm.tie.key[q] = ck[j];
        sm.tie.col[q++] = col[j];
      }
    }
    pg += total & 0xffffu;
    pe += total >> 16;
  }
  __syncthreads();
  if (threadIdx.x < cnt) {
    const uint32_t key = sm.tie.key[threadIdx.x];
    const int32_t c = sm.tie.col[threadIdx.x];
    uint32_t rank = 0;
    // Four at a time: one by one, a bin of 200 elements took 14 us, longer than all the rest of a row of 3000 columns.
#pragma unroll 2
    for (uint32_t i = 0; i < cnt; i += 4) {
      const uint4 ki = *reinterpret_cast<const uint4*>(&sm.tie.key[i]);
      const int4 ci = *reinterpret_cast<const int4*>(&sm.tie.col[i]);
      rank += ki.x > key || (ki.x == key && ci.x < c);
      rank += i + 1 < cnt && (ki.y > key || (ki.y == key && ci.y < c));
      rank += i + 2 < cnt && (ki.z > key || (ki.z == key && ci.z < c));
      rank += i + 3 < cnt && (ki.w > key || (ki.w == key && ci.w < c));
    }
    if (rank < need) o[n_above + rank] = c;
  }
  return true;
}

// The threshold of the sampled pass: a value a few standard deviations below the sample's estimate of the k-th, and the bins
// that its candidates are counted by.  Returns false (for every thread of the block alike) when the row rules the sampled pass
// out.  The result depends on the row alone, not on TH.  Leaves sm.lin zeroed (a barrier has to follow).
template <int TH>
__device__ __forceinline__ bool sample_threshold(TopkSmem& sm, const float* x, int lo, int hi, int k,
                                                 float& thr_out, LinBins& bins_out) {
  constexpr int NPT = kSampleMaxBlocks / (TH / 32) * 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = hi - lo;
  const int first = (lo + kVec - 1) & ~(kVec - 1);
  const int nblk = (hi - first) / kSampleBlock;
  // one block sampled in every sb: one in 16, fewer of a very long row, more of a short one
  const int sb = max(min(16, nblk / kSampleWant), (nblk + kSampleMaxBlocks - 1) / kSampleMaxBlocks);
  const int mblk = sb > 0 ? nblk / sb : 0;
  const int m = mblk * kSampleBlock;
  const float frac = (float)m / (float)n;
  const float mu = (float)k * frac;                       // top-k elements expected inside the sample
  const float rf = ceilf(mu + 4.f * sqrtf(mu) + 2.f);     // rank taken: about 4 sigma below the k-th value
  if (m < 1024 || rf > (float)m || rf > 0.8f * (float)kCandS * frac) return false;

  uint32_t skey[NPT];
  uint32_t svalid = 0, kmax = 0, kmin = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < NPT / 4; ++i) {
    const int j = warp + TH / 32 * i;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool in = j < mblk;
    if (in) {
      f = *reinterpret_cast<const float4*>(x + first + (j * sb + sb / 2) * kSampleBlock + lane * kVec);
      svalid |= 0xFu << (4 * i);
    }
    skey[4 * i + 0] = order_key(f.x); skey[4 * i + 1] = order_key(f.y);
    skey[4 * i + 2] = order_key(f.z); skey[4 * i + 3] = order_key(f.w);
    if (in) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        kmax = max(kmax, skey[4 * i + e]);
        kmin = min(kmin, skey[4 * i + e]);
      }
    }
  }
  key_range<TH>(sm, kmax, kmin);
  const float top = key_value(kmax);
  LinBins bins;
  if (!bins.set(top, key_value(kmin))) return false;      // a NaN makes it false too, whatever its sign
#pragma unroll
  for (int j = 0; j < NPT; ++j)
    if ((svalid >> j) & 1u) atomicAdd(&sm.lin[bins.of(key_value(skey[j]))], 1u);
  __syncthreads();
  find_threshold_bin<TH, kLinBins, true>(sm, sm.lin, (uint32_t)rf);
  // the bin's lower edge, give or take a rounding
  float thr = top - (float)(sm.bin + 1) * ((top - key_value(kmin)) * (1.f / kLinBins));
  const uint32_t enough = max(4, (int)rf / 16);
  if (sm.cnt > enough) {
    // Too many in the bin to tell the rank by: a few values far from the others have stretched the range.  The bin's own range
    // is cut into bins in turn (the sample is read again, so that other rows do not keep it in registers).
#pragma unroll 1
    for (int level = 0; level < kMaxLevels && sm.cnt > enough; ++level) {
      const int b = sm.bin;
      const uint32_t need = sm.need, hi_key = kmax, lo_key = kmin;
      kmax = 0;
      kmin = 0xffffffffu;
#pragma unroll 1
      for (int i = tid; i < m; i += TH) {
        const uint32_t key = order_key(x[first + (i / kSampleBlock * sb + sb / 2) * kSampleBlock + i % kSampleBlock]);
        if (key >= lo_key && key <= hi_key && bins.of(key_value(key)) == b) {
          kmax = max(kmax, key);
          kmin = min(kmin, key);
        }
      }
      __syncwarp();
      key_range<TH>(sm, kmax, kmin);
      if (!bins.set(key_value(kmax), key_value(kmin))) {  // all equal, or as good as
        thr = key_value(kmin);
        __syncthreads();
        break;
      }
#pragma unroll 1
      for (int i = tid; i < m; i += TH) {
        const uint32_t key = order_key(x[first + (i / kSampleBlock * sb + sb / 2) * kSampleBlock + i % kSampleBlock]);
        if (key >= kmin && key <= kmax) atomicAdd(&sm.lin[bins.of(key_value(key))], 1u);
      }
      __syncthreads();
      find_threshold_bin<TH, kLinBins, true>(sm, sm.lin, need);
      thr = key_value(kmax) - (float)(sm.bin + 1) * ((key_value(kmax) - key_value(kmin)) * (1.f / kLinBins));
    }
    // as many equal values as that cannot be staged
    if ((float)((int)rf - (int)sm.need + (int)sm.cnt) > (float)kCandS * frac) return false;
  }
  zero_bins<TH, kLinBins>(sm.lin);                        // for the candidates (all have read the counts)
  thr_out = thr;
  // candidates of one sign are binned by their keys, near enough by their logarithms: no value stretches that range
  const uint32_t base = order_key(thr);
  if (thr > 0.f || top < 0.f) {
    bins_out.base = base;
    return bins_out.set(__uint2float_rz(order_key(top) - base), 0.f);
  }
  return bins_out.set(top, thr);
}

// One ordered pass over columns [lo, hi) of the row: stages everything whose key is at or above thr's.
// Returns the staged count, or 0xffffffff once it would exceed the capacity (uniform over the block).
template <int TH>
__device__ __forceinline__ uint32_t stage_above(TopkSmem& sm, const float* x, int lo, int hi, uint32_t thr,
                                                const LinBins& bins) {
  const bool neg = (thr & 0x80000000u) == 0u;             // the threshold is a negative float
  const uint32_t tfb = neg ? ~thr : (thr ^ 0x80000000u);  // its bits as a float
  return neg ? stage_row<TH, true>(sm, x, lo, hi, tfb, bins) : stage_row<TH, false>(sm, x, lo, hi, tfb, bins);
}

// Single pass over a long row, steered by a sample.  Returns false (for every thread of the block alike)
// when the row has to take the two-pass path: geometry out of range, or the staged count missed [k, 4096].
// Needs 16-byte aligned rows.
template <int TH>
__device__ __forceinline__ bool sampled_single_pass(TopkSmem& sm, const float* x, int lo, int hi, int k,
                                                    int32_t* __restrict__ o) {
  constexpr int NPT = kCandS / TH;
  float thr;
  LinBins bins;
  if (!sample_threshold<TH>(sm, x, lo, hi, k, thr, bins)) return false;
  const uint32_t staged = stage_above<TH>(sm, x, lo, hi, order_key(thr), bins);
  if (staged == 0xffffffffu || staged < (uint32_t)k) return false;   // missed [k, capacity]: two-pass path
  return select_by_bins<TH, NPT, 1>(sm, bins, k, o, [&](int, uint32_t(&ck)[NPT], int32_t(&col)[NPT]) {
    uint32_t valid = 0;
#pragma unroll
    for (int j = 0; j < NPT; j += 4) {
      const uint32_t a = threadIdx.x * NPT + j;
      const uint4 q = *reinterpret_cast<const uint4*>(&sm.cand_key[a]);
      const int4 c = *reinterpret_cast<const int4*>(&sm.cand_idx[a]);
      ck[j] = q.x; ck[j + 1] = q.y; ck[j + 2] = q.z; ck[j + 3] = q.w;
      col[j] = c.x; col[j + 1] = c.y; col[j + 2] = c.z; col[j + 3] = c.w;
#pragma unroll
      for (int e = 0; e < 4; ++e) valid |= (uint32_t)(a + e < staged) << (j + e);
    }
    return valid;
  });
}

// A row of at most CHUNKS x 4096 - 4 columns, without a sample or staging: it stays in registers, chunks of 4096 columns, thread
// order = column order.  Returns false, for all threads alike, when the values have no usable range (infinities, NaN, all equal)
// or the threshold bin holds too many: the two-pass path settles those.
template <int TH, int CHUNKS>
__device__ __forceinline__ bool direct_row(TopkSmem& sm, const float* x, bool vec, int lo, int hi, int k,
                                           int32_t* __restrict__ o) {
  constexpr int NPT = kDirectChunk / TH;
  const int tid = threadIdx.x;
  const int i0 = (lo & ~(kVec - 1)) + tid * NPT;
  auto used = [&](int c, int j) { return i0 + c * kDirectChunk + j >= lo && i0 + c * kDirectChunk + j < hi; };
  uint32_t key[CHUNKS][NPT], kmax = 0, kmin = 0xffffffffu;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const float* xc = x + c * kDirectChunk;
#pragma unroll
    for (int j = 0; j < NPT; j += kVec) {
      float v[kVec] = {0.f, 0.f, 0.f, 0.f};
      if (vec) {                                          // a float4 that starts below hi lies inside the row's allocation
        if (i0 + c * kDirectChunk + j < hi) {
          const float4 f = *reinterpret_cast<const float4*>(xc + i0 + j);
          v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < kVec; ++e)
          if (used(c, j + e)) v[e] = xc[i0 + j + e];
      }
#pragma unroll
      for (int e = 0; e < kVec; ++e) key[c][j + e] = order_key(v[e]);
    }
  }
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int j = 0; j < NPT; ++j)
      if (used(c, j)) {
        kmax = max(kmax, key[c][j]);
        kmin = min(kmin, key[c][j]);
      }
  key_range<TH>(sm, kmax, kmin);
  LinBins bins;
  if (!bins.set(key_value(kmax), key_value(kmin))) return false;       // a NaN makes it false too, whatever its sign
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int j = 0; j < NPT; ++j)
      if (used(c, j)) atomicAdd(&sm.lin[bins.of(key_value(key[c][j]))], 1u);
  __syncthreads();
  return select_by_bins<TH, NPT, CHUNKS>(sm, bins, k, o, [&](int c, uint32_t(&ck)[NPT], int32_t(&col)[NPT]) {
    uint32_t valid = 0;
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
      ck[j] = key[c][j];
      col[j] = i0 + c * kDirectChunk + j;
      valid |= (uint32_t)used(c, j) << j;
    }
    return valid;
  });
}

// One row, one CTA: the whole selection.
template <int TH>
__device__ __forceinline__ void topk_row(TopkSmem& sm, const float* logits, int64_t ld,
                                         const int32_t* __restrict__ ks, const int32_t* __restrict__ ke, int S, int k,
                                         int32_t* __restrict__ out, int one_pass, int row) {
  constexpr int kChunkHist = TH * kVec, kChunkFinal = TH * kEltPerThread, kCandPerThread = kCand / TH;
  const int tid = threadIdx.x;
  const int lo = ks ? max(ks[row], 0) : 0;
  const int hi = ke ? min(ke[row], S) : S;
  const int n = max(hi - lo, 0);
  int32_t* o = out + (int64_t)row * k;
  if (n <= k) {
    for (int j = tid; j < k; j += TH) o[j] = j < n ? lo + j : -1;
    return;
  }
  const float* x = logits + (int64_t)row * ld;
  const bool vec = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) && (ld % kVec == 0);
  const int base = lo & ~(kVec - 1);           // chunk origin: multiple of 4, <= lo

  if (one_pass && (n <= kDirectRow || vec)) {
    if (n <= kDirectChunk - 4 ? direct_row<TH, 1>(sm, x, vec, lo, hi, k, o)
        : n <= kDirectRow     ? direct_row<TH, 2>(sm, x, vec, lo, hi, k, o)
                              : sampled_single_pass<TH>(sm, x, lo, hi, k, o))
      return;
    __syncthreads();
  }

  uint32_t prefix = 0;    // value of the decided high key bits
  int pbits = 0;          // how many high bits are decided
  uint32_t need = k;      // elements still wanted from the set matching the prefix
  uint32_t cnt = 0;       // size of the threshold bin

  // ---- 1./2. histogram passes over the row ------------------------------------
  while (true) {
    const int dbits = min(kDigitBits, 32 - pbits);
    const int shift = 32 - pbits - dbits;
    const uint32_t dmask = (1u << dbits) - 1u;
    for (int b = tid; b < kBins; b += TH) sm.hist[b] = 0;
    __syncthreads();
    if (vec) {
      // interior float4s need no window test; the (at most two) edge float4s do
      const int first_full = (lo + kVec - 1) & ~(kVec - 1);
      const int last_full = hi & ~(kVec - 1);
      if (pbits == 0) {
#pragma unroll 4
        for (int i = first_full + tid * kVec; i < last_full; i += kChunkHist) {
          const float4 f = *reinterpret_cast<const float4*>(x + i);
          atomicAdd(&sm.hist[order_key(f.x) >> shift], 1u);
          atomicAdd(&sm.hist[order_key(f.y) >> shift], 1u);
          atomicAdd(&sm.hist[order_key(f.z) >> shift], 1u);
          atomicAdd(&sm.hist[order_key(f.w) >> shift], 1u);
        }
      } else {
        const int pshift = 32 - pbits;
#pragma unroll 4
        for (int i = first_full + tid * kVec; i < last_full; i += kChunkHist) {
          const float4 f = *reinterpret_cast<const float4*>(x + i);
          const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t key = order_key(v[j]);
            if ((key >> pshift) == prefix) atomicAdd(&sm.hist[(key >> shift) & dmask], 1u);
          }
        }
      }
      // edges: [lo, first_full) and [last_full, hi)
      const int n_head = min(first_full, hi) - lo;
      const int n_tail = last_full >= first_full ? hi - last_full : 0;
      if (tid < n_head + n_tail) {
        const int i = tid < n_head ? lo + tid : last_full + (tid - n_head);
        const uint32_t key = order_key(x[i]);
        if (pbits == 0 || (key >> (32 - pbits)) == prefix) atomicAdd(&sm.hist[(key >> shift) & dmask], 1u);
      }
    } else {
      for (int i = lo + tid; i < hi; i += TH) {
        const uint32_t key = order_key(x[i]);
        if (pbits == 0 || (key >> (32 - pbits)) == prefix) atomicAdd(&sm.hist[(key >> shift) & dmask], 1u);
      }
    }
    __syncthreads();
    find_threshold_bin<TH, kBins, false>(sm, sm.hist, need);
    prefix = (pbits == 0 ? 0u : (prefix << dbits)) | sm.bin;
    need = sm.need;
    cnt = sm.cnt;
    pbits += dbits;
    __syncthreads();
    if (cnt <= (uint32_t)kCand || pbits == 32) break;
  }

  // ---- 3. ordered pass: emit what is above the threshold bin, stage the bin ----
  const uint32_t n_above = k - need;
  const bool all_tied = (pbits == 32);           // every candidate equals the k-th value
  const int pshift = 32 - pbits;
  uint32_t base_sel = 0, base_cand = 0;
  const int n_chunks = (hi - base + kChunkFinal - 1) / kChunkFinal;
  for (int c = 0; c < n_chunks; ++c) {
    const int i0 = base + c * kChunkFinal + tid * kEltPerThread;
    float v[kEltPerThread];
    uint32_t fsel = 0, fcand = 0;
    if (i0 < hi) {
      if (vec) {
#pragma unroll
        for (int q = 0; q < kEltPerThread / kVec; ++q) {
          // a float4 that starts below hi lies inside the row's allocation (ld % 4 == 0)
          const float4 f = (i0 + q * kVec < hi) ? *reinterpret_cast<const float4*>(x + i0 + q * kVec)
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
          v[q * 4 + 0] = f.x; v[q * 4 + 1] = f.y; v[q * 4 + 2] = f.z; v[q * 4 + 3] = f.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < kEltPerThread; ++j) v[j] = (i0 + j >= lo && i0 + j < hi) ? x[i0 + j] : 0.f;
      }
      const bool interior = (i0 >= lo) && (i0 + kEltPerThread <= hi);
#pragma unroll
      for (int j = 0; j < kEltPerThread; ++j) {
        const uint32_t top = pshift >= 32 ? 0u : (order_key(v[j]) >> pshift);
        const bool in = interior || (i0 + j >= lo && i0 + j < hi);
        fsel |= (uint32_t)(in && top > prefix) << j;
        fcand |= (uint32_t)(in && top == prefix) << j;
      }
    }
    const uint32_t packed = __popc(fsel) | (__popc(fcand) << 16);
    uint32_t total;
    const uint32_t excl = block_exclusive_scan<TH>(sm, packed, c & 1, total);
    if (fsel | fcand) {
      uint32_t ps = base_sel + (excl & 0xffffu);
      uint32_t pc = base_cand + (excl >> 16);
#pragma unroll
      for (int j = 0; j < kEltPerThread; ++j) {
        if (fsel & (1u << j)) {
          o[ps++] = i0 + j;
        } else if (fcand & (1u << j)) {
          if (all_tied) {
            if (pc < need) o[n_above + pc] = i0 + j;
          } else {
            sm.cand_key[pc] = order_key(v[j]);
            sm.cand_idx[pc] = i0 + j;
          }
          ++pc;
        }
      }
    }
    base_sel += total & 0xffffu;
    base_cand += total >> 16;
  }
  if (all_tied) return;
  __syncthreads();

  // ---- 4. resolve the remaining digits on the staged candidates -----------------
  uint32_t ck[kCandPerThread];
  uint32_t valid = 0;
#pragma unroll
  for (int j = 0; j < kCandPerThread; ++j) {
    const uint32_t a = tid * kCandPerThread + j;        // contiguous per thread: keeps column order
    ck[j] = a < cnt ? sm.cand_key[a] : 0u;
    valid |= (uint32_t)(a < cnt) << j;
  }
  __syncthreads();                                      // keys are in registers: hist may reuse the storage
  digit_passes<TH, kCandPerThread>(sm, ck, valid, prefix, pbits, need, 32);
  // prefix is now the exact k-th largest key; `need` of the candidates equal to it are wanted.
  // Output layout: [0, n_above) above the bin, then candidates > key, then the `need` tied ones.
  emit_candidates<TH, kCandPerThread>(sm, ck, valid, prefix, need, n_above, k, o);
}

template <int TH, int PER_SM>
__global__ void __launch_bounds__(TH, PER_SM)
topk_select_kernel(const float* logits, int64_t ld, const int32_t* __restrict__ ks,
                   const int32_t* __restrict__ ke, int S, int k, int32_t* __restrict__ out, int one_pass) {
  __shared__ TopkSmem sm;
  launch_dependents();
  logits = grid_wait(logits);                            // read by plain loads: they may have been written while this kernel ran
  topk_row<TH>(sm, logits, ld, ks, ke, S, k, out, one_pass, blockIdx.x);
}

// sample = 0 forces the two-pass path on every row (the test hook that pits the two paths against each other)
int topk_select_launch(const float* logits, int64_t ld, const int32_t* ks, const int32_t* ke, int T, int S, int k,
                       int32_t* out, int sample, int overlapped, cudaStream_t stream) {
  if (T == 0 || k == 0) return DSA_OK;
  // Up to one row per SM a row has 1024 threads, beyond that 512, three rows to an SM: 7 rows of up to 33000 columns 11.0 us with 512,
  // 8.9 with 1024, 64 x 131072 18.5 and 13.3; 160 x 9000 11.5 and 15.5, 4096 x 32768 175 and 283.  (256 threads, five rows to an SM:
  // 4096 x 32768 207, 2048 x 2048 21.5.)
  if (T <= sm_count())
    launch_after(overlapped, topk_select_kernel<1024, 1>, dim3(T), 1024, 0, stream, logits, ld, ks, ke, S, k, out, sample);
  else
    launch_after(overlapped, topk_select_kernel<512, 3>, dim3(T), 512, 0, stream, logits, ld, ks, ke, S, k, out, sample);
  return check_launch("topk_select");
}

}  // namespace dsa
