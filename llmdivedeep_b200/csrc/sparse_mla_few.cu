// Token-sparse MLA prefill for calls of at most 32 heads (a tensor-parallel rank's share of the heads, small models): the function
// of sparse_mla.cu with scores and output TRANSPOSED, so that the heads are the N of the tensor-core tiles and not the M.
//   S^T [64 keys x N heads] = K Q^T     (M = 64, 36 K-steps over the 576 dims, both operands in shared memory)
//   O^T [512 dims x N heads] += V^T P^T (four M = 128 tiles, 4 K-steps over a block's 64 keys; V^T is the gathered latent rows
//                                        read through an MN-major descriptor, so nothing is transposed in memory)
// N is 16 or 32.  In the other kernel 16 heads fill an eighth of a 128-row tile that costs the tensor pipe as much as a full
// one, and the two CTAs of a pair exchange tiles that are mostly empty.  Here a CTA does a token by itself: every row of the list
// crosses from L2 once, 1152 bytes, to 148 SMs.
// Persistent CTAs, one per SM, each walking tokens with running counters, so that the gather and the scores of the next token run
// under the last softmax and the output of this one.  A list of more than four blocks is taken in two halves, each with a softmax
// reference, row sums and an output accumulator of its own, merged at the end: where a call has at most one token for every two
// SMs, a cluster of two CTAs takes a half each and 256 dims of the merge, and the bits of a row are the same as when one CTA
// takes both (they must not depend on the size of the call: rows are dealt to ranks).
//   * warps 0-3: softmax and output.  An M = 64 accumulator keeps its rows in lanes 0-15 of each quadrant: a warp has 16 keys and
//     reads them with 16x256b loads, two keys and two heads of every eight to a lane.  Block maxima go over the lanes by three
//     shuffles and over the warps through shared memory; P leaves through stmatrix.trans as [head][key] rows, the K-major B operand.
//   * warp 4: MMA issue, whatever is ready first.  warp 5: reads every list once for its last used slot (which decides the
//     number of blocks) and for positions out of range, and sends for Q.
//   * warps 6-21: gather, four rows of a block each, by cp.async that arrive on the block's barrier by themselves.  The latent
//     rows lie in a ring of panel pairs (128 dims of 64 keys), freed one by one as P.V has read them, the rope panels in another.
// What bounds it: the issue of 52 MMAs a block, 47 cycles each whatever their N (2450 cycles; the tensor pipe itself is 13 % busy
// with 16 heads, 22 % with 32; the gather alone would take 1900); in calls of few tokens the chain of one list.  us, keys of 16384:
// the kernel for many heads, this one with a list in one piece (and read 16 slots a lane at a time for its end), as it is now.
//   16 heads, 2048 keys: 1 token 33.9, 52.2, 25.5; 74 tokens 36.4, 53.1, 27.0; 148 tokens 71.5, 54.0, 44.1; 2048 tokens 1090, 566, 548
//             256 keys:  1 token 9.9, 10.9, 9.5;   74 tokens 11.0, 11.3, 9.9;  2048 tokens 272, 91, 86
//   32 heads, 2048 keys: 1 token 34.1, 61.7, 29.8; 74 tokens 36.6, 62.5, 31.6; 148 tokens 71.6, 63.5, 53.2; 2048 tokens 1090, 701, 680
//             256 keys:  1 token 10.1, 12.5, 11.1; 74 tokens 11.0, 13.0, 11.6; 2048 tokens 281, 117, 117
// (At 256 keys and up to 74 tokens 17 to 32 heads stay up to 10 % behind; halves of two blocks end that and cost 10 % at 2048 tokens.)
// Tried: 128 keys a score tile (fewer MMAs, but then 1 1/4 blocks fit and the gather waits for P.V: 835 against 607); 64 heads as
// one N = 64 tile (Q takes the room of a block: 1127 against 1051 for the pair kernel, which therefore keeps them); the output put
// off until the next token's first P is on its way (spills: 668 against 610).
// Every wait is bounded (dsa_common.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math_constants.h>

#include "dsa_common.cuh"
#include "dsa_host.h"

namespace dsa {

struct FewArgs {
  const uint8_t* kv;              // [S_kv, 576] bf16 rows
  const int32_t* idx;             // [T, K] selected key positions (negative = empty)
  __nv_bfloat16* out;             // [T, H, 512]
  int T, H, K, S_kv;
  float scale_log2e;
  int* status;
};

constexpr int kFewGatherWarps = 16, kFewSoftmaxWarps = 4;
constexpr int kFewMmaWarp = kFewSoftmaxWarps, kFewStageWarp = kFewMmaWarp + 1, kFewGatherWarp0 = kFewStageWarp + 1;
constexpr int kFewThreads = (kFewGatherWarp0 + kFewGatherWarps) * 32;
constexpr int kFewBlk = 64;                            // keys per block
constexpr int kFewPanel = kFewBlk * 128;               // 64 keys x 64 dims, 128-byte swizzled
constexpr int kFewRowBytes = 1152, kFewDv = 512;
constexpr int kFewValidRing = 8;
constexpr int kFewTokRing = 4;
constexpr int kFewWhole = 4;                           // lists of more blocks than this are taken in two halves (below, the merge costs what they save)
// Slots of a list that a lane looks at together, without a branch.  With 16, and one for a bad position, the look was most of a
// call's start: 16 heads, 148 tokens x 2048 keys 54.0 -> 44.1 us.
constexpr int kFewLook = 32;

template <int N>
struct FewCfg {
  static constexpr int PAIRS = N == 16 ? 11 : 9;                    // ring of latent panel pairs (16 KB, 128 dims of a block); four to a block
  static constexpr int ROPES = 3;                                   // ring of rope panels (8 KB), free again after the scores
  static constexpr int PBUFS = 2;
  static constexpr int Q_BYTES = 9 * N * 128, P_BYTES = N * 128;
  static constexpr int BAR_BYTES = 512;
  static constexpr int SMEM = PAIRS * 2 * kFewPanel + ROPES * kFewPanel + Q_BYTES + PBUFS * P_BYTES + BAR_BYTES + kFewValidRing * kFewBlk +
                              6 * kFewSoftmaxWarps * N * 4;
  static constexpr uint32_t COL_O = 0, COL_S = 8 * N, COLS = COL_S + 2 * N <= 256 ? 256 : 512;      // O of two halves
  static_assert(SMEM <= 232448 && COL_S + 2 * N <= COLS, "budget of one CTA");
};

// 16 lanes x 256 bits: of every 8 columns i, lane t gets columns 2 (t % 4), + 1 of row t / 4 (registers 4 i, 4 i + 1) and of row
// t / 4 + 8 (4 i + 2, 4 i + 3)
__device__ __forceinline__ void few_ld_s(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ uint32_t few_pack(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float few_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void few_cp16(void* dst, const void* src, int src_bytes) {      // src_bytes 0: zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void few_cp_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The weights of the two halves' outputs, from their row sums and references (log2 units).
__device__ __forceinline__ void few_weights(float l0, float m0, float l1, float m1, float& w0, float& w1) {
  const float top = fmaxf(m0, m1);
  const float f0 = m0 == -CUDART_INF_F ? 0.f : few_exp2(m0 - top), f1 = m1 == -CUDART_INF_F ? 0.f : few_exp2(m1 - top);
  const float den = __fadd_rn(__fmul_rn(f0, l0), __fmul_rn(f1, l1));
  const float inv = den > 0.f ? 1.f / den : 0.f;
  w0 = __fmul_rn(f0, inv);
  w1 = __fmul_rn(f1, inv);
}
__device__ __forceinline__ float few_ld_peer(uint32_t addr) {
  float x;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(addr) : "memory");
  return x;
}
__device__ __forceinline__ uint32_t mapa_peer(uint32_t addr, uint32_t cta) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void few_ld_weights(const float* src, float (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const float4 f = *reinterpret_cast<const float4*>(src + i);
    w[i] = f.x; w[i + 1] = f.y; w[i + 2] = f.z; w[i + 3] = f.w;
  }
}
// 16 heads from h0 on of the dims d0 + lane of a token's output: two neighbouring dims to a word, the even lane takes the pair
// of the even head, the odd lane that of the odd one.
__device__ __forceinline__ void few_store(__nv_bfloat16* out, int heads, int h0, int d0, int lane, const float (&x)[16]) {
  const bool even = !(lane & 1);
  __nv_bfloat16* o = out + (int64_t)h0 * kFewDv + d0 + (lane & ~1);
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const float y = __shfl_xor_sync(0xffffffffu, even ? x[i + 1] : x[i], 1);
    const int h = i + (lane & 1);
    if (h0 + h < heads) *reinterpret_cast<uint32_t*>(o + h * kFewDv) = even ? few_pack(x[i], y) : few_pack(y, x[i + 1]);
  }
}
// every thread of both CTAs; what was written before is seen after
__device__ __forceinline__ void few_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// PAIR: a cluster of two CTAs to a token, each with one half of its list.
template <int N, bool PAIR>
__global__ void __launch_bounds__(kFewThreads, 1)
sparse_mla_few_kernel(const __grid_constant__ CUtensorMap tmap_q, const FewArgs a, const int n_units) {
  using C = FewCfg<N>;
  constexpr int NH = N / 8;                            // groups of eight heads: a thread has two adjacent heads of each
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* pair_s = smem;                              // [PAIRS][2 panels]
  uint8_t* rope_s = pair_s + C::PAIRS * 2 * kFewPanel; // [ROPES]
  uint8_t* q_s = rope_s + C::ROPES * kFewPanel;        // nine panels [N heads x 128 B]
  uint8_t* p_s = q_s + C::Q_BYTES;                     // P^T as [N heads][64 keys], swizzled
  uint64_t* bars = reinterpret_cast<uint64_t*>(p_s + C::PBUFS * C::P_BYTES);
  uint64_t* kv_full = bars + 0;                        // [4] gather -> MMA, by block
  uint64_t* pair_free = bars + 4;                      // [PAIRS <= 11] P.V of those 128 dims has read the pair
  uint64_t* rope_free = bars + 15;                     // [ROPES <= 3] the block's scores have read the panel
  uint64_t* s_full = bars + 18;                        // [2] MMA -> softmax
  uint64_t* p_full = bars + 20;                        // [2] softmax -> MMA
  uint64_t* pv_done = bars + 22;                       // [2] P.V of the block complete
  uint64_t* q_full = bars + 24;
  uint64_t* q_free = bars + 25;                        // the unit's last scores have read Q
  uint64_t* tok_full = bars + 26;                      // [4] the unit's number of blocks is known
  uint64_t* tok_free = bars + 30;                      // [4]
  uint64_t* meet = bars + 34;                          // the four softmax warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 35);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* tok_s = const_cast<int*>(abort_flag) + 1;             // [4]
  uint8_t* valid_s = reinterpret_cast<uint8_t*>(bars) + C::BAR_BYTES; // [8 blocks][64] 1 = the slot is in use
  // [2][4 warps][N] block maxima by block parity.  The half that the block does not use is free: a warp's row of it takes the
  // factors of a rescale, and all of it the row sums at the end of a unit.
  float* max_s = reinterpret_cast<float*>(valid_s + kFewValidRing * kFewBlk);
  float* half_s = max_s + 2 * kFewSoftmaxWarps * N;    // [row sums, references][4 warps][N] of the first half (PAIR: of this CTA's)
  float* wgt_s = half_s + 2 * kFewSoftmaxWarps * N;    // [4 warps][2][N] weights of the halves' outputs

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (warp == 0) {
    for (int i = lane; i < 35; i += 32) {
      const uint32_t count = i < 4 ? kFewGatherWarps * 33u
                             : (i == 20 || i == 21 || i == 34) ? uint32_t(kFewSoftmaxWarps)
                             : (i >= 30 && i < 34) ? uint32_t(kFewSoftmaxWarps + 1 + kFewGatherWarps) : 1u;
      mbar_init(bars + i, count);
    }
    mbar_fence_init();
    if (lane == 0) *abort_flag = 0;
  } else if (warp == kFewMmaWarp) {
    tmem_alloc(tmem_slot, C::COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // A unit is a token.  Every role walks u = blockIdx.x, + gridDim.x, ... (PAIR: one unit) with running counters: nu units, n
  // blocks, nq units with blocks.  Blocks [b0, b1) of a list are this CTA's; from first_half(nb) on, a list has its second
  // softmax state and output.
  const int rank = PAIR ? blockIdx.x & 1 : 0, u0 = PAIR ? blockIdx.x >> 1 : blockIdx.x, du = PAIR ? n_units : gridDim.x;
  auto first_half = [](int nb) { return nb > kFewWhole ? (nb + 1) / 2 : nb; };
  auto my_blocks = [&](int nb, int& b0, int& b1) {
    b0 = PAIR && rank ? first_half(nb) : 0;
    b1 = PAIR && !rank ? first_half(nb) : nb;
  };
  auto unit_blocks = [&](uint32_t nu, bool& ok) -> int {     // number of blocks of the CTA's nu-th unit; the warp's reading frees the slot
    ok = mbar_wait_warp(&tok_full[nu % kFewTokRing], (nu / kFewTokRing) & 1, abort_flag, a.status);
    const int nb = ok ? tok_s[nu % kFewTokRing] : 0;
    __syncwarp();
    if (lane == 0) mbar_arrive(&tok_free[nu % kFewTokRing]);
    return nb;
  };

  if (warp == kFewStageWarp) {
    // ------------- the last used slot of every list (it decides the number of blocks), and Q -------------
    uint32_t nu = 0, nq = 0;
    bool ok = true;
    for (int u = u0; u < n_units && ok; u += du, ++nu) {
      const int32_t* row = a.idx + (int64_t)u * a.K;
      int last = -1, top = -1;
#pragma unroll 1
      for (int j0 = lane; j0 < a.K; j0 += 32 * kFewLook) {      // all of a lane's loads are requested before the first is looked at
        int id[kFewLook];
#pragma unroll
        for (int i = 0; i < kFewLook; ++i) id[i] = j0 + i * 32 < a.K ? __ldg(row + j0 + i * 32) : -1;
#pragma unroll
        for (int i = 0; i < kFewLook; ++i) {
          if (id[i] >= 0 && id[i] < a.S_kv) last = j0 + i * 32;
          top = max(top, id[i]);
        }
      }
      last = __reduce_max_sync(0xffffffffu, last);
      if (top >= a.S_kv && a.status) atomicCAS(a.status, kStatusOk, kStatusBadIndex);
      const int nb = (last + kFewBlk) / kFewBlk;
      ok = mbar_wait_warp(&tok_free[nu % kFewTokRing], ((nu / kFewTokRing) & 1) ^ 1, abort_flag, a.status);
      if (!ok) break;
      if (lane == 0) {
        tok_s[nu % kFewTokRing] = nb;
        mbar_arrive(&tok_full[nu % kFewTokRing]);
      }
      __syncwarp();
      int b0, b1;
      my_blocks(nb, b0, b1);
      if (b0 == b1) continue;
      ok = mbar_wait_warp(q_free, (nq & 1) ^ 1, abort_flag, a.status);
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(q_full, C::Q_BYTES);
      __syncwarp();
      if (lane < 9) tma_load_2d(q_s + lane * N * 128, &tmap_q, lane * 32, u * a.H, q_full);   // x in 4-byte units
      ++nq;
    }
  } else if (warp == kFewMmaWarp) {
    // ------------------------------- MMA issuer -------------------------------
    constexpr uint32_t idesc_qk = umma_idesc(1, 1, 0, 0, kFewBlk, N);
    constexpr uint32_t idesc_pv = umma_idesc(1, 1, 1, 0, 128, N);
    const uint64_t qdesc = umma_smem_desc(smem_u32(q_s), 16, 1024, kSwz128);
    const uint64_t kdesc = umma_smem_desc(smem_u32(pair_s), 16, 1024, kSwz128);
    const uint64_t rdesc = umma_smem_desc(smem_u32(rope_s), 16, 1024, kSwz128);
    const uint64_t vdesc = umma_smem_desc(smem_u32(pair_s), kFewPanel, 1024, kSwz128);
    const uint64_t pdesc = umma_smem_desc(smem_u32(p_s), 16, 1024, kSwz128);
    constexpr uint64_t kPair = (2 * kFewPanel) >> 4, kOne = kFewPanel >> 4, kQPanel = (N * 128) >> 4;
    uint32_t nu = 0, nq = 0, n = 0;
    bool ok = true;
    for (int u = u0; u < n_units && ok; u += du, ++nu) {
      const int nb = unit_blocks(nu, ok);
      if (!ok) break;
      int b0, b1;
      my_blocks(nb, b0, b1);
      if (b0 == b1) continue;
      ok = mbar_wait_warp(q_full, nq & 1, abort_flag, a.status);
      if (!ok) break;
      const uint32_t end = n + (b1 - b0), half = PAIR ? end : n + first_half(nb);
      uint32_t qk = n, pv = n, begun = n, d_o = tmem + C::COL_O, idle = 0;      // begun: first block of the half
      // Whatever is ready first: the scores of the next block, at most two ahead of P.V (whose P says that the score buffer
      // has been read), or P.V of the oldest (whose P, for a unit's first block, says that the last unit's O has been read).
      while (pv < end) {
        if (qk < end && qk < pv + 2 && __all_sync(0xffffffffu, mbar_try_wait(&kv_full[qk & 3], (qk >> 2) & 1))) {
          fence_async_smem();                          // the rows were written by cp.async, the tensor core reads through the async proxy
          tc_fence_after();
          if (elect_one()) {
            const uint32_t d = tmem + C::COL_S + (qk & 1) * N;
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
              const uint64_t kd = kdesc + ((4 * qk + mt) % C::PAIRS) * kPair;
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                umma_f16_ss(d, kd + (ks >> 2) * kOne + 2 * (ks & 3), qdesc + (2 * mt + (ks >> 2)) * kQPanel + 2 * (ks & 3), idesc_qk, (mt | ks) != 0);
            }
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_f16_ss(d, rdesc + (qk % C::ROPES) * kOne + 2 * ks, qdesc + 8 * kQPanel + 2 * ks, idesc_qk, 1);
            umma_commit(&s_full[qk & 1]);
            umma_commit(&rope_free[qk % C::ROPES]);
            if (qk + 1 == end) umma_commit(q_free);
          }
          __syncwarp();
          ++qk;
          idle = 0;
        } else if (pv < qk && __all_sync(0xffffffffu, mbar_try_wait(&p_full[pv & 1], (pv >> 1) & 1))) {
          tc_fence_after();
          if (elect_one()) {
            const uint64_t pd = pdesc + (pv % C::PBUFS) * (C::P_BYTES >> 4);
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
              const uint32_t slot = (4 * pv + mt) % C::PAIRS;
              const uint64_t vd = vdesc + slot * kPair;
#pragma unroll
              for (int ks = 0; ks < 4; ++ks)           // 16 keys: 16 rows x 128 B further into each panel, 32 B along P's rows
                umma_f16_ss(d_o + mt * N, vd + ks * (2048 >> 4), pd + 2 * ks, idesc_pv, pv != begun || ks != 0);
              umma_commit(&pair_free[slot]);
            }
            umma_commit(&pv_done[pv & 1]);
          }
          __syncwarp();
          if (++pv == half) {
            begun = half;
            d_o += 4 * N;
          }
          idle = 0;
        } else if (++idle > kFastSpins) {
          if (idle > kSpinLimit || aborted_warp(abort_flag)) {      // the same for all lanes: they leave together
            *abort_flag = 1;
            if (a.status) atomicCAS(a.status, kStatusOk, kStatusWaitTimeout);
            ok = false;
            break;
          }
          __nanosleep(40);
        }
      }
      n = end;
      ++nq;
    }
  } else if (warp >= kFewGatherWarp0) {
    // ----------------------------- gather: four rows of every block to a warp -----------------------------
    const int r0 = 4 * (warp - kFewGatherWarp0);
    uint32_t nu = 0, n = 0;
    bool ok = true;
    // lane group g of eight has the id of row r0 + g; requested a block ahead, across units too
    auto load_id = [&](int u, int blk) -> int {
      const int j = blk * kFewBlk + r0 + (lane >> 3);
      return u < n_units && j < a.K ? __ldg(a.idx + (int64_t)u * a.K + j) : -1;
    };
    const int guess = PAIR && rank ? first_half((a.K + kFewBlk - 1) / kFewBlk) : 0;      // before the list's end is known
    int nxt = load_id(u0, guess);
    for (int u = u0; u < n_units && ok; u += du, ++nu) {
      const int nb = unit_blocks(nu, ok);
      if (!ok) break;
      int b0, b1;
      my_blocks(nb, b0, b1);
      if (PAIR ? b0 != guess : nb == 0) nxt = PAIR ? load_id(u, b0) : load_id(u + du, 0);
      for (int j = b0; j < b1; ++j, ++n) {
        const int id = nxt < a.S_kv ? nxt : -1;        // -1 = empty slot; bad positions are flagged by the warp that read the list
        nxt = j + 1 < b1 ? load_id(u, j + 1) : load_id(u + du, 0);
        {
          const uint32_t slot = n % C::ROPES;
          if (n >= C::ROPES) ok = mbar_wait_warp(&rope_free[slot], (n / C::ROPES - 1) & 1, abort_flag, a.status);
          if (!ok) break;
          const int r = r0 + (lane >> 3);
          few_cp16(rope_s + slot * kFewPanel + r * 128 + (((lane ^ r) & 7) << 4),
                   a.kv + (int64_t)max(id, 0) * kFewRowBytes + kFewDv * 2 + (lane & 7) * 16, id >= 0 ? 16 : 0);
        }
        const int id0 = __shfl_sync(0xffffffffu, id, (lane >> 4) * 8), id1 = __shfl_sync(0xffffffffu, id, 16 + (lane >> 4) * 8);
        const uint8_t* src0 = a.kv + (int64_t)max(id0, 0) * kFewRowBytes + (lane & 15) * 16;
        const uint8_t* src1 = a.kv + (int64_t)max(id1, 0) * kFewRowBytes + (lane & 15) * 16;
        const int ra = r0 + (lane >> 4), rb = ra + 2;
        const uint32_t off0 = ((lane >> 3) & 1) * kFewPanel + ra * 128 + (((lane ^ ra) & 7) << 4);
        const uint32_t off1 = ((lane >> 3) & 1) * kFewPanel + rb * 128 + (((lane ^ rb) & 7) << 4);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          const uint32_t g = 4 * n + mt, slot = g % C::PAIRS;
          if (ok && g >= C::PAIRS) ok = mbar_wait_warp(&pair_free[slot], (g / C::PAIRS - 1) & 1, abort_flag, a.status);
          if (!ok) break;
          uint8_t* dst = pair_s + slot * 2 * kFewPanel;
          few_cp16(dst + off0, src0 + mt * 256, id0 >= 0 ? 16 : 0);
          few_cp16(dst + off1, src1 + mt * 256, id1 >= 0 ? 16 : 0);
        }
        if (!ok) break;
        if ((lane & 7) == 0) valid_s[(n % kFewValidRing) * kFewBlk + r0 + (lane >> 3)] = id >= 0;
        few_cp_arrive(&kv_full[n & 3]);                // this thread's arrival, once its copies have landed ...
        __syncwarp();
        if (lane == 0) mbar_arrive(&kv_full[n & 3]);   // ... and the warp's, for the validity bytes
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // nothing of this thread's is in flight when it leaves
  } else {
    // ------------- softmax and output: warp w has keys 16 w.. of a block, and dims 32 w.. of every 128 of the output -------------
    const uint32_t t_row = tmem + (uint32_t(warp * 32) << 16);
    uint32_t nu = 0, n = 0, met = 0;
    bool ok = true;
    auto all_meet = [&]() -> bool {                    // the four warps: what was written to shared memory before is seen after
      __syncwarp();
      if (lane == 0) mbar_arrive(meet);
      return mbar_wait_warp(meet, met++ & 1, abort_flag, a.status);
    };
    // this warp's row: heads 8 i + 2 (lane % 4), + 1 of every thread's values
    auto put_row = [&](float* row, const float(&v)[2 * NH]) {
      if (lane < 4) {
#pragma unroll
        for (int i = 0; i < NH; ++i) *reinterpret_cast<float2*>(row + 8 * i + 2 * lane) = make_float2(v[2 * i], v[2 * i + 1]);
      }
    };
    auto sum_lanes = [&](float(&l)[2 * NH]) {          // over the lanes that share a head
#pragma unroll
      for (int o = 4; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 2 * NH; ++i) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
    };
    for (int u = u0; u < n_units && ok; u += du, ++nu) {
      const int nb = unit_blocks(nu, ok);
      if (!ok) break;
      int b0, b1;
      my_blocks(nb, b0, b1);
      if (b0 == b1) {                                  // nothing selected: zero rows (or no second half)
        for (int i = warp * 32 + lane; nb == 0 && rank == 0 && i < a.H * (kFewDv / 8); i += kFewSoftmaxWarps * 32)
          reinterpret_cast<uint4*>(a.out + (int64_t)u * a.H * kFewDv)[i] = make_uint4(0, 0, 0, 0);
        continue;
      }
      float m[2 * NH], l[2 * NH];                      // heads 8 i + 2 (lane % 4), + 1: references (log2), sums over this thread's keys
#pragma unroll
      for (int i = 0; i < 2 * NH; ++i) { m[i] = -CUDART_INF_F; l[i] = 0.f; }
      uint32_t begun = n, stop = n + (PAIR ? b1 - b0 : first_half(nb)), t_o = t_row + C::COL_O;
      while (true) {                                   // over the halves
        for (; n != stop; ++n) {
          ok = mbar_wait_warp(&s_full[n & 1], (n >> 1) & 1, abort_flag, a.status);
          if (!ok) break;
          tc_fence_after();
          uint32_t sv[4 * NH];
#pragma unroll
          for (int i = 0; i < NH; i += 2) few_ld_s(t_row + C::COL_S + (n & 1) * N + 8 * i, *reinterpret_cast<uint32_t(*)[8]>(&sv[4 * i]));
          const uint8_t* valid = valid_s + (n % kFewValidRing) * kFewBlk + 16 * warp + (lane >> 2);
          const bool va = valid[0], vb = valid[8];
          tmem_wait_ld();
          tc_fence_before();
          float s[4 * NH], bm[2 * NH];
#pragma unroll
          for (int i = 0; i < NH; ++i) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              s[4 * i + e] = va ? __uint_as_float(sv[4 * i + e]) : -CUDART_INF_F;
              s[4 * i + 2 + e] = vb ? __uint_as_float(sv[4 * i + 2 + e]) : -CUDART_INF_F;
              bm[2 * i + e] = fmaxf(s[4 * i + e], s[4 * i + 2 + e]);
            }
          }
#pragma unroll
          for (int o = 4; o < 32; o <<= 1)
#pragma unroll
            for (int i = 0; i < 2 * NH; ++i) bm[i] = fmaxf(bm[i], __shfl_xor_sync(0xffffffffu, bm[i], o));
          float* mx = max_s + (n & 1) * 4 * N;
          put_row(mx + warp * N, bm);
          ok = all_meet();
          if (!ok) break;
          bool grown = false;
          float f[2 * NH];
#pragma unroll
          for (int i = 0; i < NH; ++i) {
            float2 b = make_float2(-CUDART_INF_F, -CUDART_INF_F);
#pragma unroll
            for (int w = 0; w < kFewSoftmaxWarps; ++w) {
              const float2 x = *reinterpret_cast<const float2*>(mx + w * N + 8 * i + 2 * (lane & 3));
              b.x = fmaxf(b.x, x.x);
              b.y = fmaxf(b.y, x.y);
            }
            const float bx[2] = {b.x * a.scale_log2e, b.y * a.scale_log2e};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float m_old = m[2 * i + e];
              const bool up = bx[e] - m_old > kMaxRaise;  // also true when m is still -inf and the maximum finite
              f[2 * i + e] = up ? few_exp2(m_old - bx[e]) : 1.f;
              if (up) m[2 * i + e] = bx[e];
              grown |= up;
            }
          }
          if (__any_sync(0xffffffffu, grown)) {          // the same in all four warps
#pragma unroll
            for (int i = 0; i < 2 * NH; ++i) l[i] *= f[i];
            if (n != begun) {                            // O must be quiescent: P.V of the block before complete
              ok = mbar_wait_warp(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag, a.status);
              if (!ok) break;
              tc_fence_after();
              float* fac = max_s + ((n + 1) & 1) * 4 * N + warp * N;
              put_row(fac, f);
              __syncwarp();
#pragma unroll 1
              for (int c = 0; c < 4 * N; c += 16) {
                uint32_t ov[16];
                tmem_ld16(t_o + c, ov);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * fac[(c & (N - 1)) + i]);
                tmem_st16(t_o + c, ov);
              }
              tmem_wait_st();
              __syncwarp();
            }
          }
          uint32_t pk[2 * NH];                           // [group of eight heads][keys t / 4, t / 4 + 8]: two heads each
#pragma unroll
          for (int i = 0; i < NH; ++i) {
            const float m0 = m[2 * i] == -CUDART_INF_F ? 0.f : m[2 * i], m1 = m[2 * i + 1] == -CUDART_INF_F ? 0.f : m[2 * i + 1];
            const float p0 = few_exp2(fmaf(s[4 * i], a.scale_log2e, -m0)), p1 = few_exp2(fmaf(s[4 * i + 1], a.scale_log2e, -m1));
            const float p2 = few_exp2(fmaf(s[4 * i + 2], a.scale_log2e, -m0)), p3 = few_exp2(fmaf(s[4 * i + 3], a.scale_log2e, -m1));
            pk[2 * i] = few_pack(p0, p1);
            pk[2 * i + 1] = few_pack(p2, p3);
            add_bf16x2(pk[2 * i], l[2 * i], l[2 * i + 1]);
            add_bf16x2(pk[2 * i + 1], l[2 * i], l[2 * i + 1]);
          }
          if (n >= C::PBUFS) {                           // that P buffer has been read
            ok = mbar_wait_warp(&pv_done[(n - C::PBUFS) & 1], ((n - C::PBUFS) >> 1) & 1, abort_flag, a.status);
            if (!ok) break;
          }
          // transposed on the way: row = head, 16-byte chunk = eight keys
          uint8_t* p = p_s + (n % C::PBUFS) * C::P_BYTES;
#pragma unroll
          for (int i = 0; i < NH; i += 2) {
            const int h = 8 * (i + (lane >> 4)) + (lane & 7), ch = 2 * warp + ((lane >> 3) & 1);
            asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
                         ::"r"(smem_u32(p + h * 128 + ((ch ^ (h & 7)) << 4))), "r"(pk[2 * i]), "r"(pk[2 * i + 1]), "r"(pk[2 * i + 2]), "r"(pk[2 * i + 3])
                         : "memory");
          }
          fence_async_smem();                            // visible to the tensor core's reads
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[n & 1]);
        }
        if (PAIR || !ok || nb <= kFewWhole || t_o != t_row + C::COL_O) break;
        // the first half's sums and references, read after the unit's last meeting
        sum_lanes(l);
        put_row(half_s + warp * N, l);
        put_row(half_s + (kFewSoftmaxWarps + warp) * N, m);
#pragma unroll
        for (int i = 0; i < 2 * NH; ++i) { m[i] = -CUDART_INF_F; l[i] = 0.f; }
        begun = n;
        stop = n + nb / 2;
        t_o += 4 * N;
      }
      if (!ok) break;
      __nv_bfloat16* out = a.out + (int64_t)u * a.H * kFewDv;
      // row sums over the warps
      const bool halves = nb > kFewWhole;
      float* sum_s = max_s + (n & 1) * 4 * N;
      sum_lanes(l);
      put_row(sum_s + warp * N, l);
      float* wgt = wgt_s + warp * 2 * N;
      if (halves) put_row(wgt + N, m);
      ok = all_meet();
      if (!ok) break;
      // a head's weights are computed once (a quotient by every thread for every tile: 48 -> 85 us for 2048 tokens x 64 keys)
      if (lane < N) {
        auto over_warps = [&](const float* r) { return (r[lane] + r[N + lane]) + (r[2 * N + lane] + r[3 * N + lane]); };
        const float sum = over_warps(sum_s);
        if (!halves) {
          wgt[lane] = sum > 0.f ? 1.f / sum : 0.f;
        } else if constexpr (PAIR) {                   // for the peer, which merges the other 256 dims
          half_s[lane] = sum;
          half_s[N + lane] = wgt[N + lane];
        } else {
          float w0, w1;
          few_weights(over_warps(half_s), half_s[(kFewSoftmaxWarps + warp) * N + lane], sum, wgt[N + lane], w0, w1);
          wgt[lane] = w0;
          wgt[N + lane] = w1;
        }
      }
      __syncwarp();
      ok = mbar_wait_warp(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag, a.status);
      if (!ok) break;
      tc_fence_after();
      if (PAIR && halves) {
        // the peer's two tiles of 128 dims, [tile][head][dim], where the (idle) panels were
        float* give = reinterpret_cast<float*>(pair_s) + warp * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < 2 * N; c += 16) {
          uint32_t ov[16];
          tmem_ld16(t_row + C::COL_O + (rank ^ 1) * 2 * N + c, ov);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) give[(c + i) * 128] = __uint_as_float(ov[i]);
        }
      } else if (!halves) {
#pragma unroll 1
        for (int c = 0; c < 4 * N; c += 16) {          // 16 heads of this lane's dim of a 128-dim tile
          uint32_t ov[16];
          tmem_ld16(t_row + C::COL_O + c, ov);
          float w[16], x[16];
          few_ld_weights(wgt + (c & (N - 1)), w);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = __fmul_rn(__uint_as_float(ov[i]), w[i]);
          few_store(out, a.H, c & (N - 1), (c / N) * 128 + warp * 32, lane, x);
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < 4 * N; c += 16) {
          uint32_t ov[16], ow[16];
          tmem_ld16(t_row + C::COL_O + c, ov);
          tmem_ld16(t_row + C::COL_O + 4 * N + c, ow);
          float w[16], x[16];
          few_ld_weights(wgt + (c & (N - 1)), w);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = __fmul_rn(__uint_as_float(ov[i]), w[i]);
          few_ld_weights(wgt + N + (c & (N - 1)), w);
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = __fmaf_rn(__uint_as_float(ow[i]), w[i], x[i]);
          few_store(out, a.H, c & (N - 1), (c / N) * 128 + warp * 32, lane, x);
        }
      }
      tc_fence_before();
      ok = all_meet();                                 // sum_s may be written again
    }
  }

  __syncwarp();
  if constexpr (PAIR) {
    few_cluster_sync();                                // both halves are complete, and what they give one another is written
    const int nb = tok_s[0];
    if (warp < kFewSoftmaxWarps && nb > kFewWhole && !aborted_warp(abort_flag)) {
      const uint32_t t_o = tmem + (uint32_t(warp * 32) << 16) + C::COL_O + rank * 2 * N;
      float* wgt = wgt_s + warp * 2 * N;
      if (lane < N) {
        const uint32_t peer = mapa_peer(smem_u32(half_s + lane), rank ^ 1);
        const float l = half_s[lane], m = half_s[N + lane], lp = few_ld_peer(peer), mp = few_ld_peer(peer + 4 * N);
        float w0, w1;
        few_weights(rank ? lp : l, rank ? mp : m, rank ? l : lp, rank ? m : mp, w0, w1);
        wgt[lane] = w0;
        wgt[N + lane] = w1;
      }
      __syncwarp();
      const uint32_t taken = mapa_peer(smem_u32(reinterpret_cast<float*>(pair_s) + warp * 32 + lane), rank ^ 1);
#pragma unroll 1
      for (int c = 0; c < 2 * N; c += 16) {
        uint32_t ov[16];
        float x[16];
        tmem_ld16(t_o + c, ov);
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = few_ld_peer(taken + (c + i) * 512);
        float w0[16], w1[16];
        few_ld_weights(wgt + (c & (N - 1)), w0);
        few_ld_weights(wgt + N + (c & (N - 1)), w1);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float mine = __uint_as_float(ov[i]);
          x[i] = __fmaf_rn(rank ? mine : x[i], w1[i], __fmul_rn(rank ? x[i] : mine, w0[i]));
        }
        few_store(a.out + (int64_t)u0 * a.H * kFewDv, a.H, c & (N - 1), (2 * rank + c / N) * 128 + warp * 32, lane, x);
      }
    }
    __syncwarp();
    few_cluster_sync();                                // the peer has read what this CTA gave it
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                                   // a wait gave up: let the copies in flight land (bounded)
    if (threadIdx.x == 0)
      for (int w = 0; w < 64; ++w) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kFewMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, C::COLS);
  }
}

int make_tmap_2d_bytes(CUtensorMap* m, const void* base, uint64_t rows, uint64_t inner_bytes, uint64_t row_pitch,
                       uint32_t box_bytes, uint32_t box_rows);

template <int N, bool PAIR>
static int launch_few(const void* q, const FewArgs& a, cudaStream_t stream) {
  using C = FewCfg<N>;
  if (a.H > N) return set_error(DSA_ERR_SHAPE, "sparse_mla: %d heads in a kernel for %d", a.H, N);
  CUtensorMap tq;
  const int rc = make_tmap_2d_bytes(&tq, q, (uint64_t)a.T * a.H, kFewRowBytes, kFewRowBytes, 128, N);
  if (rc) return rc;
  auto kern = sparse_mla_few_kernel<N, PAIR>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
    return set_error(DSA_ERR_CUDA, "sparse_mla: cannot raise dynamic shared memory to %d", C::SMEM);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(PAIR ? 2 * a.T : min(a.T, sm_count()));
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = PAIR ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, tq, a, a.T);          // its error is the launch check's
  return check_launch("sparse_mla");
}

// Two CTAs to a token where that takes one round of them and lists may have two halves (2048 keys, 16 heads: 74 tokens 27.0
// us, 148 by one CTA each 44.1; two rounds of clusters would take longer).  The bits of a row do not
// depend on it: both forms keep the halves apart and merge them by the same operations.
template <int N>
static int launch_few(const void* q, const FewArgs& a, cudaStream_t stream) {
  return a.K > kFewWhole * kFewBlk && a.T <= sm_count() / 2 ? launch_few<N, true>(q, a, stream) : launch_few<N, false>(q, a, stream);
}

int sparse_mla_few_launch(const void* q, const void* kv, const int32_t* idx, void* out, int T, int H, int S_kv, int K,
                          float scale, int32_t* status, cudaStream_t stream) {
  FewArgs a{};
  a.kv = static_cast<const uint8_t*>(kv);
  a.idx = idx;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.T = T; a.H = H; a.K = K; a.S_kv = S_kv;
  a.scale_log2e = scale * 1.4426950408889634f;
  a.status = status;
  if (H <= 16) return launch_few<16>(q, a, stream);
  return launch_few<32>(q, a, stream);
}

}  // namespace dsa
