// Token-sparse MLA prefill for calls of at most 32 heads (a tensor-parallel rank's share of the heads, small models): the function
// of sparse_mla.cu with scores and output TRANSPOSED, so that the heads are the N of the tensor-core tiles and not the M.
//   S^T [64 keys x N heads] = K Q^T     (M = 64, 36 K-steps over the 576 dims, both operands in shared memory)
//   O^T [512 dims x N heads] += V^T P^T (four M = 128 tiles, 4 K-steps over a block's 64 keys; V^T is the gathered latent rows
//                                        read through an MN-major descriptor, so nothing is transposed in memory)
// N is 16 or 32.  In the other kernel 16 heads fill an eighth of a 128-row tile that costs the tensor pipe as much as a full
// one, and the two CTAs of a pair exchange tiles that are mostly empty.  Here a CTA does a token by itself: every row of the list
// crosses from L2 once, 1152 bytes, to 148 SMs.
// Persistent CTAs, one per SM, each walking tokens with running counters, so that the gather and the scores of the next token run
// under the last softmax and the output of this one.
//   * warps 0-3: softmax and output.  An M = 64 accumulator keeps its rows in lanes 0-15 of each quadrant: a warp has 16 keys and
//     reads them with 16x256b loads, two keys and two heads of every eight to a lane.  Block maxima go over the lanes by three
//     shuffles and over the warps through shared memory; P leaves through stmatrix.trans as [head][key] rows, the K-major B operand.
//   * warp 4: MMA issue, whatever is ready first.  warp 5: reads every list once for its last used slot (which decides the
//     number of blocks) and for positions out of range, and sends for Q.
//   * warps 6-21: gather, four rows of a block each, by cp.async that arrive on the block's barrier by themselves.  The latent
//     rows lie in a ring of panel pairs (128 dims of 64 keys), freed one by one as P.V has read them, the rope panels in another.
// What bounds it: the tensor pipe, whose 52 MMAs a block cost 47 cycles each whatever their N (2450 cycles; the gather alone would
// take 1900).  us before (the pair kernel) and now: 16 heads, 2048 tokens x 2048 of 16384 keys 985 -> 571, 4096 tokens 1938 -> 1105, 2048
// tokens x 256 keys 276 -> 92; 32 heads 992 -> 705.  Tried: 128 keys a score tile (fewer MMAs, but then 1 1/4 blocks fit and the
// gather waits for P.V: 835 against 607); 64 heads as one N = 64 tile (Q takes the room of a block: 1127 against 1051 for the pair
// kernel, which therefore keeps them); the output put off until the next token's first P is on its way (spills: 668 against 610).
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

template <int N>
struct FewCfg {
  static constexpr int PAIRS = N == 16 ? 11 : 9;                    // ring of latent panel pairs (16 KB, 128 dims of a block); four to a block
  static constexpr int ROPES = 3;                                   // ring of rope panels (8 KB), free again after the scores
  static constexpr int PBUFS = 2;
  static constexpr int Q_BYTES = 9 * N * 128, P_BYTES = N * 128;
  static constexpr int BAR_BYTES = 512;
  static constexpr int SMEM = PAIRS * 2 * kFewPanel + ROPES * kFewPanel + Q_BYTES + PBUFS * P_BYTES + BAR_BYTES + kFewValidRing * kFewBlk +
                              2 * kFewSoftmaxWarps * N * 4;
  static constexpr uint32_t COL_O = 0, COL_S = 4 * N, COLS = COL_S + 2 * N <= 256 ? 256 : 512;
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

template <int N>
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

  // A unit is a token.  Every role walks u = blockIdx.x, + gridDim.x, ... with running counters: nu units, n blocks, nq units
  // with blocks.
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
    for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++nu) {
      const int32_t* row = a.idx + (int64_t)u * a.K;
      int last = -1;
      for (int j0 = 0; j0 < a.K; j0 += 512) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int j = j0 + i * 32 + lane;
          const int id = j < a.K ? __ldg(row + j) : -1;
          if (id >= 0 && id < a.S_kv) last = j;
          if (id >= a.S_kv && a.status) atomicCAS(a.status, kStatusOk, kStatusBadIndex);
        }
      }
      last = __reduce_max_sync(0xffffffffu, last);
      const int nb = (last + kFewBlk) / kFewBlk;
      ok = mbar_wait_warp(&tok_free[nu % kFewTokRing], ((nu / kFewTokRing) & 1) ^ 1, abort_flag, a.status);
      if (!ok) break;
      if (lane == 0) {
        tok_s[nu % kFewTokRing] = nb;
        mbar_arrive(&tok_full[nu % kFewTokRing]);
      }
      __syncwarp();
      if (nb == 0) continue;
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
    for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++nu) {
      const int nb = unit_blocks(nu, ok);
      if (!ok) break;
      if (nb == 0) continue;
      ok = mbar_wait_warp(q_full, nq & 1, abort_flag, a.status);
      if (!ok) break;
      const uint32_t end = n + nb;
      uint32_t qk = n, pv = n, idle = 0;
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
                umma_f16_ss(tmem + C::COL_O + mt * N, vd + ks * (2048 >> 4), pd + 2 * ks, idesc_pv, pv != n || ks != 0);
              umma_commit(&pair_free[slot]);
            }
            umma_commit(&pv_done[pv & 1]);
          }
          __syncwarp();
          ++pv;
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
    int nxt = load_id(blockIdx.x, 0);
    for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++nu) {
      const int nb = unit_blocks(nu, ok);
      if (!ok) break;
      if (nb == 0) nxt = load_id(u + gridDim.x, 0);
      for (int j = 0; j < nb; ++j, ++n) {
        const int id = nxt < a.S_kv ? nxt : -1;        // -1 = empty slot; bad positions are flagged by the warp that read the list
        nxt = j + 1 < nb ? load_id(u, j + 1) : load_id(u + gridDim.x, 0);
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
    for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++nu) {
      __nv_bfloat16* out = a.out + (int64_t)u * a.H * kFewDv;
      const int nb = unit_blocks(nu, ok);
      if (!ok) break;
      if (nb == 0) {                                   // nothing selected: zero rows
        for (int i = warp * 32 + lane; i < a.H * (kFewDv / 8); i += kFewSoftmaxWarps * 32)
          reinterpret_cast<uint4*>(out)[i] = make_uint4(0, 0, 0, 0);
        continue;
      }
      float m[2 * NH], l[2 * NH];                      // heads 8 i + 2 (lane % 4), + 1: references (log2), sums over this thread's keys
#pragma unroll
      for (int i = 0; i < 2 * NH; ++i) { m[i] = -CUDART_INF_F; l[i] = 0.f; }
      for (int j = 0; j < nb; ++j, ++n) {
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
        if (lane < 4) {
#pragma unroll
          for (int i = 0; i < NH; ++i) *reinterpret_cast<float2*>(mx + warp * N + 8 * i + 2 * lane) = make_float2(bm[2 * i], bm[2 * i + 1]);
        }
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
          if (j > 0) {                                 // O must be quiescent: P.V of the block before complete
            ok = mbar_wait_warp(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag, a.status);
            if (!ok) break;
            tc_fence_after();
            float* fac = max_s + ((n + 1) & 1) * 4 * N + warp * N;
            if (lane < 4) {
#pragma unroll
              for (int i = 0; i < NH; ++i) *reinterpret_cast<float2*>(fac + 8 * i + 2 * lane) = make_float2(f[2 * i], f[2 * i + 1]);
            }
            __syncwarp();
#pragma unroll 1
            for (int c = 0; c < 4 * N; c += 16) {
              uint32_t ov[16];
              tmem_ld16(t_row + C::COL_O + c, ov);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * fac[(c & (N - 1)) + i]);
              tmem_st16(t_row + C::COL_O + c, ov);
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
      if (!ok) break;
      // row sums: over the lanes that share a head, then over the warps
#pragma unroll
      for (int o = 4; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 2 * NH; ++i) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
      float* sum_s = max_s + (n & 1) * 4 * N;
      if (lane < 4) {
#pragma unroll
        for (int i = 0; i < NH; ++i) *reinterpret_cast<float2*>(sum_s + warp * N + 8 * i + 2 * lane) = make_float2(l[2 * i], l[2 * i + 1]);
      }
      ok = all_meet();
      if (!ok) break;
      // a head's quotient is taken once, into this warp's row of the other half (taken by every thread for every tile: 48 -> 85 us
      // for 2048 tokens x 64 keys)
      float* inv_s = max_s + ((n + 1) & 1) * 4 * N + warp * N;
      if (lane < N) {
        const float sum = (sum_s[lane] + sum_s[N + lane]) + (sum_s[2 * N + lane] + sum_s[3 * N + lane]);
        inv_s[lane] = sum > 0.f ? 1.f / sum : 0.f;
      }
      __syncwarp();
      ok = mbar_wait_warp(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag, a.status);
      if (!ok) break;
      tc_fence_after();
      const int even = (lane & 1) ^ 1;
#pragma unroll 1
      for (int c = 0; c < 4 * N; c += 16) {            // 16 heads of this lane's dim of a 128-dim tile
        uint32_t ov[16];
        tmem_ld16(t_row + C::COL_O + c, ov);
        const int h0 = c & (N - 1);
        float inv[16];
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 f = *reinterpret_cast<const float4*>(inv_s + h0 + i);
          inv[i] = f.x; inv[i + 1] = f.y; inv[i + 2] = f.z; inv[i + 3] = f.w;
        }
        tmem_wait_ld();
        // two neighbouring dims to a word: the even lane takes the pair of the even head, the odd lane that of the odd one
        __nv_bfloat16* o = out + (int64_t)h0 * kFewDv + (c / N) * 128 + warp * 32 + (lane & ~1);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float x0 = __uint_as_float(ov[i]) * inv[i], x1 = __uint_as_float(ov[i + 1]) * inv[i + 1];
          const float y = __shfl_xor_sync(0xffffffffu, even ? x1 : x0, 1);
          const int h = i + (lane & 1);
          if (h0 + h < a.H) *reinterpret_cast<uint32_t*>(o + h * kFewDv) = even ? few_pack(x0, y) : few_pack(y, x1);
        }
      }
      tc_fence_before();
      ok = all_meet();                                 // sum_s may be written again
    }
  }

  __syncwarp();
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

template <int N>
static int launch_few(const void* q, const FewArgs& args, cudaStream_t stream) {
  using C = FewCfg<N>;
  FewArgs a = args;
  CUtensorMap tq;
  const int rc = make_tmap_2d_bytes(&tq, q, (uint64_t)a.T * a.H, kFewRowBytes, kFewRowBytes, 128, N);
  if (rc) return rc;
  if (a.H > N) return set_error(DSA_ERR_SHAPE, "sparse_mla: %d heads in a kernel for %d", a.H, N);
  auto kern = sparse_mla_few_kernel<N>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
    return set_error(DSA_ERR_CUDA, "sparse_mla: cannot raise dynamic shared memory to %d", C::SMEM);
  kern<<<a.T < sm_count() ? a.T : sm_count(), kFewThreads, C::SMEM, stream>>>(tq, a, a.T);
  return check_launch("sparse_mla");
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
