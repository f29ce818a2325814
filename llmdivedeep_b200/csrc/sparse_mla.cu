// Token-sparse MLA attention on sm_100a (MQA over the shared 576-dim latent KV, 512-dim V):
//   o[t, h, :] = sum_j softmax_j(scale * q[t, h, :] . kv[idx[t, j], :]) * kv[idx[t, j], :512]
// Takes the place of the block-sparse stand-in the reference reaches through
// register_sparse_fa() (sparse_attn/DSA.py:208-249); the reference itself has no sparse-MLA
// kernel, no latent cache and no decode path (sparse_attn/DSA.py:475-477).
//
// One CLUSTER of two CTAs per (query token, group of up to 128 heads).  The 576-dim row splits
// into nine 64-dim panels: eight latent panels (they are also V) and the rope panel.  CTA c of the
// pair owns latent panels 4c..4c+3 -- its half of V -- and half of the rope panel's contraction:
//   * it gathers only those 576 bytes of every selected row (36 KB per 64-key block, five blocks in
//     flight), swizzled by the writing threads: cp.async straight out of the bf16 KV, or -- for the
//     paged FP8 latent cache of decode -- cp.async of the raw rows two blocks ahead and a conversion
//     e4m3 x group scale -> bf16 into one of four buffers;
//   * its five Q panels live in tensor memory as the A operand, so Q.K^T reads no shared memory for
//     Q, and it computes a PARTIAL score tile S_c = Q_c K_c^T (18 tcgen05.mma kind::f16 of N = 64);
//   * the two partial tiles ([128 heads x 64 keys], rounded to fp16 for the way: 16 KB) are exchanged
//     through distributed shared memory, every warp sending its own 2 KB with one bulk copy (quadrants
//     of tensor memory without heads stand by).  Each
//     side adds what arrives to its own unrounded fp32 partial scores and runs the whole softmax.  The
//     two sides' scores differ by the rounding of what was sent, so the halves of an output row come from
//     two softmaxes: each CTA normalises its half of O by the row sums of its own P, and a part of a split
//     list is weighted half by half.  P is off by at most scale * 2^-11 * |partial score of the peer|,
//     relative: less than its bf16 rounding (2^-9) while scale * |partial| is below 4.  A partial beyond
//     +-65504 saturates on the way, for the receiving side only;
//   * P is the A operand (from tensor memory) of O_c += P V_c (4 MMAs of N = 256) with the gathered
//     panels read through an MN-major descriptor.
// O is rescaled in tensor memory only when the running maximum grows by more than kMaxRaise (32 log2 units).  The row sums add up P as
// it was rounded for the tensor core, so that the rounding of a key that dominates its row cancels in the quotient: error against
// float64 2.16e-3 -> 2.11e-3 at q x 1, 2.40e-3 -> 2.04e-3 at q x 4 (of the tree before: sums of the unrounded P, reference raised
// by 8), for 0.5 % of the time.
//
// What bounds it: the time a KV buffer is held.  A block's rows are needed from the scores to P.V, with the exchange
// and the softmax in between; that round trip (gather 2400 cycles, scores 1000, exchange + softmax 3600, P.V with its
// queueing 1700), divided by five buffers, is the ~1700 cycles a block takes, against 1400 of tensor pipe.  Everything
// below therefore shortens the trip: sixteen softmax warps in two sets that take alternate blocks, eleven gather warps
// (a warp keeps about eight 512-byte requests going, whether cp.async or TMA gather4), arrivals by the copies themselves.
// 4096 tokens x 2048 keys: 3594 us with eight softmax warps in lockstep, MMAs issued from a lane-dependent branch (~137
// cycles each; see dsa_common.cuh) and TMA gather; 3125 with warp-uniform issue; 2860 with two sets of softmax warps;
// 2418 with sixteen and setmaxnreg; 2215 with this gather; 2266 with the exchange stage released by the data; 2180 with waits that
// look once before they loop; 2140 with the gather's bounds known to the compiler and no zero-fill arithmetic where a warp's slots
// are all in use (1091 TFLOP/s; short runs at full clock -- at the power cap, 1600 MHz, 2500 against 3565).  At 2180, q scaled by 2
// and 4 takes the same; by 8, where maxima do outgrow the reference, 2570 us (with the reference raised by 8: 2550, 2935 and
// 3030 us).  Tried on top: the exchange by st.async (3320:
// the stores drain slowly and clog the gather), by loads from the peer's shared memory (3560: the release at cluster
// scope costs ~2300 cycles), a quarter of the exponentials as polynomials on the FMA pipe (+3 %: the issue slots are
// short too).
//
// Roles: warps 0-15 exchange + softmax + output, warp 16 MMA issuer (owns the TMEM allocation), warps 17-27 gather.
//  Softmax warp w: set w / 8 takes the blocks of that parity, key half (w / 4) % 2, heads = TMEM lanes
// 32 (w % 4)..; a thread owns one head and half of a block's keys.  The two threads of a head tell each other their
// block maxima through shared memory (rounded up to bf16: any common reference point is exact for a softmax); from the
// maxima of all blocks in order every thread follows the running reference by itself, so that one set can run ahead of
// the other; row sums stay per thread until the end.
// Of the 71000 cycles a token takes, 54000 are its blocks; the rest is start, Q, first rows (6300), the last softmax, P.V,
// output and the pair's exit (7500) and the relaunch (1600).  Persistent pairs that run ahead into the next token were built
// and dropped (2710): without a panel of free shared memory Q and the output move by 16-byte accesses a row apart (7400
// and 8000 cycles), and the two CTAs drift against each other.
// Decode, batch 64 (a call, launch included): 105 us with eight gather warps that met at two barriers per block, 72 us with
// eleven that never wait for one another.  Loads into registers one block ahead in place of the raw stages: 94 us (the rows
// take about 3000 cycles to come).  The gather then costs issue slots, about as many as the softmax.
// Every wait is bounded (dsa_common.cuh); the two CTAs leave together through a cluster barrier.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <math_constants.h>

#include "dsa_common.cuh"
#include "dsa_host.h"

namespace dsa {

constexpr int kMlaDqk = 576;
constexpr int kMlaDv = 512;
constexpr int kMlaDvHalf = 256;
constexpr int kMlaBlk = 64;                        // keys per block
constexpr int kMlaPanels = 5;                      // panels per CTA: four latent (its V half) + rope
constexpr int kMlaBufs = 5;                        // KV buffers in shared memory
constexpr int kMlaQPanelBytes = 128 * 128;         // 128 heads x 128 B
constexpr int kMlaKPanelBytes = kMlaBlk * 128;     // 64 keys x 128 B
constexpr int kMlaRopeOff = 4 * kMlaKPanelBytes;   // in a buffer: four latent panels, then this CTA's 64 rope bytes of every row
constexpr int kMlaKBytes = kMlaRopeOff + kMlaBlk * 64;        // 36864 per buffer
constexpr int kMlaXBytes = 128 * kMlaBlk * 2;      // one partial score tile, fp16: 16384
constexpr int kMlaXWarp = kMlaXBytes / 8;          // ... a warp's part of it
constexpr int kMlaValidRing = 8;                   // validity bytes (64 per block) for the softmax: >= blocks in flight
// The registers of the launch (896 threads x 72) are dealt out again: setmaxnreg moves what the issuing and gathering
// warps do not need to the softmax.
template <bool FP8_PAGED>
struct MlaRegs {                                   // decode's gather converts in registers
  static constexpr int kSoftmax = FP8_PAGED ? 88 : 96, kOther = FP8_PAGED ? 48 : 40;
  static_assert(512 * kSoftmax + 384 * kOther <= 896 * 72, "more registers than the launch has");
};
constexpr int kMlaMaxParts = 8;                    // parts of a split list
constexpr int kMlaMaxK = 2048;                     // slots of a list
constexpr int kMlaThreads = 896, kMlaSoftmaxWarps = 16, kMlaMmaWarp = 16, kMlaGatherWarp0 = 17, kMlaGatherWarps = 11;
template <int R>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
// Waits here loop unrolled by four: with the compact loop decode is 7 % slower (batch 64 68.6 us against 64.2, both with the first
// look in front) and prefill the same.
__device__ __forceinline__ bool mla_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  return mbar_wait_warp<4>(bar, parity, abort_flag, status);
}
constexpr int kMlaLooks = (kMlaMaxK + kMlaThreads - 1) / kMlaThreads;
constexpr int kMlaBarBytes = 512;                  // mbarriers and a few words
constexpr int kMlaPairBytes = 4 * 2 * 128 * 2;     // block maxima: [block mod 4][key half][head], bf16
constexpr int kMlaSmemBytes = kMlaBufs * kMlaKBytes + 2 * kMlaXBytes + kMlaBarBytes +
                              kMlaValidRing * kMlaBlk + kMlaPairBytes;
static_assert(kMlaSmemBytes <= 232448, "shared memory budget of one CTA");
constexpr int kLatentTokenBytes = 656;             // 512 e4m3 + 4 fp32 scales + 64 bf16 rope
constexpr int kLatentPage = 64;
// tensor-memory columns: O 256, S 64, P 32, Q 5 x 32
constexpr uint32_t kColO = 0, kColS = 256, kColP = kColS + kMlaBlk, kColQ = kColP + kMlaBlk / 2, kMlaTmemCols = 512;
static_assert(kColQ + kMlaPanels * 32 <= kMlaTmemCols, "tensor memory budget");

struct MlaArgs {
  const uint8_t* kv;              // prefill: [S_kv, 576] bf16 rows
  const uint8_t* cache;           // decode: [num_pages*64, 656] bytes
  const int32_t* block_table;     // decode: [B, table_stride]
  const int32_t* idx;             // [T, K] selected key positions (negative = empty)
  __nv_bfloat16* out;             // [T, H, 512]
  int64_t table_stride;
  int T, H, K;
  int S_kv;                       // prefill: rows of kv; decode: logical positions per sequence
  int num_phys_rows;              // decode: rows of the cache
  float scale_log2e;              // softmax scale * log2(e)
  int* status;
  int n_full;                     // the first n_full queries are one unit (CTA pair) each; ...
  int n_split;                    // ... the slot list of every later one is cut into n_split parts, a unit each (decode)
  float* part_o;                  // [(T - n_full) * n_split, H, 512] fp32 normalised partial outputs
  float* part_lse;                // [(T - n_full) * n_split, 2, H] log2-sum-exp of each part as each CTA of the pair has it (-inf = empty part)
  int tma_out;                    // the output tensor map is valid: full 128-head groups leave through TMA stores
};

// ---- cluster helpers ----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Arrive on the peer's barrier to say "this warp has READ the tile".  Relaxed: a release at cluster scope costs a memory
// fence of thousands of cycles per block, and nothing written by this thread has to become visible.  But a relaxed arrival
// orders nothing, and straight after the loads it overtakes them -- they queue behind the gather's copies in the load/store
// unit, and the next tile then lands on top of this one before it is read (seen: a few tokens in ten thousand).  So the
// arrival takes the data as its operand: each lane gives a value computed from EVERY word that it loaded, the vote needs all
// lanes' values, and the arrival is predicated on the vote, so that it cannot issue before the loads have returned, whatever
// the compiler does with the code around it.  `x` comes out of fmaxf, which returns numbers or the canonical NaN: it never is
// the bit pattern compared with (a signalling NaN), which the compiler cannot know.  (A register-OR of the loaded words
// as that value, to send the arrival earlier, cost more than it gained: 2228 -> 2280 us.)
__device__ __forceinline__ void mbar_arrive_remote_after(uint32_t cluster_addr, float x, bool leader) {
  const bool seen = __any_sync(0xffffffffu, __float_as_uint(x) != 0x7f812345u);
  if (leader)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n\t}"
        ::"r"(cluster_addr), "r"(static_cast<uint32_t>(seen)) : "memory");
}
// this CTA's shared memory -> the peer's, completion counted on the peer's mbarrier
__device__ __forceinline__ void bulk_copy_to_peer(uint32_t dst_cluster, const void* src, uint32_t bytes, uint32_t bar_cluster) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst_cluster), "r"(smem_u32(src)), "r"(bytes), "r"(bar_cluster) : "memory");
}

// one [rows x 128 B] panel, shared memory (128-B swizzle) -> global, tracked by the thread's bulk group
__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(smem_u32(src)) : "memory");
}
__device__ __forceinline__ void bulk_commit_and_wait_read() {      // shared memory may be reused / released afterwards
  asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {      // out-of-range values saturate to +-65504
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// a pair of fp16 values plus a pair of fp32 values, one mixed-precision add each
__device__ __forceinline__ void add_f16x2(uint32_t h, float x, float y, float& sx, float& sy) {
  asm("{\n\t.reg .b16 l, u;\n\tmov.b32 {l, u}, %2;\n\tadd.rn.f32.f16 %0, l, %3;\n\tadd.rn.f32.f16 %1, u, %4;\n\t}"
      : "=f"(sx), "=f"(sy) : "r"(h), "f"(x), "f"(y));
}
// A warp's part of a partial score tile is [32 heads][32 keys] fp16, 64 bytes per thread.  The 16-byte chunks c (0..3) of a
// row are rotated by the lane pair, so that the eight lanes of a quarter-warp hit different banks.
__device__ __forceinline__ int xchg_off(int lane, int c) { return lane * 64 + (((c ^ (lane >> 1)) & 3) << 4); }
// fp32 -> bf16 bits, rounded towards +infinity
__device__ __forceinline__ uint32_t bf16_bits_round_up(float x) {
  const uint32_t b = __float_as_uint(x);
  return ((b >> 31) || (b & 0x7fffffffu) >= 0x7f800000u) ? (b >> 16) : ((b + 0xffffu) >> 16);
}

// ---- paged FP8 latent cache (decode) ------------------------------------------------------------
__device__ __forceinline__ void cp_async_16(void* dst, const void* src, int src_bytes) {      // src_bytes 0: zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_16_all(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// counts as this thread's arrival on the barrier when all cp.async it has issued so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// A gather warp's raw rows of one block: per row this CTA's 256 e4m3 values, the four scales, this CTA's 64 rope bytes.
constexpr int kRawRow = 256 + 16 + 64, kRawRows = (kMlaBlk + kMlaGatherWarps - 1) / kMlaGatherWarps, kRawBytes = kRawRows * kRawRow;
constexpr int kRawInBuf = kMlaKBytes / kRawBytes;                     // of the 2 x 11 pieces, those in the fifth KV buffer
constexpr int kMlaSmemDecode = kMlaSmemBytes + (2 * kMlaGatherWarps - kRawInBuf) * kRawBytes;
static_assert(kRawRows % 2 == 0 && kMlaSmemBytes % 16 == 0 && kMlaSmemDecode <= 232448, "raw rows of decode");
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Eight e4m3 values times their group scale, rounded to bf16; an empty slot's zeros (values and scale) stay zeros.
__device__ __forceinline__ uint4 e4m3x8_to_bf16(uint2 raw, float sc) {
  const uint32_t w[2] = {raw.x, raw.y};
  const uint64_t sc2 = pack_f32x2(sc, sc);
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_fp8x2_storage_t pr = static_cast<__nv_fp8x2_storage_t>((w[i >> 1] >> (16 * (i & 1))) & 0xffffu);
    const __half2_raw h2 = __nv_cvt_fp8x2_to_halfraw2(pr, __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h2));
    float x, y;
    unpack_f32x2(mul_f32x2(pack_f32x2(f.x, f.y), sc2), x, y);
    o[i] = pack_bf16x2(x, y);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// OVERLAPPED: a launch that may start under the end of the top-k's (decode of few sequences; in the others its loads and their
// place cost 2 %: batch 148 122.3 -> 124.9 us).
template <bool FP8_PAGED, bool OVERLAPPED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kMlaThreads, 1)
sparse_mla_kernel(const __grid_constant__ CUtensorMap tmap_q,
                  const __grid_constant__ CUtensorMap tmap_o, const MlaArgs a) {
  constexpr int NB = FP8_PAGED ? kMlaBufs - 1 : kMlaBufs;      // KV buffers in use (decode: the fifth one's space holds raw rows)
  extern __shared__ __align__(1024) uint8_t smem[];            // the swizzled panels need 1024-byte alignment
  uint8_t* kv_s = smem;                                        // five buffers: four panels [64 keys x 128 B] and 64 x 64 B
  uint8_t* send_s = kv_s + kMlaBufs * kMlaKBytes;              // this CTA's partial score tile on its way out
  uint8_t* recv_s = send_s + kMlaXBytes;                       // the peer's
  uint64_t* bars = reinterpret_cast<uint64_t*>(recv_s + kMlaXBytes);
  uint64_t* q_full = bars + 0;
  uint64_t* q_moved = bars + 1;                      // Q is in tensor memory, its staging areas are free
  uint64_t* o_final = bars + 2;
  uint64_t* s_free = bars + 3;                       // a set has read S into registers
  uint64_t* p_full = bars + 4;                       // softmax -> MMA
  // by block parity: a set looks at every second block only, and a barrier of its own cannot run two phases ahead of it
  uint64_t* s_full = bars + 5;                       // [2] MMA -> softmax
  uint64_t* pv_done = bars + 7;                      // [2] P.V of a block finished: O is quiescent, P is free
  uint64_t* pm_full = bars + 9;                      // [2][4 quadrants] both key halves' block maxima are in pm_s
  uint64_t* recv_full = bars + 17;                   // [16 warps] the peer's part of a partial tile has landed in recv_s
  uint64_t* xchg_free = bars + 33;                   // [16] the peer has read what this CTA's warp sent
  uint64_t* kv_full = bars + 49;                     // [5] gather -> MMA
  uint64_t* kv_free = bars + 54;                     // [5] P.V of the block finished: its KV buffer is free
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 59);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* last_s = reinterpret_cast<int*>(tmem_slot + 2);         // short rows: the last usable slot
  uint8_t* valid_s = reinterpret_cast<uint8_t*>(bars) + kMlaBarBytes;       // [kMlaValidRing][64] 1 = the slot of the block is in use
  uint16_t* pm_s = reinterpret_cast<uint16_t*>(valid_s + kMlaValidRing * kMlaBlk);          // block maxima, rounded up to bf16

  const int cta = blockIdx.x & 1, peer = cta ^ 1;              // rank in the cluster = V half = contraction part
  const int unit = blockIdx.x >> 1;
  const int part = FP8_PAGED ? unit - a.n_full : -1;           // >= 0: a part of a split slot list (prefill's are never cut)
  const int n_split = part < 0 ? 1 : a.n_split, t = part < 0 ? unit : a.n_full + part / n_split, split = part < 0 ? 0 : part % n_split;
  const int hg = blockIdx.z;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int k_per = ((a.K + n_split - 1) / n_split + kMlaBlk - 1) / kMlaBlk * kMlaBlk;   // slots per part
  const int k_lo = min(a.K, split * k_per), k_cnt = min(a.K, k_lo + k_per) - k_lo;
  const int32_t* idx_row = a.idx + (int64_t)t * a.K + k_lo;
  const int heads_here = min(128, a.H - hg * 128);
  const int n_quad = (heads_here + 31) / 32;                   // quadrants of tensor memory with heads in them: the others' warps stand by
  // the five Q panels wait at the end of the KV buffers (from buffer kQBuf0 on) for their move into tensor memory
  constexpr int kQStage = NB * kMlaKBytes - kMlaPanels * kMlaQPanelBytes, kQBuf0 = kQStage / kMlaKBytes;
  static_assert(kQStage >= 0 && kQStage % 1024 == 0, "Q staging");
  auto q_stage = [&](int lp) -> uint8_t* { return kv_s + kQStage + lp * kMlaQPanelBytes; };

  // ---- set-up, arranged so that nothing waits for anything it does not need ------------------------------------
  // every warp requests the last 32 slots of the list (they decide the number of key blocks), the gather warps their slots of the
  // first block and every thread its share of the whole list.  A kernel that started under the top-k's end reads it
  // after the wait for that, and by loads that may not be served from before; its set-up comes first.
  if constexpr (OVERLAPPED) launch_dependents();
  int tail = -1, slot_pos = -1;
  int look[kMlaLooks];
  const int tail_j = k_cnt - 32 + lane;
  const int slot = warp >= kMlaGatherWarp0 && lane < kRawRows ? warp - kMlaGatherWarp0 + lane * kMlaGatherWarps : kMlaBlk;
  auto list_at = [&](int j) { return OVERLAPPED ? idx_row[j] : __ldg(idx_row + j); };
  auto request_list = [&]() {
    if constexpr (OVERLAPPED) idx_row = grid_wait(idx_row);
    tail = tail_j >= 0 ? list_at(tail_j) : -1;
    slot_pos = slot < kMlaBlk && slot < k_cnt ? list_at(slot) : -1;
#pragma unroll
    for (int u = 0; u < kMlaLooks; ++u) {
      const int j = threadIdx.x + u * kMlaThreads;
      look[u] = j < k_cnt - 32 ? list_at(j) : -1;
    }
  };
  if constexpr (!OVERLAPPED) request_list();
  // Meanwhile warp 0 initialises the barriers (one per lane) and sends for Q (one panel per lane) and the MMA warp allocates
  // tensor memory
  if (warp == 0) {
    for (int i = lane; i < 59; i += 32) {
      const uint32_t count = i == 1 ? 16u                                            // q_moved: lane 0 of the softmax warps
                             : (i == 3 || i == 4) ? 2u * n_quad                      // s_free, p_full: lane 0 of a set's warps
                             : (i >= 9 && i <= 16) ? 2u                              // pm_full: the two warps of a quadrant
                             : (i >= 49 && i <= 53) ? (FP8_PAGED ? uint32_t(kMlaGatherWarps) : kMlaGatherWarps * 33u)
                                                    : 1u;                            // the others
      mbar_init(bars + i, count);
    }
    mbar_fence_init();
    if (lane == 0) {
      *abort_flag = 0;
      *last_s = -1;
    }
    __syncwarp();
    if (lane == 0) mbar_expect_tx(q_full, kMlaPanels * kMlaQPanelBytes);
    __syncwarp();
    // Q is on its way before anything else happens: into this CTA's own shared memory, counted on its own barrier
    if (lane < kMlaPanels)                             // x in 4-byte units: 32 per panel
      tma_load_2d(q_stage(lane), &tmap_q, (lane < 4 ? cta * 4 + lane : 8) * 32, t * a.H + hg * 128, q_full);
    if (lane == kMlaPanels && a.tma_out) tma_prefetch_desc(&tmap_o);
  } else if (warp == kMlaMmaWarp) {
    tmem_alloc(tmem_slot, kMlaTmemCols);
    tmem_relinquish();
  }
  if constexpr (OVERLAPPED) request_list();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // The last usable slot decides the number of key blocks (the same number in both CTAs of the pair).  It is among the last 32
  // but for short rows (the first 2048 of every prompt): there the shares of all threads decide.  Rows 0-295, K = 2048, 128
  // heads: 103 us with every warp walking back 128 slots a turn, 55 with the shares requested here, 50 with them under way
  // since the start (full rows pay nothing for it: 4096 x 2048 keys 2280 us without, 2255 with).
  int nblk;
  {
    const uint32_t hit = __ballot_sync(0xffffffffu, tail >= 0 && tail < a.S_kv);
    int last = k_cnt - 1 - __clz(hit);
    if (hit == 0) {                                    // the same answer in every warp
      last = -1;
#pragma unroll
      for (int u = 0; u < kMlaLooks; ++u)
        if (look[u] >= 0 && look[u] < a.S_kv) last = threadIdx.x + u * kMlaThreads;
      last = __reduce_max_sync(0xffffffffu, last);
      if (lane == 0 && last >= 0) atomicMax(last_s, last);
      __syncthreads();
      last = *last_s;
    }
    nblk = (last + kMlaBlk) / kMlaBlk;
  }
  if (nblk == 0) {   // nothing selected: the output row is zero (a part: weight zero in the combine); no cluster traffic yet
    if (threadIdx.x < 128 && threadIdx.x < heads_here) {
      if (part < 0) {
        uint4* o = reinterpret_cast<uint4*>(a.out + ((int64_t)t * a.H + hg * 128 + threadIdx.x) * kMlaDv + cta * kMlaDvHalf);
        for (int c = 0; c < kMlaDvHalf * 2 / 16; ++c) o[c] = make_uint4(0, 0, 0, 0);
      } else {
        const int64_t prow = (int64_t)part * a.H + hg * 128 + threadIdx.x;
        float4* o = reinterpret_cast<float4*>(a.part_o + prow * kMlaDv + cta * kMlaDvHalf);
        for (int c = 0; c < kMlaDvHalf / 4; ++c) o[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        a.part_lse[((int64_t)part * 2 + cta) * a.H + hg * 128 + threadIdx.x] = -CUDART_INF_F;
      }
    }
    // an index that is out of range is still reported
    for (int j = threadIdx.x; j < k_cnt; j += kMlaThreads)
      if (idx_row[j] >= a.S_kv && a.status) atomicCAS(a.status, kStatusOk, kStatusBadIndex);
    if (threadIdx.x == 0) mbar_wait(q_full, 0, abort_flag, a.status);     // the Q copy must have landed before the CTA goes
    if (warp == kMlaMmaWarp) tmem_dealloc(*tmem_slot, kMlaTmemCols);
    return;
  }
  const uint32_t tmem = *tmem_slot;
  // The peer's barriers must be initialised before anything is sent to it.  Every thread arrives here; the warps that
  // talk to the peer (softmax) wait before their first remote access, the others only before they leave, so that the
  // round trip through the cluster barrier is off the path to the first MMA.
  cluster_arrive();
  bool left = false;                                           // this warp has arrived at the barrier that the pair leaves through

  if (warp >= kMlaSoftmaxWarps) regs_dec<MlaRegs<FP8_PAGED>::kOther>();
  else regs_inc<MlaRegs<FP8_PAGED>::kSoftmax>();
  if (warp == kMlaMmaWarp) {
    // ------------------------------- MMA issuer -------------------------------
    // The partial scores of a block travel to the peer and through the softmax while the next blocks are scored: P.V of a
    // block is issued about two blocks after its scores.  MMAs complete in issue order.  The whole warp walks the loop on
    // warp-uniform values and elects a lane for the instructions (dsa_common.cuh).
    {
      constexpr uint32_t idesc_qk = umma_idesc(1, 1, 0, 0, 128, kMlaBlk);
      constexpr uint32_t idesc_pv = umma_idesc(1, 1, 0, 1, 128, kMlaDvHalf);
      bool ok = mla_wait(q_moved, 0, abort_flag, a.status);
      const uint64_t kdesc0 = umma_smem_desc(smem_u32(kv_s), 16, 1024, kSwz128);
      const uint64_t vdesc0 = umma_smem_desc(smem_u32(kv_s), kMlaKPanelBytes, 1024, kSwz128);
      const uint64_t rdesc0 = umma_smem_desc(smem_u32(kv_s + kMlaRopeOff), 16, 512, kSwz64);
      const uint32_t rope_ks = 2 * cta;              // this CTA's two K-steps of the rope panel
      // P.V of block j: four MMAs (N = 256) and the commits that release the block's KV buffer, P and O
      auto pv_mmas = [&](int j) {
        tc_fence_after();
        if (elect_one()) {
          const uint64_t vd = vdesc0 + uint64_t(j % NB) * (kMlaKBytes >> 4);
#pragma unroll
          for (int ks = 0; ks < kMlaBlk / 16; ++ks)     // 16 keys per step: 16 rows x 128 B further into each panel
            umma_f16_ts(tmem + kColO, tmem + kColP + 8 * ks, vd + ks * (2048 >> 4), idesc_pv, (j | ks) != 0);
          umma_commit(&kv_free[j % NB]);
          umma_commit(&pv_done[j & 1]);
          if (j == nblk - 1) umma_commit(o_final);
        }
        __syncwarp();
      };
      auto issue_qk = [&](int i) {
        fence_async_smem();                            // the rows were written by cp.async or st, the tensor core reads through the async proxy
        tc_fence_after();
        if (elect_one()) {
          const uint64_t kd0 = kdesc0 + uint64_t(i % NB) * (kMlaKBytes >> 4);
#pragma unroll
          for (int lp = 0; lp < 4; ++lp)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_f16_ts(tmem + kColS, tmem + kColQ + lp * 32 + 8 * ks, kd0 + uint64_t((lp * kMlaKPanelBytes) >> 4) + 2 * ks,
                          idesc_qk, (lp | ks) != 0);
#pragma unroll
          for (int u = 0; u < 2; ++u)
            umma_f16_ts(tmem + kColS, tmem + kColQ + 4 * 32 + 8 * (rope_ks + u), rdesc0 + uint64_t(i % NB) * (kMlaKBytes >> 4) + 2 * u,
                        idesc_qk, 1);
          umma_commit(&s_full[i & 1]);
        }
        __syncwarp();
      };
      // A fixed order: P.V two blocks behind the scores is about when its P is there, and what a KV buffer's round trip has
      // time for.  (Whatever is ready first, by polling three barriers: the same speed, and every look costs ~100 cycles.)
      for (int n = 0; n < nblk + 2 && ok; ++n) {
        if (n < nblk) {
          ok = mla_wait(&kv_full[n % NB], (n / NB) & 1, abort_flag, a.status);
          if (ok && n > 0) ok = mla_wait(s_free, (n - 1) & 1, abort_flag, a.status);
          if (!ok) break;
          issue_qk(n);
        }
        if (n >= 2) {
          ok = mla_wait(p_full, n & 1, abort_flag, a.status);
          if (!ok) break;
          pv_mmas(n - 2);
        }
      }
    }
  } else if (warp >= kMlaGatherWarp0) {
    // ----------------------------- gather of the selected rows -----------------------------
    const int w4 = warp - kMlaGatherWarp0;
    constexpr int kG = kMlaGatherWarps;
    // Five of a warp's six slots are always within the block: said so, prefill of 128 heads takes 2160 us instead of 2202 (4096 x 2048
    // keys), of 64 heads 1988 instead of 2044.  (Decode gains nothing.)
    if constexpr (!FP8_PAGED) __builtin_assume(w4 < kG);
    bool ok = true;
    // A warp fetches every kG-th slot of a block, six at most: lane j < 6 keeps the id of slot w4 + 11 j.
    auto load_pos = [&](int blk) -> int {
      const int j = blk * kMlaBlk + slot;
      return (slot < kMlaBlk && blk < nblk && j < k_cnt) ? list_at(j) : -1;
    };
    auto mark = [&](int blk, bool used) {
      if (slot < kMlaBlk) valid_s[(blk % kMlaValidRing) * kMlaBlk + slot] = used;
    };
    if constexpr (!FP8_PAGED) {
      // Row ids are requested one block ahead.  512 latent bytes are one 16-byte cp.async per lane, this CTA's 64 rope bytes
      // of all six rows another one.  Nobody waits for the copies here: they arrive on the block's barrier by themselves,
      // and the MMA warp orders them before the tensor core's reads (a proxy fence anywhere on the path between the two
      // will do).
      int nxt = slot_pos;
      const uint8_t* src_lat = a.kv + cta * (kMlaDvHalf * 2) + lane * 16;
      const uint8_t* src_rope = a.kv + kMlaDv * 2 + cta * 64 + (lane & 3) * 16;
      uint32_t round = 1;                              // parity of the buffer's last release
      for (int i = 0, kvb = 0; i < nblk; ++i) {
        int id = nxt;                                  // -1 = empty slot; bad positions are flagged and skipped
        if (id >= a.S_kv) {
          if (a.status) atomicCAS(a.status, kStatusOk, kStatusBadIndex);
          id = -1;
        }
        nxt = load_pos(i + 1);
        if (i == kQBuf0) ok = mla_wait(q_moved, 0, abort_flag, a.status);   // from here on the buffers held Q
        if (i >= NB) ok = mla_wait(&kv_free[kvb], round, abort_flag, a.status);
        if (!ok) break;
        mark(i, id >= 0);
        uint8_t* dst = kv_s + kvb * kMlaKBytes;
        uint8_t* dst_lat = dst + (lane >> 3) * kMlaKPanelBytes;
        // No empty slot among the warp's: nothing to zero-fill, half the address arithmetic (64 heads 1968 -> 1938 us, 128 heads 2138 ->
        // 2133, the ring's counters stepped instead of divided included).
        if (__all_sync(0xffffffffu, id >= 0 || slot >= kMlaBlk)) {
#pragma unroll
          for (int j = 0; j < kRawRows; ++j) {
            const int r = w4 + j * kG, rid = __shfl_sync(0xffffffffu, id, j);
            if (r < kMlaBlk) cp_async_16_all(dst_lat + r * 128 + (((lane ^ r) & 7) << 4), src_lat + (uint64_t)(uint32_t)rid * (kMlaDqk * 2));
          }
          const int r = w4 + (lane >> 2) * kG, rid = __shfl_sync(0xffffffffu, id, lane >> 2);
          if (lane < 4 * kRawRows && r < kMlaBlk)
            cp_async_16_all(dst + kMlaRopeOff + r * 64 + (((lane ^ (r >> 1)) & 3) << 4), src_rope + (uint64_t)(uint32_t)rid * (kMlaDqk * 2));
        } else {
#pragma unroll
          for (int j = 0; j < kRawRows; ++j) {
            const int r = w4 + j * kG, rid = __shfl_sync(0xffffffffu, id, j);
            if (r < kMlaBlk)
              cp_async_16(dst_lat + r * 128 + (((lane ^ r) & 7) << 4), src_lat + (int64_t)max(rid, 0) * (kMlaDqk * 2), rid >= 0 ? 16 : 0);
          }
          {
            const int r = w4 + (lane >> 2) * kG, rid = __shfl_sync(0xffffffffu, id, lane >> 2);
            if (lane < 4 * kRawRows && r < kMlaBlk)
              cp_async_16(dst + kMlaRopeOff + r * 64 + (((lane ^ (r >> 1)) & 3) << 4),
                          src_rope + (int64_t)max(rid, 0) * (kMlaDqk * 2), rid >= 0 ? 16 : 0);
          }
        }
        cp_async_arrive(&kv_full[kvb]);                // this thread's arrival, once its copies have landed ...
        __syncwarp();
        if (lane == 0) mbar_arrive(&kv_full[kvb]);     // ... and the warp's, for the validity bytes
        if (++kvb == NB) {
          kvb = 0;
          round ^= 1;
        }
      }
      cp_async_wait_all();                             // nothing of this thread's is in flight when it leaves
    } else {
      // Decode.  The same split of rows over the warps.  A warp keeps the raw rows of two blocks of its own in shared memory:
      // cp.async two blocks ahead (a cache row is a DRAM and often a TLB miss away, ~3000 cycles), then 8 e4m3 values per
      // lane and row through registers into the KV buffer.  The warps never wait for one another.  Positions travel four
      // blocks ahead, page-table entries three.
      constexpr int kRows = kRawRows;
      auto table_entry = [&](int pos) -> int {
        return (pos >= 0 && pos < a.S_kv) ? __ldg(a.block_table + (int64_t)t * a.table_stride + pos / kLatentPage) : -1;
      };
      auto cache_row = [&](int pos, int phys) -> int {   // -1 = empty slot; bad positions and page ids are flagged and skipped
        if (pos < 0) return -1;
        if (pos < a.S_kv && phys >= 0 && (int64_t)(phys + 1) * kLatentPage <= a.num_phys_rows)
          return phys * kLatentPage + pos % kLatentPage;
        if (a.status) atomicCAS(a.status, kStatusOk, kStatusBadIndex);
        return -1;
      };
      auto stage_of = [&](int blk) -> uint8_t* {       // the fifth KV buffer, and what does not fit there behind everything else
        const int c = (blk & 1) * kG + w4;
        return c < kRawInBuf ? kv_s + NB * kMlaKBytes + c * kRawBytes : smem + kMlaSmemBytes + (c - kRawInBuf) * kRawBytes;
      };
      const uint8_t* src_lat = a.cache + cta * kMlaDvHalf + (lane & 15) * 16;
      const uint8_t* src_rope = a.cache + kMlaDv + 16 + cta * 64 + (lane & 3) * 16;
      // request the warp's rows of a block; an empty slot is zero-filled, values and scales
      auto fetch = [&](int blk, int id) {
        uint8_t* st = stage_of(blk);
#pragma unroll
        for (int u = 0; u < kRows / 2; ++u) {          // two rows of 256 values per instruction
          const int j = 2 * u + (lane >> 4), rid = __shfl_sync(0xffffffffu, id, j);
          cp_async_16(st + j * kRawRow + (lane & 15) * 16, src_lat + (int64_t)max(rid, 0) * kLatentTokenBytes, rid >= 0 ? 16 : 0);
        }
        const int rid = __shfl_sync(0xffffffffu, id, lane >> 2);
        if (lane < kRows)                              // a row's four scales
          cp_async_16(st + lane * kRawRow + 256, a.cache + kMlaDv + (int64_t)max(id, 0) * kLatentTokenBytes, id >= 0 ? 16 : 0);
        if (lane < 4 * kRows)                          // this CTA's two K-steps of the rope panel: 64 bytes per row
          cp_async_16(st + (lane >> 2) * kRawRow + 272 + (lane & 3) * 16, src_rope + (int64_t)max(rid, 0) * kLatentTokenBytes, rid >= 0 ? 16 : 0);
        cp_async_commit();
      };
      // row ids of blocks i and i+1 (which of them are used), page-table entry and position of i+2, position of i+3
      int id_cur, id_nxt, pa, ta, pb;
      {
        const int p0 = slot_pos, p1 = load_pos(1);
        pa = load_pos(2);
        pb = load_pos(3);
        const int t0 = table_entry(p0), t1 = table_entry(p1);
        ta = table_entry(pa);
        id_cur = cache_row(p0, t0);
        fetch(0, id_cur);
        id_nxt = cache_row(p1, t1);
        fetch(1, id_nxt);
      }
      for (int i = 0; i < nblk; ++i) {
        const int kvb = i % NB;
        const int id2 = cache_row(pa, ta);             // block i+2
        pa = pb;
        ta = table_entry(pa);
        pb = load_pos(i + 4);
        if (i == kQBuf0) ok = mla_wait(q_moved, 0, abort_flag, a.status);   // from here on the buffers held Q
        if (i >= NB) ok = mla_wait(&kv_free[kvb], ((i / NB) - 1) & 1, abort_flag, a.status);
        if (!ok) break;
        mark(i, id_cur >= 0);
        id_cur = id_nxt;
        id_nxt = id2;
        cp_async_wait<1>();                            // this lane's copies of block i have landed (block i+1 may be in flight) ...
        __syncwarp();                                  // ... and the other lanes'
        const uint8_t* st = stage_of(i);
        uint8_t* dst = kv_s + kvb * kMlaKBytes;
        uint8_t* dst_lat = dst + (lane >> 3) * kMlaKPanelBytes;
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          const int r = w4 + j * kG;
          const uint2 raw = *reinterpret_cast<const uint2*>(st + j * kRawRow + lane * 8);
          const float sc = *reinterpret_cast<const float*>(st + j * kRawRow + 256 + cta * 8 + (lane >> 4) * 4);
          const uint4 v = e4m3x8_to_bf16(raw, sc);
          if (r < kMlaBlk) *reinterpret_cast<uint4*>(dst_lat + r * 128 + (((lane ^ r) & 7) << 4)) = v;
        }
        {
          const int r = w4 + (lane >> 2) * kG;
          if (lane < 4 * kRows && r < kMlaBlk)
            *reinterpret_cast<uint4*>(dst + kMlaRopeOff + r * 64 + (((lane ^ (r >> 1)) & 3) << 4)) =
                *reinterpret_cast<const uint4*>(st + (lane >> 2) * kRawRow + 272 + (lane & 3) * 16);
        }
        __syncwarp();                                  // (the MMA warp makes the writes visible to the tensor core's reads)
        if (lane == 0) mbar_arrive(&kv_full[kvb]);
        fetch(i + 2, id2);                             // into the stage just read: what was loaded from it has been stored
      }
      cp_async_wait_all();                             // nothing of this thread's is in flight when it leaves
    }
  } else {
    // ------------- partial-score exchange, softmax and output: thread = (head, half of a block's keys) -------------
    const int qd = warp & 3, hf = (warp >> 2) & 1, set = warp >> 3;      // hf: key half; set: takes the blocks of that parity
    const int row = qd * 32 + lane;                    // head = TMEM lane
    const uint32_t t_row = tmem + (uint32_t(qd * 32) << 16);
    const uint32_t peer_xchg_free = mapa_u32(smem_u32(xchg_free + warp), peer);
    const uint32_t peer_recv_full = mapa_u32(smem_u32(recv_full + warp), peer);
    float m = -CUDART_INF_F, l = 0.f;                  // m: reference of the last block seen; l: this thread's keys only
    bool ok = mla_wait(q_full, 0, abort_flag, a.status);
    if (ok) {
      // this head's row of the five Q panels, swizzled shared memory -> packed bf16 pairs in tensor memory: the ten
      // half-panels (64 B) are dealt to the four threads of the head
#pragma unroll 1
      for (int hp = warp >> 2; hp < 2 * kMlaPanels; hp += 4) {
        uint32_t qv[16];
        const uint8_t* src = q_stage(hp >> 1) + row * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 w = *reinterpret_cast<const uint4*>(src + ((((hp & 1) * 4 + c) ^ (row & 7)) << 4));
          qv[4 * c + 0] = w.x; qv[4 * c + 1] = w.y; qv[4 * c + 2] = w.z; qv[4 * c + 3] = w.w;
        }
        tmem_st16(t_row + kColQ + hp * 16, qv);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_moved);             // one arrival per warp: 512 arrivals on one barrier queue up
    }
    cluster_wait();
    // this warp's part of the set's partial tile: 32 heads x 32 keys, 2 KB
    const int xw = hf * 4 + qd;
    uint8_t* send = send_s + xw * kMlaXWarp;
    const uint8_t* recv = recv_s + xw * kMlaXWarp;
    const uint32_t peer_recv = mapa_u32(smem_u32(recv), peer);
    // block maxima, four blocks deep: a warp may be two blocks behind its partner, never four (P.V orders them)
    auto pm_of = [&](int blk) -> uint16_t* { return pm_s + (blk & 3) * 256 + row; };      // [key half][head]
    auto raise = [&](float m_old, float bmax) { return bmax - m_old > kMaxRaise ? bmax : m_old; };   // -inf - -inf: stays
    auto pair_max = [&](const uint16_t* pm) {
      return fmaxf(__uint_as_float(uint32_t(pm[0]) << 16), __uint_as_float(uint32_t(pm[128]) << 16));
    };
    if (qd < n_quad && set < nblk && lane == 0) mbar_expect_tx(&recv_full[warp], kMlaXWarp);
    for (int n = qd < n_quad ? set : nblk; n < nblk && ok; n += 2) {
      const uint32_t ph = (n >> 1) & 1;
      uint32_t sv[32];                                 // this CTA's partial scores
      ok = mla_wait(&s_full[set], ph, abort_flag, a.status);
      if (!ok) break;
      tc_fence_after();
      tmem_ld32(t_row + kColS + 32 * hf, sv);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);              // the next block's scores may overwrite S now
      if (n > 0) {                                     // the peer has read block n-1: both stages are free
        ok = mla_wait(&xchg_free[warp ^ 8], ((n - 1) >> 1) & 1, abort_flag, a.status);
        if (!ok) break;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        auto h2 = [&](int k) { return pack_f16x2(__uint_as_float(sv[8 * c + 2 * k]), __uint_as_float(sv[8 * c + 2 * k + 1])); };
        *reinterpret_cast<uint4*>(send + xchg_off(lane, c)) = make_uint4(h2(0), h2(1), h2(2), h2(3));
      }
      fence_async_smem();                              // the bulk copy reads the tile through the async proxy
      __syncwarp();
      if (elect_one()) bulk_copy_to_peer(peer_recv, send, kMlaXWarp, peer_recv_full);
      __syncwarp();
      // the reference of the block before, from that block's maxima: every thread follows the whole sequence by itself
      if (n > 0) {
        ok = mla_wait(&pm_full[(set ^ 1) * 4 + qd], ((n - 1) >> 1) & 1, abort_flag, a.status);
        if (!ok) break;
      }
      const float m_own = m;                           // what l is relative to
      if (n > 0) m = raise(m, pair_max(pm_of(n - 1)));
      const float m_prev = m;
      ok = mla_wait(&recv_full[warp], ph, abort_flag, a.status);
      if (!ok) break;
      float s[32];                                     // raw scores; the (positive) scale is folded into the exponent's FMA
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 theirs = *reinterpret_cast<const uint4*>(recv + xchg_off(lane, c));
        const uint32_t tw[4] = {theirs.x, theirs.y, theirs.z, theirs.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          add_f16x2(tw[k], __uint_as_float(sv[8 * c + 2 * k]), __uint_as_float(sv[8 * c + 2 * k + 1]), s[8 * c + 2 * k], s[8 * c + 2 * k + 1]);
        }
      }
      const uint32_t used = __ballot_sync(0xffffffffu, valid_s[(n % kMlaValidRing) * kMlaBlk + 32 * hf + lane]);
      auto largest = [&]() {
        float bm[4] = {s[0], s[1], s[2], s[3]};        // four independent chains
#pragma unroll
        for (int i = 4; i < 32; ++i) bm[i & 3] = fmaxf(bm[i & 3], s[i]);
        return fmaxf(fmaxf(bm[0], bm[1]), fmaxf(bm[2], bm[3]));
      };
      const float top = largest();                     // of every value of the tile, used or not
      float bmax = top;
      if (used != 0xffffffffu) {                       // empty slots (the tail of a short row, holes): warp-uniform
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = (used >> i) & 1u ? s[i] : -CUDART_INF_F;
        bmax = largest();
      }
      pm_of(n)[hf * 128] = static_cast<uint16_t>(bf16_bits_round_up(bmax * a.scale_log2e));
      __syncwarp();
      if (lane == 0) mbar_arrive(&pm_full[set * 4 + qd]);
      mbar_arrive_remote_after(peer_xchg_free, top, lane == 0);      // the peer may send into this stage again
      if (lane == 0 && n + 2 < nblk) mbar_expect_tx(&recv_full[warp], kMlaXWarp);
      ok = mla_wait(&pm_full[set * 4 + qd], ph, abort_flag, a.status);
      if (!ok) break;
      m = raise(m_prev, pair_max(pm_of(n)));
      if (m != m_own) l = m_own == -CUDART_INF_F ? 0.f : l * fast_exp2(m_own - m);
      bool waited_pv = n == 0;
      if (__any_sync(0xffffffffu, m != m_prev) && n > 0) {
        // O must be quiescent: P.V of the previous block has to be complete.  This thread scales its half of the columns.
        ok = mla_wait(&pv_done[set ^ 1], ((n - 1) >> 1) & 1, abort_flag, a.status);
        if (!ok) break;
        waited_pv = true;
        tc_fence_after();
        const float alpha = m != m_prev ? fast_exp2(m_prev - m) : 1.f;
#pragma unroll 1
        for (int c = hf * (kMlaDvHalf / 2); c < (hf + 1) * (kMlaDvHalf / 2); c += 16) {
          uint32_t ov[16];
          tmem_ld16(t_row + kColO + c, ov);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
          tmem_st16(t_row + kColO + c, ov);
        }
      }
      const float m_eff = (m == -CUDART_INF_F) ? 0.f : m;
      uint32_t pk[16];
      const uint64_t scale2 = pack_f32x2(a.scale_log2e, a.scale_log2e), m2 = pack_f32x2(-m_eff, -m_eff);
      float ps[4] = {0.f, 0.f, 0.f, 0.f};              // sums of the even and odd keys, two chains each
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float x0, x1;
        unpack_f32x2(fma_f32x2(pack_f32x2(s[i], s[i + 1]), scale2, m2), x0, x1);
        const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
        pk[i >> 1] = pack_bf16x2(p0, p1);
        add_bf16x2(pk[i >> 1], ps[i & 2], ps[(i & 2) + 1]);
      }
      l += (ps[0] + ps[1]) + (ps[2] + ps[3]);
      if (!waited_pv) {                                // P is single-buffered: P.V of the previous block must be done
        ok = mla_wait(&pv_done[set ^ 1], ((n - 1) >> 1) & 1, abort_flag, a.status);
        if (!ok) break;
        tc_fence_after();
      }
      tmem_st16(t_row + kColP + 16 * hf, pk);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok) cluster_arrive();                          // nothing remote is left to do for this warp: the others need not wait for its output
    left = ok;
    if (ok) ok = mla_wait(o_final, 0, abort_flag, a.status);
    // A full group of 128 heads leaves through shared memory and TMA stores: four [128 heads x 128 B] panels in the
    // (now idle) first two KV buffers, written asynchronously in whole lines.  16-byte stores from the threads -- every
    // lane its own 1 KB-strided row -- cost about 4 % of the kernel.
    const bool by_tma = a.tma_out && part < 0 && heads_here == 128;
    // the row sum over all keys: the four threads of a head add theirs, relative to the later reference, through the idle
    // third KV buffer (every warp comes to the barrier, whatever became of its waits)
    float2* sum_s = reinterpret_cast<float2*>(kv_s + 2 * kMlaKBytes);
    const int quarter = warp >> 2;                     // which quarter of the head's columns this thread writes
    if (ok) sum_s[quarter * 128 + row] = make_float2(m, l);
    named_bar_sync(3 + qd, 128);
    if (ok) {
      tc_fence_after();
      float mt = -CUDART_INF_F;
#pragma unroll
      for (int u = 0; u < 4; ++u) mt = fmaxf(mt, sum_s[u * 128 + row].x);
      l = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 ml = sum_s[u * 128 + row];
        if (ml.x != -CUDART_INF_F) l += ml.y * fast_exp2(ml.x - mt);
      }
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* orow = a.out + ((int64_t)t * a.H + hg * 128 + row) * kMlaDv + cta * kMlaDvHalf;
      const int64_t prow = (int64_t)part * a.H + hg * 128 + row;
      if (part >= 0 && quarter == 0 && row < heads_here)         // what this CTA's half of the columns is weighted with
        a.part_lse[((int64_t)part * 2 + cta) * a.H + hg * 128 + row] = l > 0.f ? mt + log2f(l) : -CUDART_INF_F;
#pragma unroll 1
      for (int c = quarter * (kMlaDvHalf / 4); c < (quarter + 1) * (kMlaDvHalf / 4); c += 32) {
        uint32_t ov[32];
        tmem_ld32(t_row + kColO + c, ov);
        tmem_wait_ld();
        if (by_tma) {
          uint8_t* prow_s = kv_s + (c >> 6) * kMlaQPanelBytes + row * 128;
          const int ch0 = (c & 63) >> 3;                 // first of this iteration's four 16-byte chunks in the 128-byte row
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(ov[i + 0]) * inv, __uint_as_float(ov[i + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(ov[i + 2]) * inv, __uint_as_float(ov[i + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(ov[i + 4]) * inv, __uint_as_float(ov[i + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(ov[i + 6]) * inv, __uint_as_float(ov[i + 7]) * inv);
            *reinterpret_cast<uint4*>(prow_s + (((ch0 + (i >> 3)) ^ (row & 7)) << 4)) = w;
          }
        } else if (row < heads_here && part >= 0) {
          float4* po = reinterpret_cast<float4*>(a.part_o + prow * kMlaDv + cta * kMlaDvHalf + c);
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            po[i >> 2] = make_float4(__uint_as_float(ov[i]) * inv, __uint_as_float(ov[i + 1]) * inv,
                                     __uint_as_float(ov[i + 2]) * inv, __uint_as_float(ov[i + 3]) * inv);
        } else if (row < heads_here) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(ov[i + 0]) * inv, __uint_as_float(ov[i + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(ov[i + 2]) * inv, __uint_as_float(ov[i + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(ov[i + 4]) * inv, __uint_as_float(ov[i + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(ov[i + 6]) * inv, __uint_as_float(ov[i + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c + i) = w;
          }
        }
      }
    }
    if (by_tma) {                                      // every softmax thread comes here, whatever became of its waits
      // a quarter of the columns is one panel and four warps: it leaves as soon as they have written it
      fence_async_smem();                              // the store below reads the panel through the async proxy
      named_bar_sync(7 + quarter, 128);
      if ((warp & 3) == 0 && elect_one() && !*abort_flag) {         // x in 4-byte units: 32 per 64-column panel
        tma_store_2d(&tmap_o, kv_s + quarter * kMlaQPanelBytes, (cta * 4 + quarter) * 32, t * a.H + hg * 128);
        bulk_commit_and_wait_read();                   // the panel has been read: the CTA may go
      }
    }
  }

  __syncwarp();
  if (warp >= kMlaSoftmaxWarps) cluster_wait();      // MMA and gather warps: the wait that pairs with the arrive above
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // a wait gave up: let the copies that may still be in flight into this CTA land (bounded) before its shared memory goes away
    if (threadIdx.x == 0)
      for (int w = 0; w < 64; ++w) __nanosleep(1000);
    __syncthreads();
  }
  if (!left) cluster_arrive();
  cluster_wait();                 // neither CTA leaves while the other may still copy into it or arrive on its barriers
  if (warp == kMlaMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, kMlaTmemCols);
  }
}

// out[t,h,:] = sum_s 2^(lse_s - M) o_s / sum_s 2^(lse_s - M): merges the parts of a split slot list, each half of the columns
// by the sums of the CTA that computed it.
// A query in eight parts: 4.8 us with loads behind the weights' loop, 3.6 so.
__global__ void __launch_bounds__(128) sparse_mla_combine_kernel(const MlaArgs a) {
  const float *lse = grid_wait(a.part_lse), *part = grid_wait(a.part_o);      // the second returns at once
  const int u = blockIdx.x, t = a.n_full + u, h = blockIdx.y;
  const int d = threadIdx.x * 4, cta = d / kMlaDvHalf;
  // every load is requested before any is used: a part's weight and values do not wait for one another
  float wgt[kMlaMaxParts];
  float4 v[kMlaMaxParts];
#pragma unroll
  for (int sp = 0; sp < kMlaMaxParts; ++sp) {
    const int64_t p = (int64_t)u * a.n_split + sp;
    wgt[sp] = sp < a.n_split ? lse[(p * 2 + cta) * a.H + h] : -CUDART_INF_F;
    v[sp] = sp < a.n_split ? *reinterpret_cast<const float4*>(part + (p * a.H + h) * kMlaDv + d) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float mx = -CUDART_INF_F, den = 0.f;
#pragma unroll
  for (int sp = 0; sp < kMlaMaxParts; ++sp) mx = fmaxf(mx, wgt[sp]);
#pragma unroll
  for (int sp = 0; sp < kMlaMaxParts; ++sp) {
    wgt[sp] = (mx == -CUDART_INF_F) ? 0.f : exp2f(wgt[sp] - mx);
    den += wgt[sp];
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int sp = 0; sp < kMlaMaxParts; ++sp) {
    acc.x += wgt[sp] * v[sp].x; acc.y += wgt[sp] * v[sp].y; acc.z += wgt[sp] * v[sp].z; acc.w += wgt[sp] * v[sp].w;
  }
  uint2 o;
  o.x = pack_bf16x2(acc.x * inv, acc.y * inv);
  o.y = pack_bf16x2(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(a.out + ((int64_t)t * a.H + h) * kMlaDv + d) = o;
}

int make_tmap_2d_bytes(CUtensorMap* m, const void* base, uint64_t rows, uint64_t inner_bytes, uint64_t row_pitch,
                       uint32_t box_bytes, uint32_t box_rows);

template <bool FP8_PAGED, bool OVERLAPPED>
static int launch_mla(const void* q, const void* kv, const MlaArgs& args, cudaStream_t stream) {
  if (args.T == 0 || args.H == 0) return DSA_OK;
  if (args.K > kMlaMaxK) return set_error(DSA_ERR_SHAPE, "sparse_mla: K (%d) exceeds %d", args.K, kMlaMaxK);
  MlaArgs a = args;
  CUtensorMap tq, to;
  int rc = make_tmap_2d_bytes(&tq, q, (uint64_t)a.T * a.H, kMlaDqk * 2, kMlaDqk * 2, 128, 128);
  if (rc) return rc;
  // the output as [T*H rows x 1024 B], stored one [128 heads x 128 B] panel at a time -- when there is a full group of
  // 128 heads, no split, and the tensor can be mapped (16-byte aligned)
  a.tma_out = 0;
  to = tq;
  if (a.n_full > 0 && a.H >= 128 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0) {
    if ((rc = make_tmap_2d_bytes(&to, a.out, (uint64_t)a.T * a.H, kMlaDv * 2, kMlaDv * 2, 128, 128))) return rc;
    a.tma_out = 1;
  }
  auto kern = sparse_mla_kernel<FP8_PAGED, OVERLAPPED>;
  constexpr int smem_bytes = FP8_PAGED ? kMlaSmemDecode : kMlaSmemBytes;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess)
    return set_error(DSA_ERR_CUDA, "sparse_mla: cannot raise dynamic shared memory to %d", smem_bytes);
  const int n_parts = a.T - a.n_full;
  const dim3 grid(2 * (a.n_full + n_parts * a.n_split), 1, (a.H + 127) / 128);
  launch_after(OVERLAPPED, kern, grid, kMlaThreads, smem_bytes, stream, tq, to, a);
  if (n_parts > 0) launch_after(OVERLAPPED, sparse_mla_combine_kernel, dim3(n_parts, a.H), 128, 0, stream, a);
  return check_launch("sparse_mla");
}

int sparse_mla_few_launch(const void* q, const void* kv, const int32_t* idx, void* out, int T, int H, int S_kv, int K,
                          float scale, int32_t* status, cudaStream_t stream);

int sparse_mla_prefill_launch(const void* q, const void* kv, const int32_t* idx, void* out, int T, int H, int S_kv,
                              int K, float scale, int32_t* status, cudaStream_t stream) {
  if (H <= 32) return sparse_mla_few_launch(q, kv, idx, out, T, H, S_kv, K, scale, status, stream);
  MlaArgs a{};
  a.kv = static_cast<const uint8_t*>(kv);
  a.idx = idx;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.T = T; a.H = H; a.K = K; a.S_kv = S_kv;
  a.scale_log2e = scale * 1.4426950408889634f;
  a.status = status;
  a.n_full = T;
  a.n_split = 1;
  return launch_mla<false, false>(q, kv, a, stream);
}

// A CTA pair per query fills the GPU in rounds of (SMs / 2 / head groups) queries; the last, partly filled round would
// take as long as a full one.  The queries of that round are cut into parts that share its pairs: as many as fit, at most
// eight, of at least 256 slots.  More parts than that lose: every part pays the set-up again and writes an fp32 partial
// output that the combine kernel reads back.  Batch 160 (two rounds and twelve queries in six parts each): 174 -> 156 us.
static int mla_pairs(int H) { return max(1, sm_count() / (2 * ((H + 127) / 128))); }
static int mla_parts_per_query(int rest, int pairs, int K) { return rest == 0 ? 1 : max(1, min(min(kMlaMaxParts, K / 256), pairs / rest)); }
static size_t mla_part_bytes(int H) { return (size_t)H * (kMlaDv + 2) * sizeof(float); }
// Enough for every batch of up to B queries.  The need of a batch goes up and down with the queries of its last round (128
// heads, 2048 slots, 148 SMs: 64 parts for 8 queries, 74 for 37, none for 38 or for 74), and a serving loop runs smaller
// batches in the buffer that it made for its largest.
size_t mla_decode_workspace_bytes(int B, int H, int K) {
  const int pairs = mla_pairs(H);
  int parts = 0;
  for (int rest = 1; rest < pairs && rest <= B; ++rest) {
    const int ns = mla_parts_per_query(rest, pairs, K);
    if (ns > 1) parts = max(parts, rest * ns);
  }
  return parts * mla_part_bytes(H);
}

int sparse_mla_decode_launch(const void* q, const void* cache, const int32_t* block_table, int64_t table_stride,
                             const int32_t* idx, void* out, int B, int H, int K, int num_pages, int max_ctx,
                             float scale, void* workspace, size_t workspace_bytes, int32_t* status, int overlapped,
                             cudaStream_t stream) {
  MlaArgs a{};
  const int pairs = mla_pairs(H), rest = B % pairs;
  int ns = mla_parts_per_query(rest, pairs, K);
  if (ns > 1) {                                        // a smaller workspace: as many parts as it holds
    const size_t fit = workspace ? workspace_bytes / mla_part_bytes(H) / rest : 0;
    if (fit < (size_t)ns) ns = fit > 1 ? (int)fit : 1;
  }
  a.n_full = B;
  a.n_split = 1;
  if (ns > 1) {
    a.n_full = B - rest;
    a.n_split = ns;
    a.part_o = static_cast<float*>(workspace);
    a.part_lse = a.part_o + (size_t)rest * ns * H * kMlaDv;
  }
  a.cache = static_cast<const uint8_t*>(cache);
  a.block_table = block_table;
  a.table_stride = table_stride;
  a.idx = idx;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.T = B; a.H = H; a.K = K; a.S_kv = max_ctx;
  a.num_phys_rows = num_pages * kLatentPage;
  a.scale_log2e = scale * 1.4426950408889634f;
  a.status = status;
  return overlapped ? launch_mla<true, true>(q, nullptr, a, stream) : launch_mla<true, false>(q, nullptr, a, stream);
}

}  // namespace dsa
