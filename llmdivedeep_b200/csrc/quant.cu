// Per-block FP8 e4m3 quantiser: one kernel for what the reference does with about eight eager
// torch kernels (sparse_attn/DSA.py:102-132): fp32 absmax over each block of 64 or 128 values,
// scale = max(absmax, 1e-6) / 448, q = x / scale rounded to e4m3.  Both divisions are IEEE
// round-to-nearest, so the bytes and scales equal the reference's CPU result exactly.
// 2 (bf16) or 4 (fp32) bytes read and 1 byte + 4/block written per value.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "dsa_common.cuh"
#include "dsa_host.h"

namespace dsa {

// V (4, 8 or 16) consecutive values per thread, in loads of 16 bytes (4 bf16 values: 8).
template <int V, typename T>
__device__ __forceinline__ void load_values(const T* __restrict__ src, float (&v)[V]) {
  if constexpr (sizeof(T) == 2) {
    uint32_t w[V / 2];
    if constexpr (V == 4) {
      const uint2 raw = __ldg(reinterpret_cast<const uint2*>(src));
      w[0] = raw.x; w[1] = raw.y;
    } else {
#pragma unroll
      for (int h = 0; h < V / 8; ++h) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src) + h);
        w[4 * h] = raw.x; w[4 * h + 1] = raw.y; w[4 * h + 2] = raw.z; w[4 * h + 3] = raw.w;
      }
    }
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {                  // bf16 -> fp32: the value is the upper half of the word
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else {
#pragma unroll
    for (int h = 0; h < V / 4; ++h) {
      const float4 raw = __ldg(reinterpret_cast<const float4*>(src) + h);
      v[4 * h] = raw.x; v[4 * h + 1] = raw.y; v[4 * h + 2] = raw.z; v[4 * h + 3] = raw.w;
    }
  }
}
// The scale of the block that LANES neighbouring lanes hold, and this thread's V values as e4m3.
template <int LANES, int V>
__device__ __forceinline__ float quant_values(const float (&v)[V], uint32_t (&w)[V / 4]) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float sc = __fdiv_rn(fmaxf(amax, 1e-6f), 448.f);
#pragma unroll
  for (int i = 0; i < V / 4; ++i) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(__fdiv_rn(v[4 * i], sc), __fdiv_rn(v[4 * i + 1], sc)), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(__fdiv_rn(v[4 * i + 2], sc), __fdiv_rn(v[4 * i + 3], sc)), __NV_SATFINITE, __NV_E4M3);
    w[i] = lo | (hi << 16);
  }
  return sc;
}

// BLOCK / V threads per block of BLOCK values.  V = 16: three (two) shuffle steps instead of five, 16 bytes per load and
// store; bound by issue (the IEEE divisions).  [32768, 64, 128] bf16: 253 us with one warp per block and 8-byte loads, 176 us so
// (4.6 TB/s).  V = 4 for calls that are over in two or three microseconds: a thread's sixteen divisions in a row are then what
// takes the time (100 blocks of 128 bf16 values 1.65 us, 1.9 with V = 16; 4800 blocks of fp32 2.3 and 2.6, of bf16 2.35 and 2.2).
template <typename T, int BLOCK, int V>
__global__ void __launch_bounds__(256) fp8_quant_kernel(const T* __restrict__ x, int64_t n_blocks,
                                                        uint8_t* __restrict__ q, float* __restrict__ scale, const int q_aligned) {
  constexpr int LANES = BLOCK / V;
  const int64_t n = n_blocks * LANES, stride = (int64_t)gridDim.x * blockDim.x;
  // whole warps stay together for the shuffles: the loop runs over warps' first threads
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const int64_t i = i0 + (threadIdx.x & 31);
    float v[V];
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = 1.f;            // lanes past the end: dividing zeros takes the slow way, 2 us for the warp
    if (i < n) load_values<V>(x + i * V, v);
    uint32_t w[V / 4];
    const float sc = quant_values<LANES, V>(v, w);
    if (i < n) {
      uint32_t* o = reinterpret_cast<uint32_t*>(q) + i * (V / 4);
      if constexpr (V == 4) {
        *o = w[0];
      } else if (q_aligned) {
        *reinterpret_cast<uint4*>(o) = make_uint4(w[0], w[1], w[2], w[3]);
      } else {                                         // the caller's q starts on a 4-byte boundary only
        o[0] = w[0]; o[1] = w[1]; o[2] = w[2]; o[3] = w[3];
      }
      if (i % LANES == 0) scale[i / LANES] = sc;
    }
  }
}

// Latent rows [N, 576] -> records of the paged FP8 latent cache, 656 bytes each: 512 e4m3 values, their four fp32 scales
// (one per 128 values, the quantiser above), 64 bf16 rope values.  One warp per token: a lane quantises 16 latent values,
// lanes 0-7 carry eight rope values each.  Reads every row once and writes every record once, in 16-byte pieces; what it
// takes the place of was a strided copy, the quantiser and three strided copies into the records.
// 131072 tokens: 406 us -> 53 us (237 MB, 4.5 TB/s); 8192 tokens: 33.7 us -> 4.8 us on the device.
template <typename T>
__global__ void __launch_bounds__(256) pack_latent_kernel(const T* __restrict__ kv, int64_t row_stride, int64_t n,
                                                          uint8_t* __restrict__ rec) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < n; t += warps) {
    const T* src = kv + t * row_stride;
    uint8_t* dst = rec + t * 656;
    uint4 rope;
    if (lane < 8) {
      if constexpr (sizeof(T) == 2) {
        rope = __ldg(reinterpret_cast<const uint4*>(src + 512) + lane);
      } else {
        const float4 a = __ldg(reinterpret_cast<const float4*>(src + 512) + 2 * lane), b = __ldg(reinterpret_cast<const float4*>(src + 512) + 2 * lane + 1);
        const __nv_bfloat162 p[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w), __floats2bfloat162_rn(b.x, b.y), __floats2bfloat162_rn(b.z, b.w)};
        rope = *reinterpret_cast<const uint4*>(p);
      }
    }
    float v[16];
    load_values<16>(src + lane * 16, v);
    uint32_t w[4];
    const float sc = quant_values<8, 16>(v, w);
    reinterpret_cast<uint4*>(dst)[lane] = make_uint4(w[0], w[1], w[2], w[3]);
    if ((lane & 7) == 0) reinterpret_cast<float*>(dst + 512)[lane >> 3] = sc;
    if (lane < 8) reinterpret_cast<uint4*>(dst + 528)[lane] = rope;
  }
}

// RoPE on the first `rope_dim` values of every head row, then the quantiser above, in one pass over a bf16
// tensor whose rows are one FP8 block each (head_dim = BLOCK): what DsaIndexer.forward does between its
// projections and the scorer (sparse_attn/DSA.py:513-524, 530-531) with a dozen eager kernels and an fp32
// intermediate four times the size of the input.  The arithmetic keeps the reference's order and roundings,
// so the bytes and scales equal those of the eager chain:
//   NeoX form (halves):   y[i] = x[i] c - x[i+h] s,  y[i+h] = x[i] s + x[i+h] c   in fp32, each product and the
//                         sum rounded separately (separate torch ops: no fused multiply-add), NOT rounded to bf16;
//   interleaved (GPT-J):  the same on (even, odd) pairs, result rounded to bf16 (the reference writes it into a
//                         tensor of x's dtype).
// Row r belongs to position r / rows_per_pos (query rows: heads per token; key rows: 1).  One warp per row.
// With `gate`, the head gates of the rows become the scorer's weights on the way: ((float(gate) * mul0) * scale) * mul1, every
// product rounded as the eager chain rounds it (sparse_attn/DSA.py:327-331, 505-511).
constexpr int kRopeV = 8;                              // values per thread of the wide form
struct RopeGate {
  const __nv_bfloat16* gate;                           // [n_rows], or null
  float* out;
  float mul0, mul1;
  __device__ __forceinline__ float fold(int64_t row, float scale) const {
    return __fmul_rn(__fmul_rn(__fmul_rn(__bfloat162float(gate[row]), mul0), scale), mul1);
  }
};
template <int BLOCK, bool INTERLEAVE>
__global__ void __launch_bounds__(256) rope_fp8_quant_kernel(const __nv_bfloat16* __restrict__ x, int64_t n_rows, int rope_dim,
                                                             int rows_per_pos, const float* __restrict__ cos_t,
                                                             const float* __restrict__ sin_t, uint8_t* __restrict__ q,
                                                             float* __restrict__ scale, const RopeGate g) {
  constexpr int PER = BLOCK / 32;
  const int lane = threadIdx.x & 31;
  const int half = rope_dim >> 1;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < n_rows; b += warps) {
    const __nv_bfloat16* src = x + b * BLOCK + lane * PER;
    float v[PER];
    if constexpr (PER == 4) {
      const uint2 raw = __ldg(reinterpret_cast<const uint2*>(src));
      const __nv_bfloat162 p0 = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
      const __nv_bfloat162 p1 = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
      v[0] = __low2float(p0); v[1] = __high2float(p0); v[2] = __low2float(p1); v[3] = __high2float(p1);
    } else {
      const __nv_bfloat162 p0 = *reinterpret_cast<const __nv_bfloat162*>(src);
      v[0] = __low2float(p0); v[1] = __high2float(p0);
    }
    const int64_t pos = static_cast<uint32_t>(b) / static_cast<uint32_t>(rows_per_pos);      // 2^32 rows do not fit the device's memory
    const float* cr = cos_t + pos * half;
    const float* sr = sin_t + pos * half;
    const int d0 = lane * PER;                          // first dim of this lane
    if constexpr (INTERLEAVE) {
      if (d0 < rope_dim) {
#pragma unroll
        for (int i = 0; i < PER; i += 2) {
          const float c = __ldg(cr + ((d0 + i) >> 1)), s = __ldg(sr + ((d0 + i) >> 1));
          const float e = __fsub_rn(__fmul_rn(v[i], c), __fmul_rn(v[i + 1], s));
          const float o = __fadd_rn(__fmul_rn(v[i], s), __fmul_rn(v[i + 1], c));
          v[i] = __bfloat162float(__float2bfloat16_rn(e));
          v[i + 1] = __bfloat162float(__float2bfloat16_rn(o));
        }
      }
    } else {
      // partner lane holds the other half of the pair (half / PER lanes away); every lane takes part in the shuffle
      const int shift = half / PER;
      float other[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) other[i] = __shfl_xor_sync(0xffffffffu, v[i], shift);
      if (d0 < rope_dim) {
        const bool first = d0 < half;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int t = first ? d0 + i : d0 + i - half;
          const float c = __ldg(cr + t), s = __ldg(sr + t);
          v[i] = first ? __fsub_rn(__fmul_rn(v[i], c), __fmul_rn(other[i], s))      // x1 c - x2 s
                       : __fadd_rn(__fmul_rn(other[i], s), __fmul_rn(v[i], c));     // x1 s + x2 c
        }
      }
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float sc = __fdiv_rn(fmaxf(amax, 1e-6f), 448.f);
    uint32_t packed = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      packed |= (uint32_t)__nv_cvt_float_to_fp8(__fdiv_rn(v[i], sc), __NV_SATFINITE, __NV_E4M3) << (8 * i);
    if constexpr (PER == 4) {
      reinterpret_cast<uint32_t*>(q + b * BLOCK)[lane] = packed;
    } else {
      reinterpret_cast<uint16_t*>(q + b * BLOCK)[lane] = (uint16_t)packed;
    }
    if (lane == 0) {
      scale[b] = sc;
      if (g.gate) g.out[b] = g.fold(b, sc);
    }
  }
}

// The same with eight values per thread, BLOCK / 8 threads per row: 16-byte loads, fewer shuffle steps.  [3000, 64, 128] 41.1 us with a
// warp per row, 31.0 so (the quantiser alone 16.2).  Sixteen values, as that one has them, need 78 registers here: no faster.
template <int BLOCK, bool INTERLEAVE>
__global__ void __launch_bounds__(256) rope_fp8_quant_wide_kernel(const __nv_bfloat16* __restrict__ x, int64_t n_rows, int rope_dim,
                                                                  int rows_per_pos, const float* __restrict__ cos_t,
                                                                  const float* __restrict__ sin_t, uint8_t* __restrict__ q,
                                                                  float* __restrict__ scale, const RopeGate g) {
  constexpr int V = kRopeV, LANES = BLOCK / V;
  const int lane = threadIdx.x & 31, half = rope_dim >> 1;
  const int d0 = (lane & (LANES - 1)) * V;             // first dim of this lane
  const bool rotated = d0 < rope_dim, first = d0 < half;
  const int64_t n = n_rows * LANES, stride = (int64_t)gridDim.x * blockDim.x;
  // whole warps stay together for the shuffles: the loop runs over warps' first threads
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const int64_t i = i0 + lane, row = i / LANES;
    float v[V];
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = 1.f;            // lanes past the end: dividing zeros takes the slow way
    if (i < n) load_values<V>(x + i * V, v);
    const int64_t pos = i < n ? static_cast<uint32_t>(row) / static_cast<uint32_t>(rows_per_pos) : 0;
    if constexpr (INTERLEAVE) {
      if (rotated) {
#pragma unroll
        for (int j = 0; j < V; j += 2) {
          const float c = __ldg(cos_t + pos * half + ((d0 + j) >> 1)), s = __ldg(sin_t + pos * half + ((d0 + j) >> 1));
          const float e = __fsub_rn(__fmul_rn(v[j], c), __fmul_rn(v[j + 1], s));
          const float o = __fadd_rn(__fmul_rn(v[j], s), __fmul_rn(v[j + 1], c));
          v[j] = __bfloat162float(__float2bfloat16_rn(e));
          v[j + 1] = __bfloat162float(__float2bfloat16_rn(o));
        }
      }
    } else {
      // the other half of the pair is half / V lanes away; every lane takes part in the shuffle
      float c[V], s[V];
      const float4* cr = reinterpret_cast<const float4*>(cos_t + pos * half + (first ? d0 : d0 - half));
      const float4* sr = reinterpret_cast<const float4*>(sin_t + pos * half + (first ? d0 : d0 - half));
#pragma unroll
      for (int j = 0; j < V; j += 4) {
        const float4 c4 = rotated ? __ldg(cr + j / 4) : make_float4(1.f, 1.f, 1.f, 1.f), s4 = rotated ? __ldg(sr + j / 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        c[j] = c4.x; c[j + 1] = c4.y; c[j + 2] = c4.z; c[j + 3] = c4.w;
        s[j] = s4.x; s[j + 1] = s4.y; s[j + 2] = s4.z; s[j + 3] = s4.w;
      }
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, v[j], half / V);
        const float s1 = first ? -s[j] : s[j];         // x1 c - x2 s and x2 c + x1 s: the same roundings
        if (rotated) v[j] = __fadd_rn(__fmul_rn(v[j], c[j]), __fmul_rn(other, s1));
      }
    }
    uint32_t w[V / 4];
    const float sc = quant_values<LANES, V>(v, w);
    if (i < n) {
      *reinterpret_cast<uint2*>(q + i * V) = make_uint2(w[0], w[1]);
      if ((lane & (LANES - 1)) == 0) {
        scale[row] = sc;
        if (g.gate) g.out[row] = g.fold(row, sc);
      }
    }
  }
}

int rope_fp8_quant_launch(const void* x, int64_t n_rows, int head_dim, int rope_dim, int interleave, int rows_per_pos,
                          const float* cos_t, const float* sin_t, void* q, float* scale, const void* gate, float mul0,
                          float mul1, float* gate_out, cudaStream_t stream) {
  if (n_rows == 0) return DSA_OK;
  if (head_dim != 64 && head_dim != 128) return set_error(DSA_ERR_SHAPE, "rope_fp8_quant: head dim %d not supported (64 or 128)", head_dim);
  const __nv_bfloat16* xi = static_cast<const __nv_bfloat16*>(x);
  uint8_t* qo = static_cast<uint8_t*>(q);
  const RopeGate g{static_cast<const __nv_bfloat16*>(gate), gate_out, mul0, mul1};
  // Eight values a thread where the rotated part is made of whole threads (whole pairs of them), the addresses allow its accesses
  // and the call is not over in two microseconds anyway (a thread's divisions in a row are then what takes the time).
  const bool wide = rope_dim % (interleave ? kRopeV : 2 * kRopeV) == 0 && n_rows * (head_dim / kRopeV) >= (int64_t)sm_count() * 512 &&
                    ((reinterpret_cast<uintptr_t>(q) & 7) | ((reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15)) == 0;
  const int64_t want = wide ? (n_rows * (head_dim / kRopeV) + 255) / 256 : (n_rows + 7) / 8, most = (int64_t)sm_count() * 16;
  const int grid = (int)(want < most ? want : most);
#define DSA_ROPE_CASE(K, B, I) K<B, I><<<grid, 256, 0, stream>>>(xi, n_rows, rope_dim, rows_per_pos, cos_t, sin_t, qo, scale, g)
#define DSA_ROPE_CASES(K)                                     \
  if (head_dim == 128 && interleave) DSA_ROPE_CASE(K, 128, true); \
  else if (head_dim == 128) DSA_ROPE_CASE(K, 128, false);     \
  else if (interleave) DSA_ROPE_CASE(K, 64, true);            \
  else DSA_ROPE_CASE(K, 64, false)
  if (wide) {
    DSA_ROPE_CASES(rope_fp8_quant_wide_kernel);
  } else {
    DSA_ROPE_CASES(rope_fp8_quant_kernel);
  }
#undef DSA_ROPE_CASES
#undef DSA_ROPE_CASE
  return check_launch("rope_fp8_quant");
}

template <typename T, int BLOCK>
static void launch_fp8_quant(const void* x, int64_t n_blocks, void* q, float* scale, cudaStream_t stream) {
  const int al = (reinterpret_cast<uintptr_t>(q) & 15) == 0;
  const bool small = n_blocks * (BLOCK / 16) < (int64_t)sm_count() * (sizeof(T) == 2 ? 256 : 512);
  const int64_t want = (n_blocks * (BLOCK / (small ? 4 : 16)) + 255) / 256, most = (int64_t)sm_count() * 16;
  const int grid = (int)(want < most ? want : most);
  const T* xt = static_cast<const T*>(x);
  uint8_t* qt = static_cast<uint8_t*>(q);
  if (small) fp8_quant_kernel<T, BLOCK, 4><<<grid, 256, 0, stream>>>(xt, n_blocks, qt, scale, al);
  else fp8_quant_kernel<T, BLOCK, 16><<<grid, 256, 0, stream>>>(xt, n_blocks, qt, scale, al);
}

int fp8_quant_launch(const void* x, int x_is_bf16, int64_t n_blocks, int block, void* q, float* scale,
                     cudaStream_t stream) {
  if (n_blocks == 0) return DSA_OK;
  if (block == 128 && x_is_bf16) launch_fp8_quant<__nv_bfloat16, 128>(x, n_blocks, q, scale, stream);
  else if (block == 128) launch_fp8_quant<float, 128>(x, n_blocks, q, scale, stream);
  else if (block == 64 && x_is_bf16) launch_fp8_quant<__nv_bfloat16, 64>(x, n_blocks, q, scale, stream);
  else if (block == 64) launch_fp8_quant<float, 64>(x, n_blocks, q, scale, stream);
  else return set_error(DSA_ERR_SHAPE, "fp8_quant: block size %d not supported (64 or 128)", block);
  return check_launch("fp8_quant");
}

int pack_latent_launch(const void* kv, int kv_is_bf16, int64_t row_stride, int64_t n, void* rec, cudaStream_t stream) {
  if (n == 0) return DSA_OK;
  const int64_t want = (n + 7) / 8;
  const int grid = (int)(want < (int64_t)sm_count() * 16 ? want : (int64_t)sm_count() * 16);
  if (kv_is_bf16)
    pack_latent_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(kv), row_stride, n, static_cast<uint8_t*>(rec));
  else
    pack_latent_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(kv), row_stride, n, static_cast<uint8_t*>(rec));
  return check_launch("pack_latent");
}

}  // namespace dsa
