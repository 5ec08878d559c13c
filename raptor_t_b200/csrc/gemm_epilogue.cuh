// Shared epilogue of the tcgen05 GEMM kernels: one thread owns one accumulator row (TMEM
// lane), walks its 32-column chunks (tcgen05.ld), applies bias / GELU / the QKV scatter and
// stores 64 bytes per chunk with two 256-bit stores.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.h"
#include "sm100_ptx.cuh"

namespace rt {
namespace gemm_detail {

using namespace ptx;

__device__ __forceinline__ float gelu_tanh_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return 0.5f * x * (1.0f + t);
}

// tanh-form GELU of two values with packed fp32x2 arithmetic (half the issue slots):
//   u = x * (k0 + k1 x^2),  gelu = 0.5 x + 0.5 x tanh(u)
__device__ __forceinline__ void gelu_tanh_f2(float& x0, float& x1) {
  unsigned long long x, x2, u, k0, k1, h;
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(x0), "f"(x1));
  asm("mov.b64 %0, {%1, %1};" : "=l"(k0) : "f"(0.7978845608028654f));
  asm("mov.b64 %0, {%1, %1};" : "=l"(k1) : "f"(0.7978845608028654f * 0.044715f));
  asm("mov.b64 %0, {%1, %1};" : "=l"(h) : "f"(0.5f));
  asm("mul.rn.f32x2 %0, %1, %1;" : "=l"(x2) : "l"(x));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(u) : "l"(x2), "l"(k1), "l"(k0));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(u) : "l"(u), "l"(x));
  float u0, u1, t0, t1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(u0), "=f"(u1) : "l"(u));
  asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(u0));
  asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(u1));
  unsigned long long t, hx, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(t) : "f"(t0), "f"(t1));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(hx) : "l"(x), "l"(h));
  asm("fma.rn.f32x2 %0, %1, %2, %1;" : "=l"(r) : "l"(hx), "l"(t));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(r));
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}
template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (BF16) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  } else {
    return __half22float2(*reinterpret_cast<__half2*>(&w));
  }
}

// Extra arguments of the QKV epilogue: the [T][3H] result is never written; each
// 64-wide head slice of a row goes, with bias added (and the query scaled), straight to
// the per-sequence head-major q / k / v buffers the attention kernel reads
// (row (seq_first_token*heads + head*seq_len + token_in_seq) of a [T*heads][64] matrix).
struct QkvEpilogue {
  const uint16_t* residual;  // RT_EPI_BIAS_RESIDUAL: [M][N], added after the bias
  uint16_t* q;
  uint16_t* k;
  uint16_t* v;
  const int2* block_seq;  // per packed 64-token block: {first token of its sequence, sequence length}
  int heads;
  float q_scale;
  int splits;  // kEpiPartial: parts of K
  bool settled_w;  // nothing in flight writes W: a kernel may read it before the kernels before it have ended
};
constexpr int kEpiQkv = 3;
// Split-K form: C is fp32 [splits][M][N], part s holds the sum over its K range; no bias.  The reader of the
// parts (layernorm_parts_kernel) adds them up.
constexpr int kEpiPartial = 5;

// COLS columns, from `col` on, of one accumulator row: r[] holds the fp32 accumulators, o[] gets the 16-bit results.
template <bool BF16, int EPI, int COLS = 32>
__device__ __forceinline__ void epilogue_values(const uint32_t* r, uint32_t* o, int col, int row, int M, int N,
                                                const uint16_t* __restrict__ bias, const QkvEpilogue& qkv) {
  if constexpr (EPI == RT_EPI_NONE) {
#pragma unroll
    for (int j = 0; j < COLS / 2; ++j) o[j] = pack2<BF16>(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
  } else {
    uint32_t res[COLS / 2];
    if constexpr (EPI == RT_EPI_BIAS_RESIDUAL) {
      if (row < M) {
        const uint4* rp = reinterpret_cast<const uint4*>(qkv.residual + static_cast<size_t>(row) * N + col);
#pragma unroll
        for (int q = 0; q < COLS / 8; ++q) {
          const uint4 t = rp[q];
          res[4 * q] = t.x;
          res[4 * q + 1] = t.y;
          res[4 * q + 2] = t.z;
          res[4 * q + 3] = t.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < COLS / 2; ++q) res[q] = 0u;
      }
    }
    const uint4* bv = reinterpret_cast<const uint4*>(bias + col);
#pragma unroll
    for (int q = 0; q < COLS / 8; ++q) {
      const uint4 b4 = __ldg(bv + q);
      const uint32_t bw[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 bb = unpack2<BF16>(bw[j]);
        float x0 = __uint_as_float(r[q * 8 + 2 * j]) + bb.x;
        float x1 = __uint_as_float(r[q * 8 + 2 * j + 1]) + bb.y;
        if constexpr (EPI == RT_EPI_BIAS_GELU) gelu_tanh_f2(x0, x1);
        if constexpr (EPI == RT_EPI_BIAS_RESIDUAL) {
          const float2 rr = unpack2<BF16>(res[q * 4 + j]);
          x0 += rr.x;
          x1 += rr.y;
        }
        if constexpr (EPI == kEpiQkv) {
          if (col < qkv.heads * 64) {  // query part
            x0 *= qkv.q_scale;
            x1 *= qkv.q_scale;
          }
        }
        o[q * 4 + j] = pack2<BF16>(x0, x1);
      }
    }
  }
}

// The same, stored by the thread itself.  COLS = 8, 16 or 32: a group never straddles a head.
template <bool BF16, int EPI, int COLS = 32>
__device__ __forceinline__ void epilogue_chunk(const uint32_t* r, int col, int row, int M, int N,
                                               uint16_t* __restrict__ C, const uint16_t* __restrict__ bias,
                                               const QkvEpilogue& qkv) {
  if constexpr (EPI == kEpiPartial) {
    if (row < M) {
      float* dst = reinterpret_cast<float*>(C) + static_cast<size_t>(row) * N + col;
#pragma unroll
      for (int q = 0; q < COLS / 8; ++q) st_global_v8(dst + 8 * q, r + 8 * q);
    }
    return;
  }
  uint32_t o[COLS / 2];
  epilogue_values<BF16, EPI, COLS>(r, o, col, row, M, N, bias, qkv);
  if (row < M) {
    uint16_t* dst;
    if constexpr (EPI == kEpiQkv) {
      const int hidden = qkv.heads * 64;
      const int part = col / hidden;
      const int hcol = col - part * hidden;
      const int2 bs = __ldg(qkv.block_seq + (row >> 6));
      const size_t drow = static_cast<size_t>(bs.x) * qkv.heads + static_cast<size_t>(hcol >> 6) * bs.y + (row - bs.x);
      dst = (part == 0 ? qkv.q : part == 1 ? qkv.k : qkv.v) + drow * 64 + (hcol & 63);
    } else {
      dst = C + static_cast<size_t>(row) * N + col;
    }
    if constexpr (COLS == 8) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int q = 0; q < COLS / 16; ++q) st_global_v8(dst + 16 * q, o + 8 * q);
    }
  }
}

// Drains columns [32*c] for c = chunk0, chunk0+2, ... < width/32 of one accumulator row, two
// chunks per step so that the second TMEM load is in flight while the first chunk is processed.
//   taddr: TMEM address of column 0 of this thread's lane quarter; row: global output row.
template <bool BF16, int EPI>
__device__ __forceinline__ void epilogue_row(int width, uint32_t taddr, int row, int n0, int chunk0, int M, int N,
                                             uint16_t* __restrict__ C, const uint16_t* __restrict__ bias,
                                             const QkvEpilogue& qkv) {
  const int chunks = width / 32;
#pragma unroll 1
  for (int c = chunk0; c < chunks; c += 4) {
    uint32_t r0[32], r1[32];
    const bool two = c + 2 < chunks;
    tmem_ld32(taddr + c * 32, r0);
    if (two) tmem_ld32(taddr + (c + 2) * 32, r1);
    tc_wait_ld();
    epilogue_chunk<BF16, EPI>(r0, n0 + c * 32, row, M, N, C, bias, qkv);
    if (two) epilogue_chunk<BF16, EPI>(r1, n0 + (c + 2) * 32, row, M, N, C, bias, qkv);
  }
}

// The tile through shared memory and TMA stores: warp `set` of a lane quarter takes the 64-column chunks set, set + 2,
// ... of its 32 rows, writes them as 128-byte swizzled rows into its own 4 KB of `stage` and one lane stores
// the box (rows past the last of the tensor are clipped).  Full 128-byte lines leave the SM, where a thread's own
// 32-byte stores of a row each compete with the operand loads of the next tile.  20480 rows, K = 768: 3072 columns
// with GELU 79.8 -> 74.2 us, QKV 60.1 -> 57.0; 4096 rows: 19.3 -> 17.6 and 14.7 -> 13.7.  drained() is called once
// the accumulator has been read.
template <bool BF16, int EPI, typename F>
__device__ __forceinline__ void epilogue_tma(int width, uint32_t taddr, int row0, int lane, int n0, int set, int M,
                                             int N, const uint16_t* __restrict__ bias, const QkvEpilogue& qkv,
                                             uint8_t* stage, const CUtensorMap* map_c, const CUtensorMap* map_k,
                                             const CUtensorMap* map_v, F&& drained) {
  const int chunks = width / 64;
  const int row = row0 + lane;
  uint8_t* const line = stage + lane * 128;
  const int swz = lane & 7;
  if (set >= chunks) drained();
#pragma unroll 1
  for (int c = set; c < chunks; c += 2) {
    uint32_t r[64], o[32];
    tmem_ld32(taddr + c * 64, r);
    tmem_ld32(taddr + c * 64 + 32, r + 32);
    tc_wait_ld();
    if (c + 2 >= chunks) drained();
    const int col = n0 + c * 64;
    epilogue_values<BF16, EPI>(r, o, col, row, M, N, bias, qkv);
    epilogue_values<BF16, EPI>(r + 32, o + 16, col + 32, row, M, N, bias, qkv);
    if (lane == 0) tma_store_wait_read<0>();  // the previous box has left the staging buffer
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q)
      *reinterpret_cast<uint4*>(line + ((q ^ swz) << 4)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0 && row0 < M) {
      if constexpr (EPI == kEpiQkv) {
        // a chunk is one head, and 32 rows stay inside one 64-token block: one box of the head-major matrix
        const int hidden = qkv.heads * 64;
        const int part = col / hidden;
        const int2 bs = __ldg(qkv.block_seq + (row0 >> 6));
        const int drow = bs.x * qkv.heads + ((col - part * hidden) >> 6) * bs.y + (row0 - bs.x);
        tma_store_2d(part == 0 ? map_c : part == 1 ? map_k : map_v, stage, 0, drow);
      } else {
        tma_store_2d(map_c, stage, col, row0);
      }
      tma_store_commit();
    }
  }
}

}  // namespace gemm_detail
}  // namespace rt
