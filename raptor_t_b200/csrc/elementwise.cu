// Memory-bound kernels of the encoder layer: residual + bias + LayerNorm,
// bias + GELU(tanh), QKV bias + scale + split + head-major transpose, and the
// embedding gather + LayerNorm.  All of them move 128-bit vectors, keep
// statistics in fp32 and are sized against HBM bandwidth, not FLOPs.
//
// Reference counterparts: layers/kernels/add_bias_and_layernorm.cu:191-285,
// layers/kernels/add_bias_act.cu:86-133, layers/kernels/add_bias_and_transpose.cu:118-233,
// python/modeling_bert.py:45-60.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.h"
#include "launch.h"
#include "launch_count.h"

namespace rt {
namespace {

template <typename T>
struct Vec8;  // 8 x 16-bit = 128 bits

template <>
struct Vec8<__half> {
  static __device__ __forceinline__ void unpack(const uint4& v, float* f) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 t = __half22float2(h[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
  static __device__ __forceinline__ uint4 pack(const float* f) {
    uint4 v;
    __half2* h = reinterpret_cast<__half2*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
    return v;
  }
};

template <>
struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void unpack(const uint4& v, float* f) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  static __device__ __forceinline__ uint4 pack(const float* f) {
    uint4 v;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    return v;
  }
};

// four 16-bit values at once (64 bits)
template <typename T>
__device__ __forceinline__ void unpack4(const T* p, float* f) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  float t[8];
  Vec8<T>::unpack(make_uint4(w.x, w.y, 0u, 0u), t);
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = t[i];
}
template <typename T>
__device__ __forceinline__ void pack4(const float* f, T* p) {
  const float t[8] = {f[0], f[1], f[2], f[3], 0.f, 0.f, 0.f, 0.f};
  const uint4 w = Vec8<T>::pack(t);
  *reinterpret_cast<uint2*>(p) = make_uint2(w.x, w.y);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// residual + bias + LayerNorm: one warp per row, NV 128-bit vectors per lane.
// Two-pass statistics on the register copy (mean, then sum of squared
// deviations), fp32 throughout.  Warps walk rows with a grid stride; bias, gamma
// and beta are staged once per CTA in shared memory so that the kernel keeps few
// registers and many warps (loads in flight) per SM.
// Bound by HBM as long as loads are in flight all the time: a row's 16-bit vectors are on their way while the warp
// reduces, normalises and stores the one before (32768 rows from HBM, 768 columns 26.8 -> 25.4 us = 5.9 TB/s, a plain
// copy of the same traffic 26.6; 1024 columns 35.8 -> 32.2, 2048 columns 76.7 -> 63.7; below one row per warp up to 0.1 us
// slower: 2400 rows of 64 columns 1.79 -> 1.88).  CTAs per SM as registers allow without spills: 1024 columns with three
// 34.0 us.
// ---------------------------------------------------------------------------
constexpr int layernorm_ctas(int nv) { return nv <= 3 ? 3 : nv <= 6 ? 2 : 1; }  // resident per SM
template <typename T, int NV>
__global__ void __launch_bounds__(256, layernorm_ctas(NV))
layernorm_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ bias,
                 const T* __restrict__ residual, const T* __restrict__ gamma, const T* __restrict__ beta, int rows,
                 int hidden, float eps) {
  // bias, gamma and beta sit in shared memory: re-read per row at shared-memory latency
  // without holding registers across rows
  extern __shared__ uint4 s_par[];  // [3][hidden / 8]
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  const int warp = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int total_warps = gridDim.x * warps_per_block;
  const int vecs = hidden >> 3;
  const float inv_h = 1.0f / static_cast<float>(hidden);
  RT_PDL_LAUNCH_DEPENDENTS();
  uint4* s_bias = s_par;
  uint4* s_gamma = s_par + vecs;
  uint4* s_beta = s_par + 2 * vecs;
  for (int i = threadIdx.x; i < vecs; i += blockDim.x) {
    s_bias[i] = bias ? reinterpret_cast<const uint4*>(bias)[i] : make_uint4(0, 0, 0, 0);
    s_gamma[i] = reinterpret_cast<const uint4*>(gamma)[i];
    s_beta[i] = reinterpret_cast<const uint4*>(beta)[i];
  }
  __syncthreads();
  RT_PDL_WAIT();

  uint4 xv[NV], rv[NV];
  auto load = [&](int row) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * hidden);
    const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + static_cast<size_t>(row) * hidden) : nullptr;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      if (c < vecs) {
        xv[i] = xr[c];
        rv[i] = rr ? rr[c] : make_uint4(0, 0, 0, 0);
      }
    }
  };
  if (warp < rows) load(warp);
  for (int row = warp; row < rows; row += total_warps) {
    float v[NV][8];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      if (c < vecs) {
        float a[8], r[8], bb[8];
        Vec8<T>::unpack(xv[i], a);
        Vec8<T>::unpack(rv[i], r);
        Vec8<T>::unpack(s_bias[c], bb);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          v[i][k] = a[k] + bb[k] + r[k];
          sum += v[i][k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[i][k] = 0.f;
      }
    }
    if (row + total_warps < rows) load(row + total_warps);
    const float mean = warp_sum(sum) * inv_h;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      if (c < vecs) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float d = v[i][k] - mean;
          sq += d * d;
        }
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) * inv_h + eps);
    uint4* orow = reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * hidden);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      if (c < vecs) {
        float gg[8], be[8], o[8];
        Vec8<T>::unpack(s_gamma[c], gg);
        Vec8<T>::unpack(s_beta[c], be);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = (v[i][k] - mean) * rstd * gg[k] + be[k];
        orow[c] = Vec8<T>::pack(o);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The same over a projection given as `splits` fp32 parts [splits][rows][hidden] (split-K GEMM): sums the
// parts, adds bias and residual, normalises.  One CTA per row, four columns per thread: bound by the latency of the
// part loads (all parts of a row are in flight together).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float block_sum(float v, float* s_warp) {
  v = warp_sum(v);
  const int warps = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < warps; ++i) t += s_warp[i];
  return t;
}

template <typename T>
__global__ void __launch_bounds__(1024) layernorm_parts_kernel(T* __restrict__ out, const float* __restrict__ parts,
                                                               const T* __restrict__ bias,
                                                               const T* __restrict__ residual,
                                                               const T* __restrict__ gamma, const T* __restrict__ beta,
                                                               int rows, int hidden, int splits, float eps) {
  __shared__ float s_sum[32], s_sq[32];
  RT_PDL_LAUNCH_DEPENDENTS();
  const int col = threadIdx.x * 4;
  const size_t at = static_cast<size_t>(blockIdx.x) * hidden + col;
  const float inv_h = 1.0f / static_cast<float>(hidden);
  float bb[4], gg[4], be[4], rr[4], v[4] = {0.f, 0.f, 0.f, 0.f};
  RT_PDL_WAIT();
  unpack4(bias + col, bb);
  unpack4(gamma + col, gg);
  unpack4(beta + col, be);
  unpack4(residual + at, rr);
  const size_t stride = static_cast<size_t>(rows) * hidden;
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float4 p = *reinterpret_cast<const float4*>(parts + s * stride + at);
    v[0] += p.x;
    v[1] += p.y;
    v[2] += p.z;
    v[3] += p.w;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] += bb[k] + rr[k];
  const float mean = block_sum(v[0] + v[1] + v[2] + v[3], s_sum) * inv_h;
  float sq = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) sq += (v[k] - mean) * (v[k] - mean);
  const float rstd = rsqrtf(block_sum(sq, s_sq) * inv_h + eps);
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = (v[k] - mean) * rstd * gg[k] + be[k];
  pack4(v, out + at);
}

// ---------------------------------------------------------------------------
// The same with one warp per row, four columns of every 128 per lane: all loads of a part, or of two, are in flight
// together and nothing but shuffles joins a row.  Against one CTA per row, us alone: 320 x 768, four parts 3.6 -> 2.7,
// 512, three parts 3.7 -> 2.7, 2048, two 5.0 -> 3.3, 6144, one 11.2 -> 5.1 (37.7 MB: 7.4 TB/s, out of L2).
// ---------------------------------------------------------------------------
constexpr int kPartsThreads = 128;
template <typename T, int NV>
__global__ void __launch_bounds__(kPartsThreads, 4)
layernorm_parts_rows_kernel(T* __restrict__ out, const float* __restrict__ parts, const T* __restrict__ bias,
                            const T* __restrict__ residual, const T* __restrict__ gamma, const T* __restrict__ beta, int rows,
                       int splits, float eps) {
  constexpr int kHidden = NV * 128;
  constexpr int kWarps = kPartsThreads / 32;
  RT_PDL_LAUNCH_DEPENDENTS();
  const int col = (threadIdx.x & 31) * 4;
  const size_t stride = static_cast<size_t>(rows) * kHidden;
  RT_PDL_WAIT();
  for (int row = blockIdx.x * kWarps + (threadIdx.x >> 5); row < rows; row += gridDim.x * kWarps) {
    const size_t at = static_cast<size_t>(row) * kHidden + col;
    uint2 res[NV];
    float v[NV][4];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      res[i] = *reinterpret_cast<const uint2*>(residual + at + i * 128);
#pragma unroll
      for (int k = 0; k < 4; ++k) v[i][k] = 0.f;
    }
#pragma unroll 2
    for (int s = 0; s < splits; ++s)
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const float4 p = *reinterpret_cast<const float4*>(parts + s * stride + at + i * 128);
        v[i][0] += p.x;
        v[i][1] += p.y;
        v[i][2] += p.z;
        v[i][3] += p.w;
      }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float bb[4], rr[8];
      unpack4(bias + col + i * 128, bb);
      Vec8<T>::unpack(make_uint4(res[i].x, res[i].y, 0u, 0u), rr);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[i][k] += bb[k] + rr[k];
        sum += v[i][k];
      }
    }
    const float mean = warp_sum(sum) * (1.0f / kHidden);
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) sq += (v[i][k] - mean) * (v[i][k] - mean);
    const float rstd = rsqrtf(warp_sum(sq) * (1.0f / kHidden) + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float gg[4], be[4], o[4];
      unpack4(gamma + col + i * 128, gg);
      unpack4(beta + col + i * 128, be);
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = (v[i][k] - mean) * rstd * gg[k] + be[k];
      pack4(o, out + at + i * 128);
    }
  }
}

// ---------------------------------------------------------------------------
// bias + GELU (tanh form), in place, one 128-bit vector per thread per step.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float gelu_tanh(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return 0.5f * x * (1.0f + t);
}

template <typename T, int UNROLL>
__global__ void __launch_bounds__(256) bias_gelu_kernel(T* __restrict__ x, const T* __restrict__ bias,
                                                        size_t total_vecs, int vecs_per_row) {
  RT_PDL_LAUNCH_DEPENDENTS();
  RT_PDL_WAIT();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  uint4* xv = reinterpret_cast<uint4*>(x);
  const uint4* bv = reinterpret_cast<const uint4*>(bias);
  for (; i + (UNROLL - 1) * stride < total_vecs; i += UNROLL * stride) {
    uint4 a[UNROLL], b[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      a[u] = xv[i + u * stride];
      b[u] = bv[(i + u * stride) % vecs_per_row];
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      float f[8], bb[8];
      Vec8<T>::unpack(a[u], f);
      Vec8<T>::unpack(b[u], bb);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] = gelu_tanh(f[k] + bb[k]);
      xv[i + u * stride] = Vec8<T>::pack(f);
    }
  }
  for (; i < total_vecs; i += stride) {
    float f[8], bb[8];
    Vec8<T>::unpack(xv[i], f);
    Vec8<T>::unpack(bv[i % vecs_per_row], bb);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = gelu_tanh(f[k] + bb[k]);
    xv[i] = Vec8<T>::pack(f);
  }
}

// ---------------------------------------------------------------------------
// QKV bias + scale + split + transpose to per-sequence head-major layout.
// One CTA per (64-token block, q|k|v part).  Every 128-byte chunk (one token,
// one head) is read and written whole, so both sides are fully coalesced.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) qkv_transpose_kernel(const T* __restrict__ qkv, const T* __restrict__ bias,
                                                            T* __restrict__ q, T* __restrict__ k, T* __restrict__ v,
                                                            const int32_t* __restrict__ seq_prefix, int n_seq,
                                                            int heads, float q_scale) {
  RT_PDL_LAUNCH_DEPENDENTS();
  RT_PDL_WAIT();
  const int blk = blockIdx.x;   // packed 64-token block
  const int part = blockIdx.y;  // 0 q, 1 k, 2 v
  __shared__ int s_first_blk, s_nblk;
  if (threadIdx.x == 0) {
    int lo = 0, hi = n_seq;  // largest s with seq_prefix[s] <= blk
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (seq_prefix[mid] <= blk) lo = mid; else hi = mid;
    }
    s_first_blk = seq_prefix[lo];
    s_nblk = seq_prefix[lo + 1] - seq_prefix[lo];
  }
  __syncthreads();
  const int hidden = heads * 64;
  const int vec_per_part = hidden >> 3;                 // vectors per token in this part
  const int seq_tok0 = s_first_blk * 64;
  const int seq_len = s_nblk * 64;
  const int tok_in_seq0 = (blk - s_first_blk) * 64;
  T* dst_base = (part == 0 ? q : part == 1 ? k : v) + static_cast<size_t>(seq_tok0) * hidden;
  const float scale = part == 0 ? q_scale : 1.0f;
  const uint4* src = reinterpret_cast<const uint4*>(qkv);
  const uint4* bsrc = reinterpret_cast<const uint4*>(bias) + part * vec_per_part;
  const int total = 64 * vec_per_part;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int t = i / vec_per_part;       // token in block
    const int c = i - t * vec_per_part;   // vector in this part's row
    const int h = c >> 3, dv = c & 7;
    const size_t tok = static_cast<size_t>(blk) * 64 + t;
    const uint4 a = src[tok * (3 * vec_per_part) + part * vec_per_part + c];
    float f[8], bb[8];
    Vec8<T>::unpack(a, f);
    if (bias) {
      Vec8<T>::unpack(bsrc[c], bb);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = (f[e] + bb[e]) * scale;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= scale;
    }
    const size_t row = static_cast<size_t>(h) * seq_len + tok_in_seq0 + t;
    reinterpret_cast<uint4*>(dst_base + row * 64)[dv] = Vec8<T>::pack(f);
  }
}

// ---------------------------------------------------------------------------
// embeddings: fp32 tables, one warp per token, same statistics as LayerNorm.  Bound by the gather of the word rows
// from HBM: a warp reads its rows in contiguous 512-byte pieces, all of them in flight at once (NV per table), and
// walks the tokens with a grid stride, so that gamma and beta are staged in shared memory once per CTA.  20480 tokens of 768:
// 24.6 us (44.7 with 16-byte loads at a stride of 32 and parameters read word by word), 76000 of 1024: 92 (207).
// ---------------------------------------------------------------------------
template <typename T, int NV>
__global__ void __launch_bounds__(256) embeddings_kernel(T* __restrict__ out, const int32_t* __restrict__ ids,
                                                         const int32_t* __restrict__ pos_ids,
                                                         const int32_t* __restrict__ type_ids,
                                                         const float* __restrict__ word, const float* __restrict__ pos,
                                                         const float* __restrict__ type, const float* __restrict__ gamma,
                                                         const float* __restrict__ beta, int tokens, int hidden,
                                                         float eps) {
  __shared__ float4 s_gamma[32 * NV], s_beta[32 * NV];
  RT_PDL_LAUNCH_DEPENDENTS();
  RT_PDL_WAIT();
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {  // scalar: the parameters need no alignment
    reinterpret_cast<float*>(s_gamma)[i] = gamma[i];
    reinterpret_cast<float*>(s_beta)[i] = beta[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int vecs = hidden >> 2;
  const float inv_h = 1.0f / static_cast<float>(hidden);
  for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tokens; t += warps) {
    const float4* wr = reinterpret_cast<const float4*>(word + static_cast<size_t>(ids[t]) * hidden);
    const float4* pr = reinterpret_cast<const float4*>(pos + static_cast<size_t>(pos_ids ? pos_ids[t] : 0) * hidden);
    const float4* tr = reinterpret_cast<const float4*>(type + static_cast<size_t>(type_ids ? type_ids[t] : 0) * hidden);
    float4 v[NV], pv[NV], tv[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      if (c < vecs) {
        v[i] = wr[c];
        pv[i] = pr[c];
        tv[i] = tr[c];
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (lane + 32 * i < vecs) {
        v[i].x = v[i].x + tv[i].x + pv[i].x;
        v[i].y = v[i].y + tv[i].y + pv[i].y;
        v[i].z = v[i].z + tv[i].z + pv[i].z;
        v[i].w = v[i].w + tv[i].w + pv[i].w;
        sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
      }
    }
    const float mean = warp_sum(sum) * inv_h;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (lane + 32 * i < vecs) {
        v[i].x -= mean;
        v[i].y -= mean;
        v[i].z -= mean;
        v[i].w -= mean;
        sq += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) * inv_h + eps);
    T* orow = out + static_cast<size_t>(t) * hidden;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      if (c < vecs) {
        const float4 g = s_gamma[c], b = s_beta[c];
        const float o[4] = {v[i].x * rstd * g.x + b.x, v[i].y * rstd * g.y + b.y, v[i].z * rstd * g.z + b.z,
                            v[i].w * rstd * g.w + b.w};
        pack4(o, orow + 4 * c);
      }
    }
  }
}

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

template <typename T>
static rt_status layernorm_launch(void* out, const void* x, const void* bias, const void* residual, const void* gamma,
                                  const void* beta, int rows, int hidden, float eps, cudaStream_t st) {
  const int nv = (hidden / 8 + 31) / 32;
  const int threads = 256, wpb = threads / 32;
  // one wave of resident CTAs, or two of the small ones (20480 x 768: 16.4 and 16.5 us, four waves 17.9); warps walk the
  // rows with a grid stride, so the parameters are staged in shared memory a few times per SM instead of once per 8 rows
  int blocks = std::min((rows + wpb - 1) / wpb, sm_count() * (nv <= 3 ? 6 : layernorm_ctas(nv)));
  if (blocks < 1) blocks = 1;
#define RT_LN_CASE(NV)                                                                                           \
  case NV:                                                                                                       \
    launch_kernel(layernorm_kernel<T, NV>, dim3(blocks), dim3(threads), 3 * (hidden / 8) * sizeof(uint4), st,   \
                  (T*)out, (const T*)x, (const T*)bias, (const T*)residual, (const T*)gamma, (const T*)beta, rows, \
                  hidden, eps);                                                                                  \
    break;
  switch (nv) {
    RT_LN_CASE(1)
    RT_LN_CASE(2)
    RT_LN_CASE(3)
    RT_LN_CASE(4)
    RT_LN_CASE(6)
    RT_LN_CASE(8)
    default:
      return fail(RT_ERR_UNSUPPORTED, "layernorm: hidden=%d not supported (<=1024, 1536 or 2048)", hidden);
  }
#undef RT_LN_CASE
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

// One warp per row or one CTA.  12 layers, us, one CTA / one warp per row, 20 to 30 repeats in turn:
//   512 columns  320 rows 421.9 / 417.1   640 486.8 / 480.6   1024 517.3 / 505.9   1600 587.8 / 579.7
//   640 columns  320 rows 452.1 / 444.4   640 533.9 / 523.6   1152 587.1 / 587.1   1792 647.1 / 630.2
//   768 columns  320 rows 487.4 / 478.7   512 542.0 / 538.7   576 550.0 / 556.2    704 567.4 / 575.5
//                1024 604.3 / 608.3       1472 670.9 / 671.7  1536 685.2 / 672.9   2304 793.8 / 772.1   6144 1420 / 1359
// Up to 256 rows neither is faster (768 columns 128 rows 376.2 / 380.2); 1024 columns (up to 1152 rows) are slower with
// warps, 512 rows 624.6 / 634.2, 1024 741.2 / 768.0, 896 equal: there the many small CTAs leave the next GEMM's start alone.
bool layernorm_parts_by_warps(int rows, int hidden) {
  return rows > 256 && (hidden <= 640 || (hidden <= 768 && (rows <= 512 || rows >= 1536)));
}

template <typename T>
static rt_status layernorm_parts_launch(T* out, const float* parts, int splits, const T* bias, const T* residual,
                                        const T* gamma, const T* beta, int rows, int hidden, float eps, cudaStream_t st) {
  if (!layernorm_parts_by_warps(rows, hidden)) {
    RT_CHECK_CUDA(launch_kernel(layernorm_parts_kernel<T>, dim3(rows), dim3(hidden / 4), 0, st, out, parts, bias, residual,
                                gamma, beta, rows, hidden, splits, eps));
    count_launch();
    RT_CHECK_CUDA(cudaGetLastError());
    return RT_OK;
  }
  const int per_cta = kPartsThreads / 32;
  const int blocks = std::min((rows + per_cta - 1) / per_cta, 4 * sm_count());
#define RT_PARTS_CASE(NV)                                                                                            \
  case NV:                                                                                                           \
    RT_CHECK_CUDA(launch_kernel(layernorm_parts_rows_kernel<T, NV>, dim3(blocks), dim3(kPartsThreads), 0, st, out, parts, \
                                bias, residual, gamma, beta, rows, splits, eps));                                    \
    break;
  switch (hidden / 128) {
    RT_PARTS_CASE(1)
    RT_PARTS_CASE(2)
    RT_PARTS_CASE(3)
    RT_PARTS_CASE(4)
    RT_PARTS_CASE(5)
    RT_PARTS_CASE(6)
    default:
      return fail(RT_ERR_UNSUPPORTED, "layernorm_parts: hidden=%d not supported", hidden);
  }
#undef RT_PARTS_CASE
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

// out = LayerNorm(sum of the parts + bias + residual) * gamma + beta; hidden % 128 == 0, hidden <= 1024
rt_status layernorm_parts(void* out, const float* parts, int splits, const void* bias, const void* residual,
                          const void* gamma, const void* beta, int rows, int hidden, float eps, int dtype,
                          cudaStream_t st) {
  RT_REQUIRE(hidden > 0 && hidden % 128 == 0 && hidden <= 1024, RT_ERR_UNSUPPORTED, "layernorm_parts: hidden=%d not supported",
             hidden);
  if (dtype == RT_BF16)
    return layernorm_parts_launch((__nv_bfloat16*)out, parts, splits, (const __nv_bfloat16*)bias,
                                  (const __nv_bfloat16*)residual, (const __nv_bfloat16*)gamma, (const __nv_bfloat16*)beta,
                                  rows, hidden, eps, st);
  return layernorm_parts_launch((__half*)out, parts, splits, (const __half*)bias, (const __half*)residual,
                                (const __half*)gamma, (const __half*)beta, rows, hidden, eps, st);
}

}  // namespace rt

using namespace rt;

extern "C" rt_status rt_bias_residual_layernorm(void* out, const void* x, const void* bias, const void* residual,
                                                const void* gamma, const void* beta, int rows, int hidden, float eps,
                                                int dtype, void* stream) {
  RT_REQUIRE(out && x && gamma && beta, RT_ERR_INVALID, "layernorm: null pointer");
  RT_REQUIRE(rows >= 0 && hidden > 0 && hidden % 8 == 0, RT_ERR_INVALID, "layernorm: hidden must be a multiple of 8");
  RT_REQUIRE(aligned16(out) && aligned16(x) && aligned16(gamma) && aligned16(beta) && aligned16(bias) &&
                 aligned16(residual),
             RT_ERR_INVALID, "layernorm: pointers must be 16-byte aligned");
  if (rows == 0) return RT_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == RT_F16) return layernorm_launch<__half>(out, x, bias, residual, gamma, beta, rows, hidden, eps, st);
  if (dtype == RT_BF16)
    return layernorm_launch<__nv_bfloat16>(out, x, bias, residual, gamma, beta, rows, hidden, eps, st);
  return fail(RT_ERR_INVALID, "layernorm: unknown dtype %d", dtype);
}

extern "C" rt_status rt_bias_gelu(void* x, const void* bias, int rows, int cols, int dtype, void* stream) {
  RT_REQUIRE(x && bias, RT_ERR_INVALID, "bias_gelu: null pointer");
  RT_REQUIRE(rows >= 0 && cols > 0 && cols % 8 == 0, RT_ERR_INVALID, "bias_gelu: cols must be a multiple of 8");
  RT_REQUIRE(aligned16(x) && aligned16(bias), RT_ERR_INVALID, "bias_gelu: pointers must be 16-byte aligned");
  if (rows == 0) return RT_OK;
  const size_t total = static_cast<size_t>(rows) * (cols / 8);
  const int threads = 256;
  constexpr int UNROLL = 4;
  size_t want = (total + threads * UNROLL - 1) / (threads * UNROLL);
  int blocks = static_cast<int>(std::min<size_t>(want, static_cast<size_t>(sm_count()) * 16));
  if (blocks < 1) blocks = 1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == RT_F16)
    launch_kernel(bias_gelu_kernel<__half, UNROLL>, dim3(blocks), dim3(threads), 0, st, (__half*)x,
                  (const __half*)bias, total, cols / 8);
  else if (dtype == RT_BF16)
    launch_kernel(bias_gelu_kernel<__nv_bfloat16, UNROLL>, dim3(blocks), dim3(threads), 0, st, (__nv_bfloat16*)x,
                  (const __nv_bfloat16*)bias, total, cols / 8);
  else
    return fail(RT_ERR_INVALID, "bias_gelu: unknown dtype %d", dtype);
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

extern "C" rt_status rt_qkv_bias_transpose(const void* qkv, const void* bias, void* q, void* k, void* v,
                                           const int32_t* seq_block_prefix_dev, int n_seq, int total_blocks, int heads,
                                           float q_scale, int dtype, void* stream) {
  RT_REQUIRE(qkv && q && k && v && seq_block_prefix_dev, RT_ERR_INVALID, "qkv_transpose: null pointer");
  RT_REQUIRE(n_seq > 0 && total_blocks >= 0 && heads > 0, RT_ERR_INVALID, "qkv_transpose: bad sizes");
  RT_REQUIRE(aligned16(qkv) && aligned16(bias) && aligned16(q) && aligned16(k) && aligned16(v), RT_ERR_INVALID,
             "qkv_transpose: pointers must be 16-byte aligned");
  if (total_blocks == 0) return RT_OK;
  dim3 grid(total_blocks, 3);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == RT_F16)
    launch_kernel(qkv_transpose_kernel<__half>, grid, dim3(256), 0, st, (const __half*)qkv, (const __half*)bias,
                  (__half*)q, (__half*)k, (__half*)v, seq_block_prefix_dev, n_seq, heads, q_scale);
  else if (dtype == RT_BF16)
    launch_kernel(qkv_transpose_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, (const __nv_bfloat16*)qkv,
                  (const __nv_bfloat16*)bias, (__nv_bfloat16*)q, (__nv_bfloat16*)k, (__nv_bfloat16*)v,
                  seq_block_prefix_dev, n_seq, heads, q_scale);
  else
    return fail(RT_ERR_INVALID, "qkv_transpose: unknown dtype %d", dtype);
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

extern "C" rt_status rt_embeddings(void* out, const int32_t* ids, const int32_t* pos_ids, const int32_t* type_ids,
                                   const void* word, const void* pos, const void* type, const void* gamma,
                                   const void* beta, int tokens, int hidden, float eps, int dtype, void* stream) {
  RT_REQUIRE(out && ids && word && pos && type && gamma && beta, RT_ERR_INVALID, "embeddings: null pointer");
  RT_REQUIRE(hidden > 0 && hidden % 8 == 0 && hidden <= 1024, RT_ERR_UNSUPPORTED,
             "embeddings: hidden=%d not supported (multiple of 8, <= 1024)", hidden);
  RT_REQUIRE(aligned16(out) && aligned16(word) && aligned16(pos) && aligned16(type), RT_ERR_INVALID,
             "embeddings: pointers must be 16-byte aligned");
  if (tokens == 0) return RT_OK;
  const int nv = (hidden / 4 + 63) / 64;  // pairs of 512-byte pieces per row
  const int threads = 256, wpb = 8;
  const int blocks = std::min((tokens + wpb - 1) / wpb, sm_count() * 4);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define RT_EMB(T, NV)                                                                                          \
  launch_kernel(embeddings_kernel<T, NV>, dim3(blocks), dim3(threads), 0, st, (T*)out, ids, pos_ids, type_ids, \
                (const float*)word, (const float*)pos, (const float*)type, (const float*)gamma,                \
                (const float*)beta, tokens, hidden, eps)
  if (dtype == RT_F16) {
    switch (nv) { case 1: RT_EMB(__half, 2); break; case 2: RT_EMB(__half, 4); break; case 3: RT_EMB(__half, 6); break; default: RT_EMB(__half, 8); }
  } else if (dtype == RT_BF16) {
    switch (nv) { case 1: RT_EMB(__nv_bfloat16, 2); break; case 2: RT_EMB(__nv_bfloat16, 4); break; case 3: RT_EMB(__nv_bfloat16, 6); break; default: RT_EMB(__nv_bfloat16, 8); }
  } else {
    return fail(RT_ERR_INVALID, "embeddings: unknown dtype %d", dtype);
  }
#undef RT_EMB
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}
