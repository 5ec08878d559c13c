// Which tiles a GEMM is cut into (gemm_sm100.cu).
#pragma once
#include <cuda_runtime.h>

#include "common.h"
#include "gemm_epilogue.cuh"

namespace rt {

struct GemmPlan {
  bool pair = false;   // CTA-pair kernel (256-row tiles) or single-CTA kernel (128-row tiles)
  int main_tiles = 0;  // pair kernel: this many 256-column tiles come first, the rest is `width` wide
  int width = 64;      // columns of a tile
  int splits = 1;      // parts of K (kEpiPartial only)
  double cost = 0;     // estimated microseconds
  int cluster = 0;     // > 1: K split over this many CTAs of a cluster (gemm_cluster_sm100.cu)
};

// Cheapest tiling by the measured costs of the tile shapes; parts: kEpiPartial with up to max_splits parts.
GemmPlan plan_gemm(int M, int N, int K, int max_splits, bool parts);
rt_status run_gemm(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi, int dtype,
                   cudaStream_t st, const gemm_detail::QkvEpilogue& extra, const GemmPlan& plan);

int gemm_sm_count();
// Clusters of rt_gemm_bias_residual_layernorm that the current device keeps resident: of CTA pairs (256 rows), or of
// single CTAs (128 rows, N = 768 only).  On a B200 22 and 36 for N = 768, 15 for N = 1024.
int gemm_layernorm_clusters(int N, bool pairs);

// rt_gemm, rt_gemm_bias_residual_layernorm and rt_gemm_qkv; settled_w as in QkvEpilogue.
rt_status gemm_layernorm_checked(void* out, const void* a, const void* w, const void* bias, const void* residual,
                                 const void* gamma, const void* beta, int M, int N, int K, float eps, int dtype,
                                 void* stream, bool settled_w);
rt_status gemm_checked(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epilogue,
                       int dtype, void* stream, const gemm_detail::QkvEpilogue& extra);
rt_status gemm_qkv_checked(void* q, void* k, void* v, const void* a, const void* w, const void* bias,
                           const int32_t* block_seq_dev, int M, int heads, int K, float q_scale, int dtype, void* stream,
                           bool settled_w);

}  // namespace rt
