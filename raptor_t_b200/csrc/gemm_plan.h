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
};

// Cheapest tiling by the measured costs of the tile shapes; parts: kEpiPartial with up to max_splits parts.
GemmPlan plan_gemm(int M, int N, int K, int max_splits, bool parts);
rt_status run_gemm(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi, int dtype,
                   cudaStream_t st, const gemm_detail::QkvEpilogue& extra, const GemmPlan& plan);

}  // namespace rt
