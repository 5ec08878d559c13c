// GEMM for few rows: C[M][N] = A[M][K] W[N][K]^T with the K range of a 128 x 64 output tile split over the CTAs of a
// cluster.
//
// A batch of 128 rows gives one row of tiles: 12 CTAs for 768 columns.  A CTA that walks all K blocks of such a tile
// by itself is bound by what one SM can fetch from L2 (24 KB per 64-wide K block, 288 KB for K = 768: about 2.4 us of a
// kernel of 5 us), while most SMs have nothing to do.  Here S CTAs fetch and multiply K / S each; each CTA then owns
// 64 / S columns of the tile, receives the other CTAs' fp32 sums of them in its shared memory (distributed shared
// memory stores, one cluster barrier), adds them up in rank order and runs the epilogue on them.
//
//   warp 0     TMA producer.  W slices of the first ring fill are requested before griddepcontrol.wait where the caller
//              knows that nothing in flight writes W: they come from HBM while the kernel before this one still runs.
//   warp 1     MMA issuer
//   warps 2-5  accumulator (a TMEM lane quarter each) -> column owners, sums -> epilogue
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.h"
#include "device_error.h"
#include "gemm_epilogue.cuh"
#include "launch.h"
#include "launch_count.h"
#include "sm100_ptx.cuh"
#include "tma_host.h"

namespace rt {
namespace {

using namespace ptx;
using namespace gemm_detail;

constexpr int kBM = 128, kBN = 64, kBK = 64;
// All K blocks of a CTA for K <= 768; one CTA per SM (two, with 3 stages, were packed onto half of the SMs).
constexpr int kStages = 6;
constexpr int kABytes = kBM * kBK * 2;
constexpr int kWBytes = kBN * kBK * 2;
constexpr int kStageBytes = kABytes + kWBytes;
constexpr int kSumBytes = kBM * kBN * 4;  // S x 128 rows x 64 / S columns
constexpr int kThreads = 192;
constexpr int kTmemCols = 64;
constexpr int kSmemBytes = kStages * kStageBytes + kSumBytes + 1024 + 128;

__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, const uint32_t* v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}

template <bool BF16, int EPI, int S>
__global__ void __launch_bounds__(kThreads, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    uint16_t* __restrict__ C, const uint16_t* __restrict__ bias, int M, int N, int K, int* error_flag,
                    QkvEpilogue extra) {
  constexpr int kCols = kBN / S;  // columns of the tile that this CTA owns
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sums = smem + kStages * kStageBytes;  // [S sources][kCols / 4][128 rows] float4
  uint64_t* bars = reinterpret_cast<uint64_t*>(sums + kSumBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kStages;
  uint64_t* acc_full = bars + 2 * kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  RT_PDL_LAUNCH_DEPENDENTS();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int n0 = blockIdx.x / S * kBN, m0 = blockIdx.y * kBM;
  const int k_blocks = K / kBK;
  const int kb0 = rank * k_blocks / S, n_kb = (rank + 1) * k_blocks / S - kb0;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);  // their fetch overlaps the end of the kernel before, too
    prefetch_tensormap(&map_w);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *cta_abort = 0;
    fence_barrier_init();
    if (extra.settled_w) {
      for (int i = 0; i < kStages && i < n_kb; ++i) {
        mbar_arrive_expect_tx(&full[i], kStageBytes);
        tma_load_2d(smem + i * kStageBytes + kABytes, &map_w, (kb0 + i) * kBK, n0, &full[i]);
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();  // every CTA of the cluster runs before another one writes to it
  cluster_wait();
  tc_fence_after_sync();
  RT_PDL_WAIT();  // A and the output belong to the previous kernel until here, W as well unless it is settled
  const uint32_t tmem_base = *tmem_slot;
  AbortCtx ab{cta_abort, error_flag};

  if (warp == 0) {
    if (lane == 0) {
      for (int i = 0; i < n_kb; ++i) {
        const int s = i % kStages;
        const bool w_there = extra.settled_w && i < kStages;
        if (i >= kStages && !mbar_wait(&empty[s], (i / kStages - 1) & 1, ab, 131)) break;
        uint8_t* sa = smem + s * kStageBytes;
        if (!w_there) mbar_arrive_expect_tx(&full[s], kStageBytes);
        tma_load_2d(sa, &map_a, (kb0 + i) * kBK, m0, &full[s]);
        if (!w_there) tma_load_2d(sa + kABytes, &map_w, (kb0 + i) * kBK, n0, &full[s]);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_f16(kBM, kBN, BF16 ? 1 : 0, false);
    const bool elected = elect_one();
    const uint32_t smem_base = smem_u32(smem);
    bool ok = true;
    for (int i = 0; i < n_kb; ++i) {
      const int s = i % kStages;
      if (!mbar_wait(&full[s], (i / kStages) & 1, ab, 132)) { ok = false; break; }
      tc_fence_after_sync();
      const uint64_t da = make_smem_desc_sw128(smem_base + s * kStageBytes);
      const uint64_t dw = make_smem_desc_sw128(smem_base + s * kStageBytes + kABytes);
      if (elected) {
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k)
          mma_ss(tmem_base, da + (k * 32 >> 4), dw + (k * 32 >> 4), idesc, i > 0 || k > 0 ? 1u : 0u);
        tc_commit(&empty[s]);
      }
      __syncwarp();
    }
    if (ok && elected) tc_commit(acc_full);
    __syncwarp();
  } else {
    const int quarter = warp & 3, row = quarter * 32 + lane;
    uint32_t r[kBN];
    if (mbar_wait(acc_full, 0, ab, 133)) {
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      tmem_ld32(taddr, r);
      tmem_ld32(taddr + 32, r + 32);
      tc_wait_ld();
      const uint32_t mine = smem_u32(sums) + (rank * (kCols / 4) * kBM + row) * 16;
#pragma unroll
      for (int owner = 0; owner < S; ++owner) {
        const uint32_t dst = map_to_rank(mine, owner);
#pragma unroll
        for (int j = 0; j < kCols / 4; ++j) st_cluster_v4(dst + j * kBM * 16, r + owner * kCols + 4 * j);
      }
    }
  }
  // every CTA's sums have arrived (and nobody is written to any more)
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (warp >= 2) {
    const int row = (warp & 3) * 32 + lane;
    float x[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) x[j] = 0.f;
#pragma unroll
    for (int src = 0; src < S; ++src)
#pragma unroll
      for (int j = 0; j < kCols / 4; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(sums + ((src * (kCols / 4) + j) * kBM + row) * 16);
        x[4 * j] += v.x;
        x[4 * j + 1] += v.y;
        x[4 * j + 2] += v.z;
        x[4 * j + 3] += v.w;
      }
    uint32_t bits[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) bits[j] = __float_as_uint(x[j]);
    epilogue_chunk<BF16, EPI, kCols>(bits, n0 + rank * kCols, m0 + row, M, N, C, bias, extra);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <bool BF16, int EPI, int S>
rt_status launch_cluster(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, cudaStream_t st,
                         const QkvEpilogue& extra) {
  CUtensorMap ma, mw;
  RT_TRY(make_tensor_map_2d(&ma, a, M, K, K, kBM, kBK, true));
  RT_TRY(make_tensor_map_2d(&mw, w, N, K, K, kBN, kBK, true));
  auto kern = gemm_cluster_kernel<BF16, EPI, S>;
  RT_TRY(ensure_kernel_smem(reinterpret_cast<const void*>(kern), kSmemBytes, true));
  int* err = device_error_word();
  RT_REQUIRE(err != nullptr, RT_ERR_CUDA, "gemm: cannot allocate the device error word");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(N / kBN * S, (M + kBM - 1) / kBM);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  RT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mw, static_cast<uint16_t*>(c), static_cast<const uint16_t*>(bias), M, N,
                                   K, err, extra));
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

template <bool BF16, int EPI>
rt_status dispatch_s(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, cudaStream_t st,
                     const QkvEpilogue& extra, int cluster) {
  if (cluster == 8) return launch_cluster<BF16, EPI, 8>(c, a, w, bias, M, N, K, st, extra);
  if (cluster == 4) return launch_cluster<BF16, EPI, 4>(c, a, w, bias, M, N, K, st, extra);
  return launch_cluster<BF16, EPI, 2>(c, a, w, bias, M, N, K, st, extra);
}

template <bool BF16>
rt_status dispatch(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi, cudaStream_t st,
                   const QkvEpilogue& extra, int cluster) {
  switch (epi) {
    case RT_EPI_NONE: return dispatch_s<BF16, RT_EPI_NONE>(c, a, w, bias, M, N, K, st, extra, cluster);
    case RT_EPI_BIAS: return dispatch_s<BF16, RT_EPI_BIAS>(c, a, w, bias, M, N, K, st, extra, cluster);
    case RT_EPI_BIAS_GELU: return dispatch_s<BF16, RT_EPI_BIAS_GELU>(c, a, w, bias, M, N, K, st, extra, cluster);
    case RT_EPI_BIAS_RESIDUAL: return dispatch_s<BF16, RT_EPI_BIAS_RESIDUAL>(c, a, w, bias, M, N, K, st, extra, cluster);
    case kEpiQkv: return dispatch_s<BF16, kEpiQkv>(c, a, w, bias, M, N, K, st, extra, cluster);
    case kEpiPartial: return dispatch_s<BF16, kEpiPartial>(c, a, w, bias, M, N, K, st, extra, cluster);
  }
  return fail(RT_ERR_INVALID, "gemm: unknown epilogue %d", epi);
}

}  // namespace

rt_status gemm_cluster_dispatch(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi,
                                bool bf16, cudaStream_t st, const gemm_detail::QkvEpilogue& extra, int cluster) {
  return bf16 ? dispatch<true>(c, a, w, bias, M, N, K, epi, st, extra, cluster)
              : dispatch<false>(c, a, w, bias, M, N, K, epi, st, extra, cluster);
}

}  // namespace rt
