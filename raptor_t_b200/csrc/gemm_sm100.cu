// Persistent, warp-specialised tcgen05 GEMM for sm_100a:
//     C[M][N] = A[M][K] * W[N][K]^T  (+ bias) (+ GELU),  16-bit in/out, fp32 accumulate.
//
// One CTA per SM walks 128 x BN output tiles.  Warp 0 streams A and W k-slices
// (64 elements = one 128-byte swizzle atom) into a shared-memory ring with TMA;
// warp 1 issues tcgen05.mma (M=128, N=BN, K=16) into one of two TMEM
// accumulators; warps 2-9 drain the other accumulator (tcgen05.ld), apply the
// epilogue and store, so the epilogue of tile i overlaps the main loop of
// tile i+1.  Stands in for the cuBLAS calls of layers/kernels/mat_mul.cpp:58-76
// (which accumulate in fp16; this kernel accumulates in fp32).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "common.h"
#include "device_error.h"
#include "gemm_epilogue.cuh"
#include "gemm_plan.h"
#include "launch.h"
#include "launch_count.h"
#include "sm100_ptx.cuh"
#include "tma_host.h"

namespace rt {

// SM count of the current device (queried once per device).
int gemm_sm_count() {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
    cache[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

namespace {

using namespace ptx;
using namespace gemm_detail;

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kGemmThreads = 320;      // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int kEpilogueThreads = 256;  // two warps per TMEM lane quarter, alternating 32-column chunks

// Costs of the tile choice (plan_gemm), microseconds on a B200 with weights and activations in L2, fitted to
// M = 128 ... 20480 rows of the projections of 768- and 1024-wide models: per launch, per 64-wide K block of a
// tile, per tile.  A 256-column pair tile does the most work per byte it loads and wins once its waves are full;
// below that, narrower tiles on more SMs are faster (768 columns, K = 3072, 4096 rows: 48 pair tiles of 256
// columns 19.9 us, 64 of 192 15.9 us, 192 single-CTA tiles of 128 25.1 us).  For as many waves of 256 columns the
// pairs stay ahead: alone, us, single CTAs / pairs, 1024 columns: 3840 rows K = 4096 29.5 / 26.8, 5120 33.1 / 30.9, 8192
// 54.6 / 49.7, 4454 rows K = 4096 31.0 / 28.8.  Up to K = 2048 single CTAs are faster alone (K = 1024, 3840 rows 9.6 / 10.5)
// but not in the chain of a forward (12 layers of 1024 columns: FFN up of 1024 tokens 781 / 775, QKV of 1536 930 / 922).
struct TileCost {
  int width;
  double launch, k_block, tile;
  double at(int waves, int k_blocks) const { return launch + waves * (k_blocks * k_block + tile); }
};
constexpr TileCost kSingleTiles[3] = {{64, 2.3, 0.2, 0.45}, {128, 2.6, 0.235, 0.6}, {256, 3.2, 0.29, 2.1}};
constexpr TileCost kPairTiles[3] = {{128, 3.6, 0.2, 0.5}, {192, 3.6, 0.24, 1.0}, {256, 3.8, 0.29, 1.2}};
// the last, partial wave of 256-column pair tiles cut into narrower ones
constexpr TileCost kTailTiles[2] = {{64, 0, 0.15, 0.5}, {128, 0, 0.2, 0.6}};
constexpr int kClusterWidth = 64;  // columns of a tile of gemm_cluster_sm100.cu
constexpr double kPartBytesPerUs = 6e6;  // fp32 parts, written and read through L2

template <int BN>
struct GemmCfg {
  static constexpr int kStages = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = BN * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;  // power of two: 128, 256, 512
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/;
};

template <int BN, bool BF16, int EPI>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
            uint16_t* __restrict__ C, const uint16_t* __restrict__ bias, int M, int N, int K, int* error_flag,
            QkvEpilogue qkv) {
  using Cfg = GemmCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kStages * Cfg::kStageBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + Cfg::kStages;
  uint64_t* acc_full = bars + 2 * Cfg::kStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  RT_PDL_LAUNCH_DEPENDENTS();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);  // their fetch overlaps the end of the kernel before, too
    prefetch_tensormap(&map_w);
    for (int s = 0; s < Cfg::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kEpilogueThreads);
    }
    *cta_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  RT_PDL_WAIT();  // operands and the output buffer belong to the previous kernel until here
  const uint32_t tmem_base = *tmem_slot;
  AbortCtx ab{cta_abort, error_flag};

  const int n_tiles_n = N / BN;
  const int n_tiles_m = (M + kBM - 1) / kBM;
  const int mn_tiles = n_tiles_m * n_tiles_n;
  const int splits = EPI == kEpiPartial ? qkv.splits : 1;
  const int n_tiles = mn_tiles * splits;
  const int k_blocks = K / kBK;
  // tile t: output tile t % mn_tiles over K blocks [kb0, kb1) of part t / mn_tiles
  auto tile_of = [&](int t, int& m0, int& n0, int& kb0, int& kb1, int& part) {
    part = EPI == kEpiPartial ? t / mn_tiles : 0;
    const int u = EPI == kEpiPartial ? t % mn_tiles : t;
    m0 = (u / n_tiles_n) * kBM;
    n0 = (u % n_tiles_n) * BN;
    kb0 = EPI == kEpiPartial ? part * k_blocks / splits : 0;
    kb1 = EPI == kEpiPartial ? (part + 1) * k_blocks / splits : k_blocks;
  };
  int m0, n0, kb0, kb1, part;

  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        tile_of(t, m0, n0, kb0, kb1, part);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % Cfg::kStages;
          const uint32_t ph = (it / Cfg::kStages) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, ab, 101)) { ok = false; break; }
          uint8_t* sa = smem + s * Cfg::kStageBytes;
          mbar_arrive_expect_tx(&full[s], Cfg::kStageBytes);
          tma_load_2d(sa, &map_a, kb * kBK, m0, &full[s]);
          tma_load_2d(sa + Cfg::kABytes, &map_w, kb * kBK, n0, &full[s]);
        }
      }
      // A wait only gives up after the whole pipeline has been idle for the full
      // time-out, so no copy issued by this thread can still be in flight here.
      (void)ok;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer
    // the whole warp walks the loop, one elected lane issues (see gemm_pair_sm100.cu)
    {
      constexpr uint32_t idesc = make_idesc_f16(kBM, BN, BF16 ? 1 : 0, false);
      const bool elected = elect_one();
      const uint32_t smem_base = smem_u32(smem);
      uint32_t it = 0, tile_it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++tile_it) {
        const int a = tile_it & 1;
        const uint32_t aph = (tile_it >> 1) & 1;
        if (!mbar_wait(&acc_empty[a], aph ^ 1, ab, 102)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + a * BN;
        tile_of(t, m0, n0, kb0, kb1, part);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % Cfg::kStages;
          const uint32_t ph = (it / Cfg::kStages) & 1;
          if (!mbar_wait(&full[s], ph, ab, 103)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_base + s * Cfg::kStageBytes;
          const uint64_t da = make_smem_desc_sw128(sa);
          const uint64_t db = make_smem_desc_sw128(sa + Cfg::kABytes);
          if (elected) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              mma_ss(d_tmem, da + (k * 32 >> 4), db + (k * 32 >> 4), idesc, kb > kb0 || k > 0 ? 1u : 0u);
            tc_commit(&empty[s]);
          }
          __syncwarp();
        }
        if (ok && elected) tc_commit(&acc_full[a]);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue warps 2..9
    const int quarter = warp & 3;
    const int chunk0 = (warp - 2) >> 2;  // 0: even 32-column chunks, 1: odd chunks
    const int row_in_tile = quarter * 32 + lane;
    uint32_t tile_it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++tile_it) {
      const int a = tile_it & 1;
      const uint32_t aph = (tile_it >> 1) & 1;
      tile_of(t, m0, n0, kb0, kb1, part);
      if (!mbar_wait(&acc_full[a], aph, ab, 104)) { ok = false; break; }
      tc_fence_after_sync();
      const int row = m0 + row_in_tile;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * BN;
      uint16_t* c_part = EPI == kEpiPartial ? C + 2 * static_cast<size_t>(part) * M * N : C;  // fp32 parts
      epilogue_row<BF16, EPI>(BN, taddr, row, n0, chunk0, M, N, c_part, bias, qkv);
      tc_fence_before_sync();
      mbar_arrive(&acc_empty[a]);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

template <int BN, bool BF16, int EPI>
rt_status launch(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, cudaStream_t st,
                 const QkvEpilogue& qkv = QkvEpilogue{}) {
  using Cfg = GemmCfg<BN>;
  CUtensorMap ma, mw;
  RT_TRY(make_tensor_map_2d(&ma, a, M, K, K, kBM, kBK, true));
  RT_TRY(make_tensor_map_2d(&mw, w, N, K, K, BN, kBK, true));
  auto kern = gemm_kernel<BN, BF16, EPI>;
  RT_TRY(ensure_kernel_smem(reinterpret_cast<const void*>(kern), Cfg::kSmemBytes, false));
  int* err = device_error_word();
  RT_REQUIRE(err != nullptr, RT_ERR_CUDA, "gemm: cannot allocate the device error word");
  const int tiles = ((M + kBM - 1) / kBM) * (N / BN) * (EPI == kEpiPartial ? qkv.splits : 1);
  const int grid = std::min(tiles, gemm_sm_count());
  RT_CHECK_CUDA(launch_kernel(kern, dim3(grid), dim3(kGemmThreads), Cfg::kSmemBytes, st, ma, mw, (uint16_t*)c,
                              (const uint16_t*)bias, M, N, K, err, qkv));
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

template <int BN, bool BF16>
rt_status launch_epi(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi,
                     cudaStream_t st, const QkvEpilogue& qkv) {
  switch (epi) {
    case RT_EPI_NONE: return launch<BN, BF16, RT_EPI_NONE>(c, a, w, bias, M, N, K, st);
    case RT_EPI_BIAS: return launch<BN, BF16, RT_EPI_BIAS>(c, a, w, bias, M, N, K, st);
    case RT_EPI_BIAS_GELU: return launch<BN, BF16, RT_EPI_BIAS_GELU>(c, a, w, bias, M, N, K, st);
    case RT_EPI_BIAS_RESIDUAL: return launch<BN, BF16, RT_EPI_BIAS_RESIDUAL>(c, a, w, bias, M, N, K, st, qkv);
    case kEpiQkv: return launch<BN, BF16, kEpiQkv>(c, a, w, bias, M, N, K, st, qkv);
    case kEpiPartial: return launch<BN, BF16, kEpiPartial>(c, a, w, bias, M, N, K, st, qkv);
  }
  return fail(RT_ERR_INVALID, "gemm: unknown epilogue %d", epi);
}

}  // namespace

rt_status gemm_pair_dispatch(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi,
                             bool bf16, cudaStream_t st, const gemm_detail::QkvEpilogue& qkv, int main_tiles, int tail_w);
rt_status gemm_cluster_dispatch(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi,
                                bool bf16, cudaStream_t st, const gemm_detail::QkvEpilogue& extra, int cluster);

GemmPlan plan_gemm(int M, int N, int K, int max_splits, bool to_parts) {
  const int sms = gemm_sm_count(), pairs = sms / 2;
  const int mt = (M + kBM - 1) / kBM, pair_mt = (M + 2 * kBM - 1) / (2 * kBM);
  GemmPlan best;
  best.cost = 1e30;
  auto waves = [](int tiles, int units) { return (tiles + units - 1) / units; };
  for (int s = 1; s <= max_splits; ++s) {
    const int kbs = (K / kBK + s - 1) / s;
    const double parts = to_parts ? 8.0 * s * M * N / kPartBytesPerUs : 0.0;
    auto consider = [&](double cost, bool pair, int main_tiles, int width) {
      if (cost + parts < best.cost) best = GemmPlan{pair, main_tiles, width, s, cost + parts};
    };
    for (const TileCost& c : kSingleTiles)
      if (N % c.width == 0) consider(c.at(waves(mt * (N / c.width) * s, sms), kbs), false, 0, c.width);
    for (const TileCost& c : kPairTiles)
      if (N % c.width == 0) consider(c.at(waves(pair_mt * (N / c.width) * s, pairs), kbs), true, 0, c.width);
    // whole waves of 256-column pair tiles, the rest in narrower ones (5003 rows, 3072 columns, K = 768:
    // 222 + 18 tiles of 256 columns 22.7 us, 222 and 72 of 64 columns 21.2 us)
    const int tiles = pair_mt * (N / 256), full = tiles / pairs, rest = tiles % pairs;
    if (to_parts || N % 256 != 0 || full == 0 || rest == 0) continue;
    for (const TileCost& c : kTailTiles)
      consider(kPairTiles[2].at(full, kbs) + c.at(waves(rest * (256 / c.width), pairs), kbs), true, full * pairs, c.width);
  }
  // Two rows of tiles at most and K long enough to be worth sharing: split over clusters, as far as that leaves SMs for
  // the kernel behind to be resident early.  Not by cost: one launch alone says little about the chain (12 layers, us:
  // 128 rows 446 -> 381, 256 rows 481 -> 441; with 4 CTAs for each of 36 or 48 tiles 428, for each of the 36 tiles of 384 rows
  // 495 -> 531).  Alone, weights from HBM, us, tiles / clusters: 128 rows 768 x 768 5.9 / 4.8, 3072 x 768 6.3 / 5.6, 768 x 3072
  // 13.1 / 5.9, 1024 x 4096 16.4 / 7.7; 256 rows 2304 x 768 6.0 / 5.3, 768 x 3072 13.0 / 6.8.
  // Left out where the split alone is slower: many pairs of CTAs that read the same few lines of A (columns x K: 64 rows
  // 4736 x 512 4.51 / 4.86, 4096 x 512 4.54 / 4.68, 4736 x 768 5.40 / 5.57, but 4096 x 768 5.39 / 5.23, 4736 x 1024 6.25 / 5.50;
  // 32 rows 3072 x 768 5.17 / 5.33, 2560 x 1536 7.63 / 8.37, but 2304 x 768 5.19 / 4.53, 3072 x 3072 12.47 / 8.68), and eight
  // blocks of K of few rows (32 rows 768 x 512 3.79 / 3.93, 1 row 1536 x 512 3.87 / 4.02, but 32 rows 768 x 640 4.15 / 3.89).
  if (M <= 2 * kBM && K >= (M < 64 ? 10 : 8) * kBK) {
    const int tiles = mt * (N / kClusterWidth);
    const int cluster = tiles * 8 <= 96 ? 8 : tiles * 4 <= 128 ? 4 : tiles * 2 <= sms ? 2 : 0;
    const bool slower = cluster == 2 && ((M < 64 && K < 32 * kBK && tiles > 36) ||
                                         (M < 96 && K < 16 * kBK && tiles > (K < 12 * kBK ? 56 : 64)));
    if (cluster && !slower) best = GemmPlan{false, 0, kClusterWidth, 1, 3.0, cluster};
  }
  return best;
}

rt_status run_gemm(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi, int dtype,
                   cudaStream_t st, const gemm_detail::QkvEpilogue& extra, const GemmPlan& plan) {
  const bool bf = dtype == RT_BF16;
  if (plan.cluster) return gemm_cluster_dispatch(c, a, w, bias, M, N, K, epi, bf, st, extra, plan.cluster);
  if (plan.pair) return gemm_pair_dispatch(c, a, w, bias, M, N, K, epi, bf, st, extra, plan.main_tiles, plan.width);
  if (plan.width == 256) return bf ? launch_epi<256, true>(c, a, w, bias, M, N, K, epi, st, extra)
                                   : launch_epi<256, false>(c, a, w, bias, M, N, K, epi, st, extra);
  if (plan.width == 128) return bf ? launch_epi<128, true>(c, a, w, bias, M, N, K, epi, st, extra)
                                   : launch_epi<128, false>(c, a, w, bias, M, N, K, epi, st, extra);
  return bf ? launch_epi<64, true>(c, a, w, bias, M, N, K, epi, st, extra)
            : launch_epi<64, false>(c, a, w, bias, M, N, K, epi, st, extra);
}

rt_status gemm_checked(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epilogue,
                       int dtype, void* stream, const gemm_detail::QkvEpilogue& extra) {
  RT_REQUIRE(c && a && w, RT_ERR_INVALID, "gemm: null pointer");
  RT_REQUIRE(M >= 0 && N > 0 && K > 0 && N % 64 == 0 && K % 64 == 0, RT_ERR_INVALID,
             "gemm: need N %% 64 == 0 and K %% 64 == 0 (got M=%d N=%d K=%d)", M, N, K);
  RT_REQUIRE(epilogue == RT_EPI_NONE || bias != nullptr, RT_ERR_INVALID, "gemm: epilogue needs a bias vector");
  RT_REQUIRE(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(bias)) &
              15u) == 0 && (reinterpret_cast<uintptr_t>(c) & 31u) == 0,
             RT_ERR_INVALID, "gemm: A, W and bias must be 16-byte aligned, C 32-byte aligned");
  RT_REQUIRE(dtype == RT_F16 || dtype == RT_BF16, RT_ERR_INVALID, "gemm: unknown dtype %d", dtype);
  if (M == 0) return RT_OK;
  return run_gemm(c, a, w, bias, M, N, K, epilogue, dtype, static_cast<cudaStream_t>(stream), extra, plan_gemm(M, N, K, 1, false));
}

rt_status gemm_qkv_checked(void* q, void* k, void* v, const void* a, const void* w, const void* bias,
                           const int32_t* block_seq_dev, int M, int heads, int K, float q_scale, int dtype, void* stream,
                           bool settled_w) {
  RT_REQUIRE(q && k && v && a && w && bias && block_seq_dev, RT_ERR_INVALID, "gemm_qkv: null pointer");
  const int N = 3 * heads * 64;
  RT_REQUIRE(M >= 0 && M % 64 == 0 && heads > 0 && K > 0 && K % 64 == 0, RT_ERR_INVALID,
             "gemm_qkv: need M %% 64 == 0 and K %% 64 == 0 (got M=%d heads=%d K=%d)", M, heads, K);
  RT_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
               reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(bias)) &
              31u) == 0,
             RT_ERR_INVALID, "gemm_qkv: pointers must be 32-byte aligned");
  RT_REQUIRE(dtype == RT_F16 || dtype == RT_BF16, RT_ERR_INVALID, "gemm_qkv: unknown dtype %d", dtype);
  if (M == 0) return RT_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  QkvEpilogue e{nullptr, (uint16_t*)q, (uint16_t*)k, (uint16_t*)v, reinterpret_cast<const int2*>(block_seq_dev), heads,
                q_scale, 1, settled_w};
  // every tile width keeps a 32-column chunk inside one head
  return run_gemm(nullptr, a, w, bias, M, N, K, kEpiQkv, dtype, st, e, plan_gemm(M, N, K, 1, false));
}

}  // namespace rt

using namespace rt;

extern "C" rt_status rt_gemm(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epilogue,
                             int dtype, void* stream) {
  RT_REQUIRE(epilogue == RT_EPI_NONE || epilogue == RT_EPI_BIAS || epilogue == RT_EPI_BIAS_GELU, RT_ERR_INVALID,
             "gemm: unknown epilogue %d", epilogue);
  return gemm_checked(c, a, w, bias, M, N, K, epilogue, dtype, stream, gemm_detail::QkvEpilogue{});
}

extern "C" rt_status rt_gemm_residual(void* c, const void* a, const void* w, const void* bias, const void* residual,
                                      int M, int N, int K, int dtype, void* stream) {
  RT_REQUIRE(residual != nullptr && (reinterpret_cast<uintptr_t>(residual) & 15u) == 0, RT_ERR_INVALID,
             "gemm_residual: residual must be a 16-byte aligned device pointer");
  gemm_detail::QkvEpilogue e{};
  e.residual = static_cast<const uint16_t*>(residual);
  return gemm_checked(c, a, w, bias, M, N, K, RT_EPI_BIAS_RESIDUAL, dtype, stream, e);
}

extern "C" rt_status rt_gemm_qkv(void* q, void* k, void* v, const void* a, const void* w, const void* bias,
                                 const int32_t* block_seq_dev, int M, int heads, int K, float q_scale, int dtype,
                                 void* stream) {
  return gemm_qkv_checked(q, k, v, a, w, bias, block_seq_dev, M, heads, K, q_scale, dtype, stream, false);
}
