// Two-CTA (cta_group::2) variant of the tcgen05 GEMM: a cluster of two CTAs on neighbouring
// SMs computes one output tile of 256 rows and 64, 128, 192 or 256 columns (one launch may mix whole waves of
// 256 columns with narrower tiles for the rest, see plan_gemm).  Each CTA loads its own 128 rows of A and half of
// the tile's rows of W per 64-wide K slice (256 columns: 32 KB instead of the 48 KB a single-CTA 128 x 256 tile
// needs for the same MMA work), the leader CTA issues the M=256 K=16 MMAs for the pair, and each CTA drains its own
// 128 accumulator rows.  The single-CTA kernel is bound by the
// L2 -> shared-memory traffic of its operand tiles; the pair moves a third less per FLOP.
//
// No TMA multicast is used: both CTAs issue plain (cta_group::2) loads of their own tiles
// whose byte counts land on the leader's barrier; tcgen05.commit multicasts the "slot free"
// and "accumulator ready" arrivals to both CTAs.
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
int gemm_sm_count();  // gemm_sm100.cu
namespace {

using namespace ptx;
using namespace gemm_detail;

constexpr int kTileM = 256, kTileN = 256, kBK = 64;
constexpr int kStages = 6;
constexpr int kABytes = 128 * kBK * 2;  // this CTA's rows of A
constexpr int kBBytes = 128 * kBK * 2;  // this CTA's rows of W
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kThreads = 320;           // warp 0 TMA, warp 1 MMA (leader only), warps 2-9 epilogue
constexpr int kEpilogueThreads = 256;
constexpr int kTmemCols = 512;          // two 256-column accumulators
constexpr int kOutBytes = 32 * 64 * 2;   // one epilogue warp's output box
constexpr int kSmemBytes = kStages * kStageBytes + 8 * kOutBytes + 1024 + 256;
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");

template <bool BF16, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_wt, const __grid_constant__ CUtensorMap map_c,
                 const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, int main_tiles, int tail_w, uint16_t* __restrict__ C, const uint16_t* __restrict__ bias, int M, int N, int K, int* error_flag,
                 QkvEpilogue qkv) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_stage = smem + kStages * kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + 8 * kOutBytes);
  uint64_t* full = bars;                  // leader's copy is the one in use
  uint64_t* empty = bars + kStages;       // each CTA waits on its own copy
  uint64_t* acc_full = bars + 2 * kStages;
  uint64_t* acc_empty = acc_full + 2;     // leader's copy collects both CTAs' epilogue threads
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  RT_PDL_LAUNCH_DEPENDENTS();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const int n_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);  // their fetch overlaps the end of the kernel before, too
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_wt);
    prefetch_tensormap(&map_c);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 2 * kEpilogueThreads);
    }
    *cta_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();  // the peer's barriers exist before anything remote touches them
  cluster_wait();
  tc_fence_after_sync();
  const int n_tiles_m = (M + kTileM - 1) / kTileM;
  const int tail_n = N / tail_w;                      // tiles of tail_w columns per row block
  const int tail0 = main_tiles ? main_tiles * (kTileN / tail_w) : 0;  // of these, covered by the main tiles
  const int mn_tiles = main_tiles + n_tiles_m * tail_n - tail0;
  const int splits = EPI == kEpiPartial ? qkv.splits : 1;
  const int n_tiles = mn_tiles * splits;
  const int k_blocks = K / kBK;
  struct Tile {
    int m0, n0, width, kb0, kb1, part;
  };
  // tile t: 256 columns wide up to main_tiles, then tail_w; over K blocks [kb0, kb1) of part t / mn_tiles
  auto tile_of = [&](int t) {
    Tile r;
    r.part = EPI == kEpiPartial ? t / mn_tiles : 0;
    const int u = EPI == kEpiPartial ? t % mn_tiles : t;
    const bool main = u < main_tiles;
    const int per_row = main ? N / kTileN : tail_n;
    const int i = main ? u : u - main_tiles + tail0;
    r.width = main ? kTileN : tail_w;
    r.m0 = (i / per_row) * kTileM;
    r.n0 = (i % per_row) * r.width;
    r.kb0 = EPI == kEpiPartial ? r.part * k_blocks / splits : 0;
    r.kb1 = EPI == kEpiPartial ? (r.part + 1) * k_blocks / splits : k_blocks;
    return r;
  };

  // W of the first ring fill, where nothing in flight writes it: it comes from HBM while the kernel before still runs
  uint32_t w_ahead = 0;
  if (qkv.settled_w && threadIdx.x == 0) {
    const Tile tl = tile_of(pair);
    const CUtensorMap* mw = pair % mn_tiles < main_tiles ? &map_w : &map_wt;
    for (; w_ahead < kStages && tl.kb0 + static_cast<int>(w_ahead) < tl.kb1; ++w_ahead) {
      if (rank == 0) mbar_arrive_expect_tx(&full[w_ahead], 2 * (kABytes + (tl.width / 2) * kBK * 2));
      tma_load_2d_pair(smem + w_ahead * kStageBytes + kABytes, mw, (tl.kb0 + w_ahead) * kBK,
                       tl.n0 + rank * (tl.width / 2), &full[w_ahead]);
    }
  }
  RT_PDL_WAIT();  // operands and the output buffer belong to the previous kernel until here
  const uint32_t tmem_base = *tmem_slot;
  AbortCtx ab{cta_abort, error_flag};

  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer (both CTAs)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < n_tiles && ok; t += n_pairs) {
        const Tile tl = tile_of(t);
        const int m0 = tl.m0 + rank * 128;
        const int n0 = tl.n0 + rank * (tl.width / 2);
        const CUtensorMap* mw = t % mn_tiles < main_tiles ? &map_w : &map_wt;
        const uint32_t bytes = 2 * (kABytes + (tl.width / 2) * kBK * 2);  // of both CTAs
        for (int kb = tl.kb0; kb < tl.kb1; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, ab, 111)) { ok = false; break; }
          uint8_t* sa = smem + s * kStageBytes;
          if (rank == 0 && it >= w_ahead) mbar_arrive_expect_tx(&full[s], bytes);
          tma_load_2d_pair(sa, &map_a, kb * kBK, m0, &full[s]);
          if (it >= w_ahead) tma_load_2d_pair(sa + kABytes, mw, kb * kBK, n0, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer (leader CTA)
    // The whole warp walks the loop and one elected lane issues: descriptors and loop state are then
    // warp-uniform values, which the tensor-core instructions take directly (inside a single-lane branch
    // every descriptor is moved over from a per-thread register first, and that serial latency per
    // 64-wide K slice is of the order of the slice's 512 clocks of MMA work).
    if (rank == 0) {
      const bool leader = elect_one();
      const uint32_t smem_base = smem_u32(smem);
      uint32_t it = 0, tile_it = 0;
      bool ok = true;
      for (int t = pair; t < n_tiles && ok; t += n_pairs, ++tile_it) {
        const int a = tile_it & 1;
        const uint32_t aph = (tile_it >> 1) & 1;
        if (!mbar_wait(&acc_empty[a], aph ^ 1, ab, 112)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + a * kTileN;
        const Tile tl = tile_of(t);
        const uint32_t idesc = make_idesc_f16(kTileM, tl.width, BF16 ? 1 : 0, false);
        for (int kb = tl.kb0; kb < tl.kb1; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1;
          if (!mbar_wait(&full[s], ph, ab, 113)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_base + s * kStageBytes;
          const uint64_t da = make_smem_desc_sw128(sa);
          const uint64_t db = make_smem_desc_sw128(sa + kABytes);
          if (leader) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              mma_ss_pair(d_tmem, da + (k * 32 >> 4), db + (k * 32 >> 4), idesc, kb > tl.kb0 || k > 0 ? 1u : 0u);
            tc_commit_pair(&empty[s], 3);  // slot free in both CTAs
          }
          __syncwarp();
        }
        if (ok && leader) tc_commit_pair(&acc_full[a], 3);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue warps 2..9 (both CTAs)
    const int quarter = warp & 3;
    const int chunk0 = (warp - 2) >> 2;
    const int row_in_tile = rank * 128 + quarter * 32;
    const uint32_t leader_acc_empty[2] = {leader_smem_u32(&acc_empty[0]), leader_smem_u32(&acc_empty[1])};
    uint32_t tile_it = 0;
    bool ok = true;
    for (int t = pair; t < n_tiles && ok; t += n_pairs, ++tile_it) {
      const int a = tile_it & 1;
      const uint32_t aph = (tile_it >> 1) & 1;
      const Tile tl = tile_of(t);
      if (!mbar_wait(&acc_full[a], aph, ab, 114)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * kTileN;
      auto drained = [&]() {
        tc_fence_before_sync();
        mbar_arrive_cluster(leader_acc_empty[a]);
      };
      if constexpr (EPI == kEpiPartial) {
        uint16_t* c_part = C + 2 * static_cast<size_t>(tl.part) * M * N;  // fp32 parts
        epilogue_row<BF16, EPI>(tl.width, taddr, tl.m0 + row_in_tile + lane, tl.n0, chunk0, M, N, c_part, bias, qkv);
        drained();
      } else {
        epilogue_tma<BF16, EPI>(tl.width, taddr, tl.m0 + row_in_tile, lane, tl.n0, chunk0, M, N, bias, qkv,
                                out_stage + (warp - 2) * kOutBytes, &map_c, &map_k, &map_v, drained);
      }
    }
    if (lane == 0) tma_store_wait<0>();  // the staging buffer is read and the output written before the CTA ends
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();  // nobody leaves while its peer may still read its shared memory or signal its barriers
  cluster_wait();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

template <bool BF16, int EPI>
rt_status launch_pair(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, cudaStream_t st,
                      const QkvEpilogue& qkv, int main_tiles, int tail_w) {
  CUtensorMap ma, mw, mwt, mc, mk, mv;
  RT_TRY(make_tensor_map_2d(&ma, a, M, K, K, 128, kBK, true));
  RT_TRY(make_tensor_map_2d(&mw, w, N, K, K, 128, kBK, true));
  RT_TRY(make_tensor_map_2d(&mwt, w, N, K, K, tail_w / 2, kBK, true));
  if constexpr (EPI == kEpiQkv) {
    const uint64_t rows = static_cast<uint64_t>(M) * qkv.heads;
    RT_TRY(make_tensor_map_2d(&mc, qkv.q, rows, 64, 64, 32, 64, true));
    RT_TRY(make_tensor_map_2d(&mk, qkv.k, rows, 64, 64, 32, 64, true));
    RT_TRY(make_tensor_map_2d(&mv, qkv.v, rows, 64, 64, 32, 64, true));
  } else {
    if constexpr (EPI == kEpiPartial) mc = ma;  // fp32 parts are stored directly
    else RT_TRY(make_tensor_map_2d(&mc, c, M, N, N, 32, 64, true));
    mk = mv = mc;
  }
  auto kern = gemm_pair_kernel<BF16, EPI>;
  RT_TRY(ensure_kernel_smem(reinterpret_cast<const void*>(kern), kSmemBytes, false));
  int* err = device_error_word();
  RT_REQUIRE(err != nullptr, RT_ERR_CUDA, "gemm: cannot allocate the device error word");
  const int sms = gemm_sm_count();
  const int mn = main_tiles + ((M + kTileM - 1) / kTileM) * (N / tail_w) - (main_tiles ? main_tiles * (kTileN / tail_w) : 0);
  const int tiles = mn * (EPI == kEpiPartial ? qkv.splits : 1);
  const int pairs = std::min(tiles, sms / 2);
  // Only where the launch fills the chip.  12 layers: 4096 tokens 1177 -> 1173 us, 5312 1279 -> 1272, 1024 wide (24
  // layers) 4096 tokens 3462 -> 3421; with CTAs that wait on free SMs for longer, 256 tokens 435 -> 437, 1024 wide 1024
  // tokens 1544 -> 1550.
  QkvEpilogue args = qkv;
  args.settled_w = qkv.settled_w && pairs == sms / 2;
  RT_CHECK_CUDA(launch_kernel(kern, dim3(2 * pairs), dim3(kThreads), kSmemBytes, st, ma, mw, mwt, mc, mk, mv, main_tiles, tail_w, (uint16_t*)c,
                              (const uint16_t*)bias, M, N, K, err, args));
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

}  // namespace

// main_tiles tiles of 256 columns, the rest of the output in tiles of tail_w (GemmPlan).
rt_status gemm_pair_dispatch(void* c, const void* a, const void* w, const void* bias, int M, int N, int K, int epi,
                             bool bf16, cudaStream_t st, const gemm_detail::QkvEpilogue& qkv, int main_tiles, int tail_w) {
  switch (epi) {
    case RT_EPI_NONE:
      return bf16 ? launch_pair<true, RT_EPI_NONE>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w)
                  : launch_pair<false, RT_EPI_NONE>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w);
    case RT_EPI_BIAS:
      return bf16 ? launch_pair<true, RT_EPI_BIAS>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w)
                  : launch_pair<false, RT_EPI_BIAS>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w);
    case RT_EPI_BIAS_GELU:
      return bf16 ? launch_pair<true, RT_EPI_BIAS_GELU>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w)
                  : launch_pair<false, RT_EPI_BIAS_GELU>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w);
    case RT_EPI_BIAS_RESIDUAL:
      return bf16 ? launch_pair<true, RT_EPI_BIAS_RESIDUAL>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w)
                  : launch_pair<false, RT_EPI_BIAS_RESIDUAL>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w);
    case gemm_detail::kEpiPartial:
      return bf16 ? launch_pair<true, gemm_detail::kEpiPartial>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w)
                  : launch_pair<false, gemm_detail::kEpiPartial>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w);
    case gemm_detail::kEpiQkv:
      return bf16 ? launch_pair<true, gemm_detail::kEpiQkv>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w)
                  : launch_pair<false, gemm_detail::kEpiQkv>(c, a, w, bias, M, N, K, st, qkv, main_tiles, tail_w);
  }
  return fail(RT_ERR_INVALID, "gemm: unknown epilogue %d", epi);
}

}  // namespace rt
