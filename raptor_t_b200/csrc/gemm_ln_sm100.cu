// Projection GEMM with the whole residual + bias + LayerNorm epilogue fused in:
//   out[M][N] = LayerNorm(A[M][K] W[N][K]^T + bias + residual) * gamma + beta,   N = 768 or 1024.
//
// The two N = hidden projections of a layer (attention output and FFN down) are each followed
// by a LayerNorm over the whole row (layers/multi_headed_attention.cpp:206-210,
// layers/bert_output.cpp:19-23).  A 256 x 256 CTA-pair tile holds only a quarter or a third of
// a row, so here a CLUSTER of N/256 CTA pairs owns a block of 256 complete rows: pair p computes
// columns [256 p, 256 p + 256) with the same cta_group::2 main loop as gemm_pair_sm100.cu, and
// the epilogue
//   1. reads the fp32 accumulator into registers once, adds bias and residual there (never rounded to 16 bits), and
//      forms the mean and the squared deviations of the thread's columns,
//   2. sends both to every CTA of the cluster that holds the same rows (distributed shared memory:
//      st.async, whose bytes the receiver's mbarrier counts),
//   3. waits for all partials of its rows, forms mean and 1/sigma, normalises its columns and
//      stores the 16-bit result.
// Residual and result travel as 32-row x 64-column TMA boxes through 4 KB of shared memory per epilogue warp, bias,
// gamma and beta sit in shared memory.  The epilogue is a chain of latencies (SM clocks per tile, 20480 rows: pass 1
// 4300, exchange 1550-1800, pass 2 3500, the passes before their packed-pair arithmetic) and outlasts a K = 768 main
// loop; one under K = 3072 is hidden.  Against
// row-wise loads and stores by the threads and a second pass over TMEM: K = 3072, 8192 rows 40.2 -> 36.8 us.
// The pre-LayerNorm sum therefore never reaches HBM, the separate LayerNorm launch disappears,
// and one 16-bit rounding per sub-layer with it.  No TMA multicast is used anywhere.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>

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

constexpr int kBK = 64;
constexpr int kABytes = 128 * kBK * 2;  // this CTA's rows of A
constexpr int kThreads = 384;           // warp 0 TMA, warp 1 MMA (pair leaders only), warps 4-11 epilogue; 2, 3 lend registers
constexpr int kEpilogueThreads = 256;
// An epilogue thread holds 128 fp32 columns of its row.  The kernel is launched with 168 registers per thread
// (384 x 168 = 64512); the first warpgroup keeps 72 and the other two take 216: 128 x 72 + 256 x 216 = 64512.
constexpr int kRegsIssue = 72;
constexpr int kRegsEpilogue = 216;
constexpr int kTmemCols = 512;          // two 256-column accumulators
constexpr int kMaxNT = 4;               // N up to 1024
// row statistics: [accumulator parity][partial slot = n-tile * 2 + column-parity warp][row of this CTA]
// {mean, squared deviations from it}
constexpr int kStatsBytes = 2 * (2 * kMaxNT) * 128 * 8;
constexpr int kDrainTries = 1 << 16;    // each suspends the thread for some time
constexpr int kBoxBytes = 32 * 64 * 2;  // residual / result box of one epilogue warp
// Shape of a cluster: NT column tiles of TW columns, each computed by a CTA pair (256 rows) or by one CTA (128 rows).
template <bool PAIR, int NT, int TW>
struct LnCfg {
  static constexpr int kN = NT * TW;
  static constexpr int kCtas = PAIR ? 2 * NT : NT;
  static constexpr int kRows = PAIR ? 256 : 128;
  static constexpr int kWRows = PAIR ? TW / 2 : TW;  // rows of W that one CTA loads
  static constexpr int kStageBytes = kABytes + kWRows * kBK * 2;
  static constexpr int kStages = kStageBytes <= 32 * 1024 ? 5 : 4;
  static constexpr int kParamBytes = 3 * TW * 4;  // bias, gamma, beta of this CTA's columns, fp32
  static constexpr int kSmemBytes = kStages * kStageBytes + 8 * kBoxBytes + kStatsBytes + kParamBytes + 1024 + 256;
};

__device__ __forceinline__ uint32_t map_to_rank(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// Asynchronous store of two floats to a CTA of the cluster; its 8 bytes are counted on that CTA's barrier, so the
// sender needs neither a release fence nor an arrival of its own.
__device__ __forceinline__ void st_async_f2(uint32_t cluster_addr, float a, float b, uint32_t cluster_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(
                   cluster_addr),
               "f"(a), "f"(b), "r"(cluster_bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_acquire_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait with cluster-scope acquire (the partial sums were written by other CTAs)
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, const AbortCtx& ab, int where) {
  if (mbar_try_wait_acquire_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait_acquire_cluster(bar, parity)) return true;
    if (*ab.cta_flag) return false;
    if (clock64() - t0 > ab.limit) break;
  }
  *ab.cta_flag = 1;
  atomicCAS(ab.global_flag, 0, where);
  return false;
}
// packed fp32 pairs: half the issue slots of the scalar forms
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// TMA load into THIS CTA's shared memory whose bytes are counted on the pair leader's barrier
__device__ __forceinline__ void tma_load_2d_to_leader(void* smem_dst, const CUtensorMap* m, int x, int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}

template <bool BF16, bool PAIR, int NT, int TW>
__global__ void __launch_bounds__(kThreads, 1)
gemm_ln_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               const __grid_constant__ CUtensorMap map_res, const __grid_constant__ CUtensorMap map_out,
               const uint16_t* __restrict__ bias, const uint16_t* __restrict__ gamma, const uint16_t* __restrict__ beta,
               int M, int K, float eps, bool settled_w, int* error_flag) {
  using Cfg = LnCfg<PAIR, NT, TW>;
  constexpr int N = Cfg::kN, kStages = Cfg::kStages, kStageBytes = Cfg::kStageBytes;
  constexpr int kTileN = 256;  // TMEM columns between the two accumulators
  constexpr int kSlots = 2 * NT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* boxes = smem + kStages * kStageBytes;                             // [8 epilogue warps]
  float2* stats = reinterpret_cast<float2*>(boxes + 8 * kBoxBytes);          // [2][2 * kMaxNT][128]
  float* params = reinterpret_cast<float*>(boxes + 8 * kBoxBytes + kStatsBytes);  // [3][TW]
  uint64_t* bars = reinterpret_cast<uint64_t*>(boxes + 8 * kBoxBytes + kStatsBytes + Cfg::kParamBytes);
  uint64_t* full = bars;                  // the pair leader's copy is the one in use
  uint64_t* empty = bars + kStages;       // each CTA waits on its own copy
  uint64_t* acc_full = bars + 2 * kStages;
  uint64_t* acc_empty = acc_full + 2;     // the pair leader's copy collects both CTAs' epilogue threads
  uint64_t* stats_full = acc_empty + 2;   // every CTA's own: partial sums of its rows from all NT column tiles
  uint64_t* res_full = stats_full + 2;    // one per epilogue warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + 8);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  RT_PDL_LAUNCH_DEPENDENTS();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();               // 0 .. kCtas - 1
  const uint32_t tile = PAIR ? rank >> 1 : rank;         // column tile
  const uint32_t hrow = PAIR ? rank & 1 : 0;             // which 128 of a pair's 256 rows this CTA holds
  const uint32_t leader = PAIR ? rank & ~1u : rank;      // cluster rank of the MMA-issuing CTA
  const int cluster_id = blockIdx.x / Cfg::kCtas;
  const int n_clusters = gridDim.x / Cfg::kCtas;
  auto peer_of = [&](int t) { return PAIR ? static_cast<uint32_t>(2 * t) + hrow : static_cast<uint32_t>(t); };

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);  // their fetch overlaps the end of the kernel before, too
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_res);
    prefetch_tensormap(&map_out);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], (PAIR ? 2 : 1) * kEpilogueThreads);
      mbar_init(&stats_full[a], 1);  // one local arrival that announces the bytes of all column tiles
    }
    for (int w = 0; w < 8; ++w) mbar_init(&res_full[w], 1);
    *cta_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_slot, kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, kTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();  // every peer's barriers exist before anything remote touches them
  cluster_wait();
  tc_fence_after_sync();
  const int n_tiles_m = (M + Cfg::kRows - 1) / Cfg::kRows;
  const int k_blocks = K / kBK;
  const int w_row0 = tile * TW + hrow * Cfg::kWRows;
  // W of the first ring fill, where nothing in flight writes it: it comes from HBM while the kernel before still runs
  // (12 layers, 4096 tokens: with the same in gemm_pair_sm100.cu 1158 -> 1145 us)
  uint32_t w_ahead = 0;
  if (settled_w && threadIdx.x == 0) {
    for (; w_ahead < kStages && static_cast<int>(w_ahead) < k_blocks; ++w_ahead) {
      uint8_t* sw = smem + w_ahead * kStageBytes + kABytes;
      if constexpr (PAIR) {
        if (hrow == 0) mbar_arrive_expect_tx(&full[w_ahead], 2 * kStageBytes);
        tma_load_2d_to_leader(sw, &map_w, w_ahead * kBK, w_row0, map_to_rank(&full[w_ahead], leader));
      } else {
        mbar_arrive_expect_tx(&full[w_ahead], kStageBytes);
        tma_load_2d(sw, &map_w, w_ahead * kBK, w_row0, &full[w_ahead]);
      }
    }
  }
  RT_PDL_WAIT();  // operands, parameters, residual and the output buffer belong to the previous kernel until here
  const uint32_t tmem_base = *tmem_slot;
  AbortCtx ab{cta_abort, error_flag};

  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer (every CTA)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = cluster_id; t < n_tiles_m && ok; t += n_clusters) {
        const int m0 = t * Cfg::kRows + hrow * 128;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, ab, 121)) { ok = false; break; }
          uint8_t* sa = smem + s * kStageBytes;
          if constexpr (PAIR) {
            if (hrow == 0 && it >= w_ahead) mbar_arrive_expect_tx(&full[s], 2 * kStageBytes);  // both CTAs' bytes
            const uint32_t leader_bar = map_to_rank(&full[s], leader);
            tma_load_2d_to_leader(sa, &map_a, kb * kBK, m0, leader_bar);
            if (it >= w_ahead) tma_load_2d_to_leader(sa + kABytes, &map_w, kb * kBK, w_row0, leader_bar);
          } else {
            if (it >= w_ahead) mbar_arrive_expect_tx(&full[s], kStageBytes);
            tma_load_2d(sa, &map_a, kb * kBK, m0, &full[s]);
            if (it >= w_ahead) tma_load_2d(sa + kABytes, &map_w, kb * kBK, w_row0, &full[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer (pair leaders)
    // the whole warp walks the loop, one elected lane issues (see gemm_pair_sm100.cu)
    if (hrow == 0) {
      constexpr uint32_t idesc = make_idesc_f16(Cfg::kRows, TW, BF16 ? 1 : 0, false);
      const uint16_t pair_mask = static_cast<uint16_t>(3u << leader);
      const bool elected = elect_one();
      const uint32_t smem_base = smem_u32(smem);
      uint32_t it = 0, tile_it = 0;
      bool ok = true;
      for (int t = cluster_id; t < n_tiles_m && ok; t += n_clusters, ++tile_it) {
        const int a = tile_it & 1;
        const uint32_t aph = (tile_it >> 1) & 1;
        if (!mbar_wait(&acc_empty[a], aph ^ 1, ab, 122)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + a * kTileN;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1;
          if (!mbar_wait(&full[s], ph, ab, 123)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_base + s * kStageBytes;
          const uint64_t da = make_smem_desc_sw128(sa);
          const uint64_t db = make_smem_desc_sw128(sa + kABytes);
          if (elected) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              if constexpr (PAIR) mma_ss_pair(d_tmem, da + (k * 32 >> 4), db + (k * 32 >> 4), idesc, (kb | k) ? 1u : 0u);
              else mma_ss(d_tmem, da + (k * 32 >> 4), db + (k * 32 >> 4), idesc, (kb | k) ? 1u : 0u);
            }
            if constexpr (PAIR) tc_commit_pair(&empty[s], pair_mask);  // slot free in both CTAs of the pair
            else tc_commit(&empty[s]);
          }
          __syncwarp();
        }
        if (ok && elected) {
          if constexpr (PAIR) tc_commit_pair(&acc_full[a], pair_mask);
          else tc_commit(&acc_full[a]);
        }
        __syncwarp();
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------- epilogue warps 4..11 (every CTA)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
    const int quarter = warp & 3;        // TMEM lane quarter
    const int set = (warp - 4) >> 2;     // this warp takes the 64-column boxes set, set + 2 of its 32 rows
    constexpr int kBoxes = TW / 64;
    const bool two_boxes = set + 2 < kBoxes;
    const int row_local = quarter * 32 + lane;
    const uint32_t leader_acc_empty[2] = {map_to_rank(&acc_empty[0], leader), map_to_rank(&acc_empty[1], leader)};
    const int n0 = tile * TW;
    const int slot = tile * 2 + set;
    uint8_t* const box = boxes + (warp - 4) * kBoxBytes;
    uint8_t* const line = box + lane * 128;
    const int swz = lane & 7;
    uint64_t* const my_res = &res_full[warp - 4];
    bool res_on_its_way = false;
    auto row0_of = [&](int t) { return t * Cfg::kRows + static_cast<int>(hrow) * 128 + quarter * 32; };
    auto load_residual = [&](int t, int b) {
      res_on_its_way = true;
      if (lane == 0) {
        mbar_arrive_expect_tx(my_res, kBoxBytes);
        tma_load_2d(box, &map_res, n0 + b * 64, row0_of(t), my_res);
      }
    };
    uint32_t tile_it = 0, res_phase = 0;
    bool ok = true;
    if (cluster_id < n_tiles_m) load_residual(cluster_id, set);
    for (int i = threadIdx.x - 128; i < 3 * TW / 2; i += kEpilogueThreads) {  // under the first main loop
      const uint16_t* src = i < TW / 2 ? bias : i < TW ? gamma : beta;
      reinterpret_cast<float2*>(params)[i] = unpack2<BF16>(reinterpret_cast<const uint32_t*>(src + tile * TW)[i % (TW / 2)]);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueThreads) : "memory");
    for (int t = cluster_id; t < n_tiles_m && ok; t += n_clusters, ++tile_it) {
      const int a = tile_it & 1;
      const uint32_t aph = (tile_it >> 1) & 1;
      if (!mbar_wait(&acc_full[a], aph, ab, 124)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * kTileN;
      // pass 1: x = acc + bias + residual, kept in registers as its distance d from the mean of the thread's first eight
      // columns; sums of d and d^2 over all of them.  That mean is within sqrt(15) deviations of the mean of the
      // thread's 128, whatever the values are, so that sum d^2 - (sum d)^2 / n costs four bits at most, where
      // E[x^2] - mean^2 costs all that a row's mean is above its deviation.  Against that form, 768 columns: 20480 rows
      // K = 768 32.1 -> 33.0 us, K = 3072 80.2 -> 80.8; 5312 rows 22.9 -> 23.0.
      uint64_t sum2 = 0, sq2 = 0, neg_shift = 0;  // packed pairs of fp32
      float shift = 0.f;
      uint32_t x[128];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int b = set + 2 * i;
        if (b < kBoxes) {
          tmem_ld32(taddr + b * 64, x + i * 64);
          tmem_ld32(taddr + b * 64 + 32, x + i * 64 + 32);
          if (!mbar_wait(my_res, res_phase, ab, 126)) ok = false;
          else res_on_its_way = false;
          res_phase ^= ok;
          tc_wait_ld();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 r4 = *reinterpret_cast<const uint4*>(line + ((q ^ swz) << 4));
            const ulonglong2* bv = reinterpret_cast<const ulonglong2*>(params + b * 64 + q * 8);
            const ulonglong2 b01 = bv[0], b23 = bv[1];
            const uint64_t bb[4] = {b01.x, b01.y, b23.x, b23.y};
            const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
            uint64_t y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 rr = unpack2<BF16>(rw[j]);
              const uint32_t* v = x + i * 64 + q * 8 + 2 * j;
              y[j] = f2_add(f2_add(f2_pack(__uint_as_float(v[0]), __uint_as_float(v[1])), bb[j]), f2_pack(rr.x, rr.y));
            }
            if (i == 0 && q == 0) {
              const float2 first = f2_unpack(f2_add(f2_add(y[0], y[1]), f2_add(y[2], y[3])));
              shift = (first.x + first.y) * 0.125f;
              neg_shift = f2_pack(-shift, -shift);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint64_t d = f2_add(y[j], neg_shift);
              sum2 = f2_add(sum2, d);
              sq2 = f2_fma(d, d, sq2);
              const float2 f = f2_unpack(d);
              uint32_t* v = x + i * 64 + q * 8 + 2 * j;
              v[0] = __float_as_uint(f.x);
              v[1] = __float_as_uint(f.y);
            }
          }
          if (i == 0 && set + 2 < kBoxes) {
            __syncwarp();  // every lane has read its line
            if (ok) load_residual(t, set + 2);
          }
        }
      }
      const float2 sums = f2_unpack(sum2), sqs = f2_unpack(sq2);
      const float sum = sums.x + sums.y, own = sum * (two_boxes ? 1.0f / 128 : 1.0f / 64);
      const float own_mean = shift + own, dev = fmaxf(fmaf(-sum, own, sqs.x + sqs.y), 0.f);
      // the accumulator is in registers: the tile after the next may overwrite it
      tc_fence_before_sync();
      mbar_arrive_cluster(leader_acc_empty[a]);
      if (!ok) break;
      // mean and deviations go to every CTA that holds these rows (same hrow, every column tile); a peer cannot be two
      // tiles ahead (its wait for the tile between needs this CTA's), so the barrier is in this tile's phase
      if (warp == 4 && lane == 0) mbar_arrive_expect_tx(&stats_full[a], NT * kEpilogueThreads * 8);
#pragma unroll
      for (int p = 0; p < NT; ++p)
        st_async_f2(map_to_rank(stats + (a * (2 * kMaxNT) + slot) * 128 + row_local, peer_of(p)), own_mean, dev,
                    map_to_rank(&stats_full[a], peer_of(p)));
      if (!mbar_wait_cluster(&stats_full[a], aph, ab, 125)) { ok = false; break; }
      float2 part[kSlots];
      float mean = 0.f, tot_dev = 0.f;
      auto cols = [](int sl) { return 64 * ((kBoxes + 1 - (sl & 1)) / 2); };  // of the warps of this set
#pragma unroll
      for (int sl = 0; sl < kSlots; ++sl) {
        part[sl] = stats[(a * (2 * kMaxNT) + sl) * 128 + row_local];
        mean = fmaf(part[sl].x, static_cast<float>(cols(sl)) / N, mean);
      }
#pragma unroll
      for (int sl = 0; sl < kSlots; ++sl) {  // deviations about the part's mean -> about the row's
        const float d = part[sl].x - mean;
        tot_dev += fmaf(d * d, static_cast<float>(cols(sl)), part[sl].y);
      }
      const float var = tot_dev * (1.0f / N);
      const float rstd = rsqrtf(var + eps);
      // pass 2: normalise this thread's columns, store them box by box
      const int row0 = row0_of(t);
      const uint64_t to_mean = f2_pack(shift - mean, shift - mean), rstd2 = f2_pack(rstd, rstd);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int b = set + 2 * i;
        if (b < kBoxes) {
          if (i > 0) {
            if (lane == 0) tma_store_wait_read<0>();
            __syncwarp();
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const ulonglong2* gv = reinterpret_cast<const ulonglong2*>(params + TW + b * 64 + q * 8);
            const ulonglong2* ev = reinterpret_cast<const ulonglong2*>(params + 2 * TW + b * 64 + q * 8);
            const ulonglong2 g01 = gv[0], g23 = gv[1], e01 = ev[0], e23 = ev[1];
            const uint64_t gg[4] = {g01.x, g01.y, g23.x, g23.y}, ee[4] = {e01.x, e01.y, e23.x, e23.y};
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t* v = x + i * 64 + q * 8 + 2 * j;
              const uint64_t y = f2_mul(f2_add(f2_pack(__uint_as_float(v[0]), __uint_as_float(v[1])), to_mean), rstd2);
              const float2 f = f2_unpack(f2_fma(y, gg[j], ee[j]));
              o[j] = pack2<BF16>(f.x, f.y);
            }
            *reinterpret_cast<uint4*>(line + ((q ^ swz) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && row0 < M) {
            tma_store_2d(&map_out, box, n0 + b * 64, row0);
            tma_store_commit();
          }
        }
      }
      if (t + n_clusters < n_tiles_m) {  // the next row block's first box, under the stores and the main loop
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
        load_residual(t + n_clusters, set);
      }
    }
    // left early (a wait ran out): the CTA must not end under a box that is still on its way to it
    for (int i = 0; res_on_its_way && i < kDrainTries; ++i) res_on_its_way = !mbar_try_wait(my_res, res_phase);
    if (lane == 0) tma_store_wait<0>();  // the boxes are read and the result written before the CTA ends
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();  // nobody leaves while a peer may still write its shared memory or signal its barriers
  cluster_wait();
  if (warp == 1) {
    tc_fence_after_sync();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
}

// As many clusters as the current device keeps resident at once (the kernel is persistent over row blocks).
template <bool BF16, bool PAIR, int NT, int TW>
int resident_clusters() {
  using Cfg = LnCfg<PAIR, NT, TW>;
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n != 0) return n;
  auto kern = gemm_ln_kernel<BF16, PAIR, NT, TW>;
  const int limit = gemm_sm_count() / Cfg::kCtas;
  if (ensure_kernel_smem(reinterpret_cast<const void*>(kern), Cfg::kSmemBytes, false) != RT_OK) return limit;
  cudaLaunchConfig_t q{};
  q.gridDim = dim3(limit * Cfg::kCtas);
  q.blockDim = dim3(kThreads);
  q.dynamicSmemBytes = Cfg::kSmemBytes;
  cudaLaunchAttribute qa[1];
  qa[0].id = cudaLaunchAttributeClusterDimension;
  qa[0].val.clusterDim.x = Cfg::kCtas;
  qa[0].val.clusterDim.y = 1;
  qa[0].val.clusterDim.z = 1;
  q.attrs = qa;
  q.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &q) != cudaSuccess || n <= 0) n = limit;
  cache[dev].store(n, std::memory_order_relaxed);
  return n;
}

template <bool BF16, bool PAIR, int NT, int TW>
rt_status launch_ln(void* out, const void* a, const void* w, const void* bias, const void* residual, const void* gamma,
                    const void* beta, int M, int K, float eps, bool settled_w, cudaStream_t st) {
  using Cfg = LnCfg<PAIR, NT, TW>;
  constexpr int kSmemBytes = Cfg::kSmemBytes;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
  CUtensorMap ma, mw, mr, mo;
  RT_TRY(make_tensor_map_2d(&ma, a, M, K, K, 128, kBK, true));
  RT_TRY(make_tensor_map_2d(&mw, w, Cfg::kN, K, K, Cfg::kWRows, kBK, true));
  RT_TRY(make_tensor_map_2d(&mr, residual, M, Cfg::kN, Cfg::kN, 32, 64, true));
  RT_TRY(make_tensor_map_2d(&mo, out, M, Cfg::kN, Cfg::kN, 32, 64, true));
  auto kern = gemm_ln_kernel<BF16, PAIR, NT, TW>;
  RT_TRY(ensure_kernel_smem(reinterpret_cast<const void*>(kern), kSmemBytes, false));
  int* err = device_error_word();
  RT_REQUIRE(err != nullptr, RT_ERR_CUDA, "gemm_layernorm: cannot allocate the device error word");
  const int m_tiles = (M + Cfg::kRows - 1) / Cfg::kRows;
  const int clusters = std::max(1, std::min(m_tiles, resident_clusters<BF16, PAIR, NT, TW>()));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * Cfg::kCtas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = Cfg::kCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  RT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mw, mr, mo, static_cast<const uint16_t*>(bias),
                                   static_cast<const uint16_t*>(gamma), static_cast<const uint16_t*>(beta), M, K, eps,
                                   settled_w, err));
  count_launch();
  RT_CHECK_CUDA(cudaGetLastError());
  return RT_OK;
}

}  // namespace
}  // namespace rt

namespace rt {
int gemm_layernorm_clusters(int N, bool pairs) {
  if (N == 768) return pairs ? resident_clusters<true, true, 3, 256>() : resident_clusters<true, false, 4, 192>();
  return resident_clusters<true, true, 4, 256>();
}

rt_status gemm_layernorm_checked(void* out_dev, const void* a_dev, const void* w_dev, const void* bias_dev,
                                 const void* residual_dev, const void* gamma_dev, const void* beta_dev, int M, int N, int K,
                                 float eps, int dtype, void* stream, bool settled_w) {
  RT_REQUIRE(out_dev && a_dev && w_dev && bias_dev && residual_dev && gamma_dev && beta_dev, RT_ERR_INVALID,
             "gemm_layernorm: null pointer");
  RT_REQUIRE(N == 768 || N == 1024, RT_ERR_UNSUPPORTED, "gemm_layernorm: N must be 768 or 1024 (got %d)", N);
  RT_REQUIRE(M >= 0 && K > 0 && K % 64 == 0, RT_ERR_INVALID, "gemm_layernorm: need K %% 64 == 0 (got M=%d K=%d)", M, K);
  RT_REQUIRE(dtype == RT_F16 || dtype == RT_BF16, RT_ERR_INVALID, "gemm_layernorm: unknown dtype %d", dtype);
  const uintptr_t all = reinterpret_cast<uintptr_t>(out_dev) | reinterpret_cast<uintptr_t>(a_dev) |
                        reinterpret_cast<uintptr_t>(w_dev) | reinterpret_cast<uintptr_t>(bias_dev) |
                        reinterpret_cast<uintptr_t>(residual_dev) | reinterpret_cast<uintptr_t>(gamma_dev) |
                        reinterpret_cast<uintptr_t>(beta_dev);
  RT_REQUIRE((all & 31u) == 0, RT_ERR_INVALID, "gemm_layernorm: pointers must be 32-byte aligned");
  if (M == 0) return RT_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Clusters of four single CTAs (128 rows x 192 columns each) while all row blocks are resident at once: 36 of them
  // cover 144 SMs, where 16 clusters of three pairs have 96 (K = 3072, 4096 rows: 21.7 against 25.0 us).  Beyond,
  // pairs: they load a third less per FLOP.
  const bool bf = dtype == RT_BF16;
  const int blocks = (M + 127) / 128;
#define RT_LN_LAUNCH(PAIR, NT, TW)                                                                                  \
  (bf ? launch_ln<true, PAIR, NT, TW>(out_dev, a_dev, w_dev, bias_dev, residual_dev, gamma_dev, beta_dev, M, K, eps, settled_w, st) \
      : launch_ln<false, PAIR, NT, TW>(out_dev, a_dev, w_dev, bias_dev, residual_dev, gamma_dev, beta_dev, M, K, eps, settled_w, st))
  if (N == 768) {
    if (blocks <= gemm_layernorm_clusters(N, false)) return RT_LN_LAUNCH(false, 4, 192);
    return RT_LN_LAUNCH(true, 3, 256);
  }
  return RT_LN_LAUNCH(true, 4, 256);
#undef RT_LN_LAUNCH
}
}  // namespace rt

extern "C" rt_status rt_gemm_bias_residual_layernorm(void* out_dev, const void* a_dev, const void* w_dev,
                                                     const void* bias_dev, const void* residual_dev,
                                                     const void* gamma_dev, const void* beta_dev, int M, int N, int K,
                                                     float eps, int dtype, void* stream) {
  return rt::gemm_layernorm_checked(out_dev, a_dev, w_dev, bias_dev, residual_dev, gamma_dev, beta_dev, M, N, K, eps, dtype,
                                    stream, false);
}
