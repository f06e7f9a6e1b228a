// Products of many activation rows on pairs of CTAs: tcgen05.mma.cta_group::2, 256 weight rows x 256 (or 128) activation rows a pair.
//
// With one CTA a tile of 128 x 256 needs 48 KB of operands per 64-wide K block, which at full tensor rate (512 cycles) is 96
// bytes a cycle; an SM takes in about 58 from L2, and that bounded the single-CTA kernel (6144 x 4096 at 4096 rows: 2.4 GB in 182
// us). In a pair each CTA loads its own 128 weight rows and HALF of the activation rows, which both multiply: 32 KB per K
// block. Gated products hold a gate and an up tile of 256 rows, 256 wide where K is long (48 KB per K block of twice the work; both
// accumulators fill the tensor memory, so the epilogue is exposed), else 128 wide with two buffers.
//
// Roles per CTA of 320 threads: warp 0 loads (plain tile loads into its own shared memory, bytes counted on the even CTA's
// barrier), warp 1 of the even CTA issues the MMAs of both, warps 2..9 are the epilogue, two warps per TMEM lane quarter
// with half of the columns each. Freed stages and finished accumulators are announced in both CTAs by the commit; the even CTA's
// issuer waits for the epilogue warps of both.
#include <algorithm>

#include "xpool/gemm_pair.cuh"
#include "xpool/pdl.cuh"
#include "xpool/tensormap.hpp"

namespace xpool {
namespace gemm {

constexpr int kPThreads = 320, kPEpiWarps = 8;
constexpr int kPBudget = 220 * 1024;

struct PairLayout {
  int stages, a_bytes, b_bytes, stage_bytes, total_bytes;
};
__host__ __device__ inline PairLayout pair_layout(int bn, int dual) {
  PairLayout L;
  L.a_bytes = kTileM * kTileK * 2 * (dual ? 2 : 1);
  L.b_bytes = bn / 2 * kTileK * 2;
  L.stage_bytes = L.a_bytes + L.b_bytes;
  L.stages = (kPBudget - 2048) / L.stage_bytes;
  if (L.stages > kMaxStages) L.stages = kMaxStages;
  L.total_bytes = L.stages * L.stage_bytes + 1024 + 512;
  return L;
}

// Tile t of the pair: CTA `rank` owns weight rows m0 .. + 127; the activation rows are the pair's.
__device__ __forceinline__ TileCoord pair_coord(const Problem& p, int t, int rank) {
  TileCoord c;
  c.split = 0;
  c.mn = t;
  c.kb0 = 0;
  c.kbn = k_blocks(p);
  c.out_off = 0;
  if (p.tile_table != nullptr) {
    const int4 e = p.tile_table[2 * t + rank];
    c.m0 = e.y;
    c.n0 = e.z;
    c.row_end = e.w;
    c.w_row0 = e.x * p.w_rows_per_group + e.y;
    return c;
  }
  const int tm = (p.n_out + 2 * kTileM - 1) / (2 * kTileM);
  c.m0 = (t % tm) * 2 * kTileM + rank * kTileM;
  c.n0 = (t / tm) * p.bn;
  c.w_row0 = c.m0;
  c.row_end = p.rows;
  return c;
}

template <bool kWide>
__global__ void __launch_bounds__(kPThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ Problem p, int nacc,
                 uint32_t* status) {
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(sm100::cluster_rank());
  const PairLayout L = pair_layout(p.bn, p.dual);
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Barriers* bar = reinterpret_cast<Barriers*>(tiles + static_cast<size_t>(L.stages) * L.stage_bytes);
  const int acc_cols = p.bn * (p.dual ? 2 : 1);
  constexpr uint32_t kCols = 512;
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      sm100::mbar_init(&bar->full[s], 1);
      sm100::mbar_init(&bar->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      sm100::mbar_init(&bar->acc_full[a], 1);
      sm100::mbar_init(&bar->acc_empty[a], 2 * kPEpiWarps);
    }
    sm100::mbar_fence_init();
  }
  if (warp == 1) {
    sm100::tmem_alloc_pair(&bar->tmem_base, kCols);
    sm100::tmem_relinquish_pair();
  }
  sm100::tc_fence_before_sync();
  __syncthreads();
  sm100::cluster_sync();       // both CTAs' barriers and tensor memory are there
  sm100::tc_fence_after_sync();

  const int pairs = gridDim.x / 2, pair = blockIdx.x / 2;
  // (a table is written by the kernels before this one: its length is read behind the wait)
  auto tile_count = [&] { return p.tile_table != nullptr ? *p.n_tiles / 2 : (p.n_out + 2 * kTileM - 1) / (2 * kTileM) * ((p.rows + p.bn - 1) / p.bn); };
  const uint32_t tiles_addr = sm100::smem_u32(tiles);
  const uint32_t full0 = sm100::smem_u32(&bar->full[0]), empty0 = sm100::smem_u32(&bar->empty[0]);
  const uint32_t stages = static_cast<uint32_t>(L.stages);
  const bool dual = p.dual != 0;

  if (warp == 0) {
    const bool leader = sm100::elect_one();
    const uint64_t tw = reinterpret_cast<uint64_t>(&tmap_w), tx = reinterpret_cast<uint64_t>(&tmap_x);
    const uint64_t pol_w = sm100::l2_policy_evict_normal(), pol_x = sm100::l2_policy_evict_last();
    const uint32_t full_even = sm100::map_rank(full0, 0);
    auto load_w = [&](const TileCoord& c, int kb, uint32_t stage) {
      if (!leader) return;
      if (rank == 0) sm100::mbar_arrive_expect_tx_addr(full0 + stage * 8, 2u * L.stage_bytes);
      const uint32_t dst = tiles_addr + stage * L.stage_bytes;
      sm100::tma_load_2d_pair(dst, tw, full_even + stage * 8, kb * kTileK, c.w_row0, pol_w);
      if (dual) sm100::tma_load_2d_pair(dst + kTileM * kTileK * 2, tw, full_even + stage * 8, kb * kTileK, p.up_offset + c.w_row0, pol_w);
    };
    auto load_x = [&](const TileCoord& c, int kb, uint32_t stage) {
      if (leader)
        sm100::tma_load_2d_pair(tiles_addr + stage * L.stage_bytes + L.a_bytes, tx, full_even + stage * 8, kb * kTileK, c.n0 + rank * (p.bn / 2), pol_x);
    };
    int early = 0;
    if (p.w_static && p.tile_table == nullptr && pair < tile_count()) {
      const TileCoord c = pair_coord(p, pair, rank);
      early = min(c.kbn, L.stages);
      for (int i = 0; i < early; ++i) load_w(c, i, i);
    }
    pdl::wait();
    pdl::release();
    const int tiles_total = tile_count();
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int t = pair; ok && t < tiles_total; t += pairs) {
      const TileCoord c = pair_coord(p, t, rank);
      const uint64_t deadline = sm100::global_timer_ns() + sm100::kPipelineWaitNs;
      for (int i = 0; i < c.kbn; ++i) {
        if (t != pair || i >= early) {
          ok = sm100::mbar_wait_warp(empty0 + stage * 8, phase ^ 1, deadline);
          if (!ok) break;
          load_w(c, i, stage);
        }
        load_x(c, i, stage);
        if (++stage == stages) stage = 0, phase ^= 1;
      }
    }
    if (!ok) {
      record_status(status, kTimeoutProducer);
      __nanosleep(1000000);    // copies in flight get a bounded time to land before the CTAs go
    }
  } else if (warp == 1) {
    pdl::wait();
    pdl::release();
    const int tiles_total = tile_count();
    if (rank == 0) {
      const bool leader = sm100::elect_one();
      const uint32_t idesc = sm100::umma_idesc_bf16(2 * kTileM, static_cast<uint32_t>(p.bn));
      const uint64_t da0 = sm100::umma_desc_sw128(tiles_addr), du0 = sm100::umma_desc_sw128(tiles_addr + kTileM * kTileK * 2);
      const uint64_t db0 = sm100::umma_desc_sw128(tiles_addr + L.a_bytes), dstage = static_cast<uint64_t>(L.stage_bytes >> 4);
      const uint32_t tmem = bar->tmem_base;
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = true;
      for (int t = pair; ok && t < tiles_total; t += pairs) {
        const uint64_t deadline = sm100::global_timer_ns() + sm100::kPipelineWaitNs;
        const int kbn = k_blocks(p);
        ok = sm100::mbar_wait_warp(sm100::smem_u32(&bar->acc_empty[acc]), acc_phase ^ 1, deadline);
        if (!ok) break;
        sm100::tc_fence_after_sync();
        const uint32_t tg = tmem + acc * acc_cols, tu = tg + p.bn;
        uint32_t accum = 0;
        for (int i = 0; i < kbn; ++i) {
          ok = sm100::mbar_wait_warp(full0 + stage * 8, phase, deadline);
          if (!ok) break;
          sm100::tc_fence_after_sync();
          const uint64_t da = da0 + stage * dstage, du = du0 + stage * dstage, db = db0 + stage * dstage;
          if (leader) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              sm100::umma_bf16_pair(tg, da + 2 * k, db + 2 * k, idesc, k > 0 ? 1u : accum);
              if (dual) sm100::umma_bf16_pair(tu, du + 2 * k, db + 2 * k, idesc, k > 0 ? 1u : accum);
            }
            sm100::umma_commit_pair(empty0 + stage * 8);
          }
          accum = 1;
          if (++stage == stages) stage = 0, phase ^= 1;
        }
        if (ok && leader) sm100::umma_commit_pair(sm100::smem_u32(&bar->acc_full[acc]));
        if (++acc == static_cast<uint32_t>(nacc)) acc = 0, acc_phase ^= 1;
      }
      if (!ok) record_status(status, kTimeoutMma);
    }
  } else {
    pdl::wait();
    pdl::release();
    const int tiles_total = tile_count();
    const int ew = warp & 3, half = (warp - 2) >> 2;
    const uint32_t empty_even = sm100::map_rank(sm100::smem_u32(&bar->acc_empty[0]), 0);
    uint32_t acc = 0, acc_phase = 0;
    for (int t = pair; t < tiles_total; t += pairs) {
      const TileCoord c = pair_coord(p, t, rank);
      const uint64_t deadline = sm100::global_timer_ns() + sm100::kPipelineWaitNs;
      if (!sm100::mbar_wait_warp(sm100::smem_u32(&bar->acc_full[acc]), acc_phase, deadline)) {
        record_status(status, kTimeoutEpilogue);
        break;
      }
      sm100::tc_fence_after_sync();
      const uint32_t tmem_acc = bar->tmem_base + acc * acc_cols + (static_cast<uint32_t>(ew * 32) << 16);
      const int f = c.m0 + ew * 32 + lane, cols = min(p.bn, c.row_end - c.n0);
      epilogue_columns<kWide>(p, c, f, c.w_row0 + ew * 32 + lane, tmem_acc, half * (p.bn / 2), min(cols, (half + 1) * (p.bn / 2)), stores_wide<kWide>(p, c.m0 + ew * 32));
      sm100::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive_cluster(empty_even + acc * 8);
      if (++acc == static_cast<uint32_t>(nacc)) acc = 0, acc_phase ^= 1;
    }
  }
  __syncwarp();
  sm100::tc_fence_before_sync();
  __syncthreads();
  sm100::cluster_sync();       // neither CTA's memory goes while the pair's MMAs, arrivals or copies may touch it
  if (warp == 1) {
    sm100::tc_fence_after_sync();
    sm100::tmem_dealloc_pair(bar->tmem_base, kCols);
  }
}

// Pairs that can be resident together: two SMs of a pair belong to one GPC.
static int resident_pairs(int dev, int sms) {
  static int known[64] = {};
  if (dev < 0 || dev >= 64) return 0;
  if (known[dev] == 0) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
      return 0;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(sms / 2 * 2);
    cfg.blockDim = dim3(kPThreads);
    cfg.dynamicSmemBytes = pair_layout(256, 0).total_bytes;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<false>, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return 0;
    }
    known[dev] = n;
  }
  return std::min(known[dev], sms / 2);
}

// us a launch, single CTAs -> pairs:
//                            500 rows         1000 rows        4096 rows
//   4096 x 1024              12.2 -> 12.6     16.2 -> 14.3     38.4 -> 31.4
//   1024 x 3072              16.0 -> 24.4     18.8 -> 24.4     29.7 -> 26.8
//   6144 x 4096              39.2 -> 34.5     64.7 -> 58.6     182 -> 166
//   4096 x 4096              28.7 -> 32.7     37.7 -> 34.3     120 -> 109
//   gate/up 6144 x 1024      16.2 -> 13.4     23.5 -> 18.3     53.6 -> 44.7
//   gate/up 24576 x 4096     112 -> 105       181 -> 164       704 -> 652
// so pairs take a call whose tiles, counted by the rows in them, fill 0.6 of the SMs: with fewer the single-CTA kernel cuts finer.
// Callers that name a tile width, a split or an SM count mean that kernel.
int pair_width(const XpGemmArgs& a, int sms) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (a.tile_table != nullptr) {     // grouped: where a group's rows fill the wide tiles that the caller chose
    const bool fits = a.tile_pairs && a.n_out % (2 * kTileM) == 0 && (a.bn == 128 || a.bn == 256) && a.splits <= 1 && a.num_sms == 0 &&
                      a.smem_limit == 0 && !a.fp8 && !a.w_tiled;
    return fits && resident_pairs(dev, sms) > 0 ? a.bn : 0;
  }
  if (a.fp8 || a.w_tiled || a.batch > 1 || a.splits > 0 || a.bn > 0 || a.num_sms > 0 || a.smem_limit > 0 || a.rows <= 256)
    return 0;
  auto filled = [&](int width) { return static_cast<double>(a.rows) / ((a.rows + width - 1) / width * width); };
  const int width = a.dual && (a.k < 2048 || filled(256) < 0.7) ? 128 : 256;
  const int tiles = (a.n_out + 2 * kTileM - 1) / (2 * kTileM) * ((a.rows + width - 1) / width);
  if (tiles * filled(width) < 0.6 * (sms / 2)) return 0;
  return resident_pairs(dev, sms) > 0 ? width : 0;
}

int pair_launch(const XpGemmArgs& a, Problem p, const CUtensorMap& tmap_w, int width, bool wide_epilogue, int sms) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int resident = resident_pairs(dev, sms);
  CUtensorMap tx;
  if (tmap::cache().get(&tx, a.x, a.rows, a.k, static_cast<uint64_t>(a.ldx > 0 ? a.ldx : a.k) * 2, width / 2, 2) != 0) return -21;
  p.bn = width;
  p.splits = 1;
  const int tiles = p.tile_table != nullptr ? resident : (p.n_out + 2 * kTileM - 1) / (2 * kTileM) * ((p.rows + width - 1) / width);
  const int nacc = width * (p.dual ? 2 : 1) * 2 <= 512 ? 2 : 1;
  const cudaError_t e = pdl::launch(wide_epilogue ? gemm_pair_kernel<true> : gemm_pair_kernel<false>, 2 * std::min(resident, tiles), kPThreads,
                                    pair_layout(width, p.dual).total_bytes, reinterpret_cast<cudaStream_t>(a.stream), 2, tmap_w, tx, p, nacc, a.status);
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}

}  // namespace gemm
}  // namespace xpool
