// Products of up to 16 activation rows: y = x w^T with the weights streamed from memory straight into registers.
//
// Such a product is bound by reading w once, and a launch of a small layer lasts a few microseconds, so what counts is the
// time from launch to the last load and from the last load to the last store. A warp takes 16 features and a slice of K:
// the four lanes that share a feature read 64 contiguous bytes of its row per step, 8 to 16 independent 16-byte loads per
// lane are in flight, and mma.m16n8k16 multiplies the registers as they are (weights on the M axis, eight activation rows on
// the N axis). The order of K inside a step is permuted alike on both operands, so neither goes through shared memory: lane q
// of a feature holds elements 8 q .. 8 q + 7 and calls the first four the columns {2 q, 2 q + 1, 2 q + 8, 2 q + 9} of one mma
// and the last four those of the next. Slices of K are cut between the warps of a CTA and, for matrices of few features, the
// CTAs of a cluster; their sums meet in (distributed) shared memory and are added in a fixed order. Weights are requested
// before the kernel waits for its predecessor on the stream.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "xpool/gemm_stream.cuh"
#include "xpool/gemm_ws.cuh"
#include "xpool/mma_sync.cuh"
#include "xpool/pdl.cuh"

namespace xpool {
namespace gemm {

constexpr int kSWarps = 8, kSThreads = kSWarps * 32;
constexpr int kSFeat = 16;     // features per warp (the dual form: of the gate and as many of the up matrix)
constexpr int kSMaxCluster = 4;
constexpr int kSStep = 32;     // elements of K per step: 16 bytes a lane

struct StreamArgs {
  const __nv_bfloat16* w;
  const __nv_bfloat16* x;
  int ldw, ldx;
  int parts;             // warps of a CTA that share features: 1, 2, 4 or 8
  int cluster;           // CTAs that share features
  int w_static;          // weights may be read before the predecessor has ended
  Problem p;
};

// (a coherent load: where w_static is 0 the previous kernel may still write w after this one has begun)
__device__ __forceinline__ uint4 ldg_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// One output element (row r of its group, feature f), the arithmetic of the tiled kernel's epilogue.
__device__ __forceinline__ void finish_element(const Problem& p, int group, int r, int f, float g, float u) {
  const float bias = p.bias != nullptr ? p.bias[f] : 0.f;
  const int64_t base = static_cast<int64_t>(group) * p.out_group_stride;
  float v;
  if (p.epilogue == kEpiSwiglu) {
    const float lim = p.gate_limit > 0.f ? p.gate_limit : 3.0e38f;
    const float a = p.act_alpha == 0.f ? 1.f : p.act_alpha;
    const float gg = fminf(round_bf16(g + bias), lim);
    const float uu = fminf(fmaxf(round_bf16(u + (p.bias != nullptr ? p.bias[p.up_offset + f] : 0.f)), -lim), lim);
    const float c = p.act_cubic != 0.f ? fmaf(p.act_cubic * gg, gg, 1.f) : 1.f;
    v = __fdividef(gg, 1.f + __expf(-a * gg * c)) * (uu + p.up_add);
  } else if (p.epilogue == kEpiResidual || p.epilogue == kEpiGateMul || p.epilogue == kEpiSigmoid) {
    const float rr = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.resid)[base + static_cast<int64_t>(r) * p.ld_resid + f]);
    if (p.epilogue == kEpiSigmoid) {
      v = __fdividef(g + bias, 1.f + __expf(-rr));
    } else {
      v = round_bf16(g + bias);
      v = p.epilogue == kEpiResidual ? v + rr : __fdividef(v, 1.f + __expf(-p.act_alpha * v * fmaf(p.act_cubic * v, v, 1.f))) * rr;
    }
  } else {
    v = fmaf(g, p.out_scale == 0.f ? 1.f : p.out_scale, bias);
    if (f < p.silu_cols) v = __fdividef(v, 1.f + __expf(-v));
    if (p.relu2) v = fmaxf(v, 0.f) * fmaxf(v, 0.f);
  }
  const int64_t at = base + static_cast<int64_t>(r) * p.ld_out + f;
  if (p.epilogue == kEpiStoreF32) reinterpret_cast<float*>(p.out)[at] = v;
  else if (p.tail != nullptr && f >= p.tail_from) p.tail[static_cast<int64_t>(r) * p.ld_tail + (f - p.tail_from)] = v;
  else reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(v);
}

// NT: eights of activation rows. MT: 16-feature blocks per warp (dual: a gate and an up block). Two CTAs per SM (128 registers).
template <int NT, int MT, bool kDual>
__global__ void __launch_bounds__(kSThreads, 2)
gemm_stream_kernel(const __grid_constant__ StreamArgs a) {
  constexpr int U = 4 / MT;                                 // steps per batch of loads
  constexpr int FW = kDual ? kSFeat : MT * kSFeat;          // output features per warp
  constexpr int kRows = NT * 8, kPitch = kRows + 1;         // odd pitch: neighbouring features in different banks
  __shared__ float red[kSWarps * MT * kSFeat * kPitch];
  const Problem& p = a.p;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int wide = kSWarps / a.parts;                       // warps side by side over features
  const int wk = warp % a.parts, wm = warp / a.parts;
  const int rank = a.cluster > 1 ? static_cast<int>(blockIdx.x) % a.cluster : 0;
  const int f_cta = static_cast<int>(blockIdx.x) / a.cluster * wide * FW;
  const int group = blockIdx.y;
  const int steps = (p.k + kSStep - 1) / kSStep;
  const int all = a.parts * a.cluster, part = rank * a.parts + wk;
  const int s0 = steps * part / all, s1 = steps * (part + 1) / all;

  // rows g and g + 8 of each block; features past the end repeat the last one and are not stored
  const __nv_bfloat16* wp[MT * 2];
#pragma unroll
  for (int i = 0; i < MT * 2; ++i) {
    int f = f_cta + wm * FW + g + (i & 1) * 8 + (kDual ? 0 : (i >> 1) * kSFeat);
    f = group * p.w_rows_per_group + (f < p.n_out ? f : p.n_out - 1) + (kDual ? (i >> 1) * p.up_offset : 0);
    wp[i] = p.w_tiled ? a.w + (static_cast<int64_t>(f >> 7) * (p.k >> 6) << 13) + ((f & 127) << 6) : a.w + static_cast<int64_t>(f) * a.ldw;
  }
  const int two = p.w_tiled ? kTileM * kTileK : 2 * kSStep;   // elements from a step to the next but one
  auto load = [&](uint4 (&b)[U][MT * 2], int s) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = s + u < s1 && (s + u) * kSStep + q * 8 < p.k;
      const int64_t off = static_cast<int64_t>((s + u) >> 1) * two + ((s + u) & 1) * kSStep + q * 8;
#pragma unroll
      for (int i = 0; i < MT * 2; ++i) b[u][i] = in ? ldg_stream(wp[i] + off) : make_uint4(0, 0, 0, 0);
    }
  };
  uint4 wa[U][MT * 2], wb[U][MT * 2];
  if (a.w_static) load(wa, s0);
  pdl::wait();
  pdl::release();
  if (!a.w_static) load(wa, s0);

  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[m][n][j] = 0.f;
  const __nv_bfloat16* xp[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int r = n * 8 + g;
    xp[n] = a.x + (static_cast<int64_t>(group) * p.x_group_rows + (r < p.rows ? r : p.rows - 1)) * a.ldx + q * 8;
  }
  auto multiply = [&](const uint4 (&b)[U][MT * 2], int s) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = s + u < s1 && (s + u) * kSStep + q * 8 < p.k;
      uint4 xv[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) xv[n] = in ? *reinterpret_cast<const uint4*>(xp[n] + (s + u) * kSStep) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const uint32_t lo[4] = {b[u][2 * m].x, b[u][2 * m + 1].x, b[u][2 * m].y, b[u][2 * m + 1].y};
        const uint32_t hi[4] = {b[u][2 * m].z, b[u][2 * m + 1].z, b[u][2 * m].w, b[u][2 * m + 1].w};
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          frag::mma(acc[m][n], lo, xv[n].x, xv[n].y);
          frag::mma(acc[m][n], hi, xv[n].z, xv[n].w);
        }
      }
    }
  };
  for (int s = s0; s < s1; s += 2 * U) {
    load(wb, s + U);
    multiply(wa, s);
    load(wa, s + 2 * U);
    multiply(wb, s + U);
  }

  // red[slice of K][matrix][feature of the CTA][row]: a thread adds its elements over the CTA's slices, then over the cluster
  const int feats = wide * FW, per_slice = MT * wide * kSFeat * kPitch;
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    float* d = red + wk * per_slice + ((kDual ? m * feats : m * kSFeat) + wm * FW + g) * kPitch + q * 2;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      d[n * 8] = acc[m][n][0];
      d[n * 8 + 1] = acc[m][n][1];
      d[8 * kPitch + n * 8] = acc[m][n][2];
      d[8 * kPitch + n * 8 + 1] = acc[m][n][3];
    }
  }
  __syncthreads();
  const int total = feats * p.rows;
  const auto fold = [&](const float* at) {
    float v[kSWarps];
#pragma unroll
    for (int i = 0; i < kSWarps; ++i) v[i] = i < a.parts ? at[i * per_slice] : 0.f;
    static_assert(kSWarps == 8, "a tree of eight");
    return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  };
  if (a.cluster == 1) {
    for (int e = threadIdx.x; e < total; e += kSThreads) {
      const int fl = e % feats, r = e / feats;
      const float* at = red + fl * kPitch + r;
      const float sg = fold(at), su = kDual ? fold(at + feats * kPitch) : 0.f;
      if (f_cta + fl < p.n_out) finish_element(p, group, r, f_cta + fl, sg, su);
    }
    return;
  }
  namespace cg = cooperative_groups;
  for (int e = threadIdx.x; e < total; e += kSThreads) {
    float* at = red + (e % feats) * kPitch + e / feats;
    *at = fold(at);
    if (kDual) at[feats * kPitch] = fold(at + feats * kPitch);
  }
  cg::this_cluster().sync();
  for (int e = rank * kSThreads + threadIdx.x; e < total; e += a.cluster * kSThreads) {
    const int fl = e % feats, r = e / feats;
    float sg = 0.f, su = 0.f;
#pragma unroll
    for (int c = 0; c < kSMaxCluster; ++c) {
      if (c < a.cluster) {
        const float* at = cg::this_cluster().map_shared_rank(red, c) + fl * kPitch + r;
        sg += *at;
        if (kDual) su += at[feats * kPitch];
      }
    }
    if (f_cta + fl < p.n_out) finish_element(p, group, r, f_cta + fl, sg, su);
  }
  cg::this_cluster().sync();     // nobody's shared memory goes while another CTA reads it
}

// Rows: the tiled kernel has a fixed cost of 6 us a launch, this one reads the activations once per CTA from L2 and once per warp
// through L1. us a launch, inputs colder than L2, tiled / this kernel:
//                          1 row           8 rows          16 rows
//   4096 x 1024            6.8 / 3.2       6.8 / 3.3       6.8 / 4.2
//   gate/up 6144 x 1024    8.2 / 3.8       8.2 / 3.9       8.2 / 4.8
//   1024 x 3072            8.3 / 4.1       8.3 / 4.4       8.3 / 5.1
//   6144 x 4096            12.6 / 10.7     12.6 / 11.2     12.6 / 11.5
//   gate/up 16384 x 2560   17.5 / 14.4     17.4 / 14.7     17.5 / 15.8
//   4096 x 12288           21.5 / 16.8     21.6 / 17.5     21.7 / 19.6
//   3584 x 18944           27.2 / 23.2     27.3 / 24.3     27.2 / 28.0
//   gate/up 24576 x 4096   36.1 / 36.7     36.2 / 37.3     36.2 / 40.9
//   gate/up 37888 x 3584   41.3 / 47.3     41.5 / 48.1     41.6 / 49.0
//   151936 x 1024          51.9 / 49.3     52.5 / 55.6     53.0 / 66.7    (4 rows: 52.4 / 52.1)
//   151936 x 4096          194 / 189       196 / 199       198 / 206      (4 rows: 194 / 195)
// (a form with four eights a warp lost at 32 rows: 24576 x 4096 73.6 us.) So matrices of more than kStreamManyBytes, whose reading hides
// the tiled kernel's fixed cost, come here with up to four rows, gated ones not at all.
// From two eights on a warp takes 32 features, which halves what it reads of the activations. Calls that name a tile width,
// a split or an SM count mean the tiled kernel; rows of K that are no whole 16-byte units, and features whose weight rows the caller
// says do not exist (w_rows_total), need its zero-filled tiles.
constexpr int64_t kStreamManyBytes = 150 << 20;

bool stream_applies(const XpGemmArgs& a) {
  const int groups = a.batch > 1 ? a.batch - 1 : 0;
  const int64_t w_rows = a.n_out + static_cast<int64_t>(groups) * a.w_rows_per_group + (a.dual ? a.up_offset : 0);
  if (w_rows * a.k * 2 > kStreamManyBytes && (a.dual || a.rows > 4)) return false;
  if (a.w_rows_total > 0 && (a.w_rows_total < w_rows || (a.w_tiled && a.w_rows_total % kTileM != 0))) return false;
  const auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.rows <= kStreamMaxRows && !a.fp8 && a.tile_table == nullptr && a.splits == 0 && a.bn == 0 && a.num_sms == 0 && a.k % 8 == 0 &&
         (a.ldw == 0 || a.ldw % 8 == 0) && (a.ldx == 0 || a.ldx % 8 == 0) && aligned(a.w) && aligned(a.x) &&
         (a.epilogue == kEpiSwiglu) == (a.dual != 0) && (!a.w_tiled || a.up_offset % kTileM == 0);
}

template <int NT, int MT, bool kDual>
static int stream_go(const StreamArgs& s, dim3 grid, cudaStream_t stream) {
  const cudaError_t e = pdl::launch(gemm_stream_kernel<NT, MT, kDual>, grid, dim3(kSThreads), 0, stream, s.cluster, s);
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}

// How K is cut: estimated time (us) of a launch by waves of CTAs (two per SM), each at its share of 6.4 TB/s and at most 40 GB/s,
// plus a fixed microsecond a wave and another for the cluster's two barriers. Only the order of the estimates matters.
static void stream_split(StreamArgs* s, int n_out, int batch, int k, int dual, int feats) {
  const int steps = (k + kSStep - 1) / kSStep;
  double best = 1e30;
  for (int cuts = 1; cuts <= kSWarps * kSMaxCluster; cuts *= 2) {
    const int parts = std::min(cuts, kSWarps), cluster = cuts / parts;
    if (cuts > 1 && steps < 2 * cuts) break;
    const int per_cta = kSWarps / parts * feats;
    const double ctas = static_cast<double>((n_out + per_cta - 1) / per_cta) * cluster * batch;
    const double waves = std::ceil(ctas / 296), active = std::min(ctas, 296.0);
    const double kb = static_cast<double>(per_cta) * (dual ? 2 : 1) * k * 2 / cluster / 1000;
    const double t = waves * (1.0 + kb / std::min(6400 / active, 40.0)) + (cluster > 1 ? 1.0 : 0.0);
    if (t < best) best = t, s->parts = parts, s->cluster = cluster;
  }
}

int stream_launch(const XpGemmArgs& a) {
  StreamArgs s{};
  Problem& p = s.p;
  s.w = reinterpret_cast<const __nv_bfloat16*>(a.w);
  s.x = reinterpret_cast<const __nv_bfloat16*>(a.x);
  s.ldw = a.ldw > 0 ? a.ldw : a.k;
  s.w_static = a.w_static;
  s.ldx = a.ldx > 0 ? a.ldx : a.k;
  const int batch = a.batch > 1 ? a.batch : 1;
  p.out = a.out;
  p.resid = a.resid;
  p.bias = a.bias;
  p.n_out = a.n_out;
  p.k = a.k;
  p.rows = a.rows;
  p.ld_out = a.ld_out > 0 ? a.ld_out : a.n_out;
  p.ld_resid = a.ld_resid > 0 ? a.ld_resid : p.ld_out;
  p.epilogue = a.epilogue;
  p.dual = a.dual;
  p.up_offset = a.dual ? a.up_offset : 0;
  p.w_tiled = a.w_tiled;
  p.gate_limit = a.gate_limit;
  p.up_add = a.up_add;
  p.act_alpha = a.act_alpha;
  p.act_cubic = a.act_cubic;
  p.out_scale = a.out_scale;
  p.silu_cols = a.silu_cols;
  p.relu2 = a.relu2;
  p.tail = a.tail;
  p.tail_from = a.tail_from;
  p.ld_tail = a.ld_tail;
  p.batch = batch;
  if (batch > 1) {
    p.w_rows_per_group = a.w_rows_per_group;
    p.x_group_rows = a.x_group_rows;
    p.out_group_stride = a.out_group_stride;
  }
  const int nt = (a.rows + 7) / 8;
  const int mt = a.dual ? 1 : nt > 1 && a.n_out > kSFeat ? 2 : 1;
  stream_split(&s, a.n_out, batch, a.k, a.dual, mt * kSFeat);
  const int per_cta = kSWarps / s.parts * mt * kSFeat;
  const dim3 grid((a.n_out + per_cta - 1) / per_cta * s.cluster, batch);
  const cudaStream_t stream = reinterpret_cast<cudaStream_t>(a.stream);
  if (a.dual) return nt <= 1 ? stream_go<1, 2, true>(s, grid, stream) : stream_go<2, 2, true>(s, grid, stream);
  if (mt == 2) return stream_go<2, 2, false>(s, grid, stream);
  return nt <= 1 ? stream_go<1, 1, false>(s, grid, stream) : stream_go<2, 1, false>(s, grid, stream);
}

}  // namespace gemm
}  // namespace xpool
