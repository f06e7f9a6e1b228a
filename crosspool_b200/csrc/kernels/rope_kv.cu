// Per-token attention pre-processing in one pass over the fused QKV projection:
// optional per-head RMSNorm of q and k (Qwen3), rotary embedding (rotate-half
// convention, base theta), and the scatter of k and v into the paged KV cache.
// The reference leaves all of this to SGLang (its KV store hook only delegates,
// src/xpool/integrations/sglang/ecs/pool.py:116-121).
//
// KV cache layout per layer: [num_pages, page_size, kv_heads, head_dim] for K and
// for V; `slots[row]` = page * page_size + offset, or -1 for padding rows.
#include "xpool/api.h"
#include "xpool/sm100.cuh"
#include "xpool/pdl.cuh"

namespace xpool {
namespace rope {

// A warp takes every heads_step-th head of a row: the angles are the row's, so their sines are computed once a warp. Lane l rotates
// elements l PER .. + PER - 1 of one half with those of the other. WIDE: pairs of elements are 4-byte aligned. Bound by the latency of a
// head's loads, so what counts is warps in flight: 32 registers a thread keep every SM full of them. (Four heads of a warp in flight
// took 64 registers: 4096 rows of 32 query and 8 key heads 47.1 us, so 34.4; 591 rows with a warp a head 10.1 us, so 7.4.)
template <int D, bool WIDE>
__global__ void __launch_bounds__(256)
rope_kv_kernel(XpRopeArgs a, int heads_step) {
  constexpr int PER = D / 64;  // elements per lane in each half
  const int row = blockIdx.x;
  const int lane = threadIdx.x & 31;
  const int first = blockIdx.y * 8 + (threadIdx.x >> 5);
  const int heads_total = a.q_heads + 2 * a.kv_heads, rotated = a.q_heads + a.kv_heads;
  auto load = [&](const __nv_bfloat16* p, float (&v)[PER]) {
    if constexpr (WIDE && PER == 2) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + lane * PER));
      v[0] = f.x, v[1] = f.y;
    } else {
#pragma unroll
      for (int i = 0; i < PER; ++i) v[i] = __bfloat162float(p[lane * PER + i]);
    }
  };
  auto store = [&](__nv_bfloat16* p, const float (&v)[PER]) {
    if constexpr (WIDE && PER == 2) {
      *reinterpret_cast<__nv_bfloat162*>(p + lane * PER) = __floats2bfloat162_rn(v[0], v[1]);
    } else {
#pragma unroll
      for (int i = 0; i < PER; ++i) p[lane * PER + i] = __float2bfloat16_rn(v[i]);
    }
  };
  pdl::wait();
  pdl::release_short();
  if (first >= heads_total) return;
  const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(a.qkv) + static_cast<size_t>(row) * a.ld_qkv;
  const __nv_bfloat16* qn = reinterpret_cast<const __nv_bfloat16*>(a.q_norm_weight);
  const __nv_bfloat16* kn = reinterpret_cast<const __nv_bfloat16*>(a.k_norm_weight);
  const int slot = a.slots[row];
  const float pos = static_cast<float>(a.positions[row]);
  float c[PER], s[PER];
  bool have = false;
  for (int head = first; head < heads_total; head += heads_step) {
    const bool is_q = head < a.q_heads;
    float x1[PER], x2[PER];
    load(src + static_cast<size_t>(head) * D, x1);
    load(src + static_cast<size_t>(head) * D + D / 2, x2);
    if (head < rotated) {
      const __nv_bfloat16* nw = is_q ? qn : kn;
      float n1[PER], n2[PER];
      if (nw != nullptr) {
        load(nw, n1);
        load(nw + D / 2, n2);
      }
      if (!have) {                      // beside the loads
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int idx = lane * PER + i;
          const float inv_freq = exp2f(-(2.f * idx / D) * a.log2_theta);
          sincosf(pos * inv_freq, &s[i], &c[i]);
        }
        have = true;
      }
      if (nw != nullptr) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) ss += x1[i] * x1[i] + x2[i] * x2[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = rsqrtf(ss / D + a.eps);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const float v1 = __bfloat162float(__float2bfloat16_rn(x1[i] * inv));
          const float v2 = __bfloat162float(__float2bfloat16_rn(x2[i] * inv));
          x1[i] = __bfloat162float(__float2bfloat16_rn(v1 * n1[i]));
          x2[i] = __bfloat162float(__float2bfloat16_rn(v2 * n2[i]));
        }
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const float r1 = x1[i] * c[i] - x2[i] * s[i];
        const float r2 = x2[i] * c[i] + x1[i] * s[i];
        x1[i] = r1;
        x2[i] = r2;
      }
    }
    __nv_bfloat16* dst;
    if (is_q) {
      dst = reinterpret_cast<__nv_bfloat16*>(a.q_out) + (static_cast<size_t>(row) * a.q_heads + head) * D;
    } else {
      if (slot < 0) continue;
      const int hk = head < rotated ? head - a.q_heads : head - rotated;
      dst = reinterpret_cast<__nv_bfloat16*>(head < rotated ? a.k_cache : a.v_cache) + (static_cast<size_t>(slot) * a.kv_heads + hk) * D;
    }
    store(dst, x1);
    store(dst + D / 2, x2);
  }
}

}  // namespace rope
}  // namespace xpool

extern "C" int xp_rope_kv(const XpRopeArgs* a, void* stream) {
  if (a->rows <= 0) return 0;
  const int heads_total = a->q_heads + 2 * a->kv_heads;
  // A CTA per row where the rows alone fill the SMs several times over; in a decode step every head has a warp. us, warp a head / CTA a
  // row, 16 + 8 + 8 heads of 128: 256 rows 3.0 / 3.4, 591 rows 5.2 / 5.6, 1000 rows 8.0 / 6.7; 32 + 8 + 8: 3.9 / 4.5, 7.4 / 7.7,
  // 11.8 / 9.0.
  const bool many = a->rows >= 148 * 4;
  const dim3 grid(a->rows, many ? 1 : (heads_total + 7) / 8);
  const int step = static_cast<int>(grid.y) * 8;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  auto pair = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3) == 0; };
  const bool wide = a->ld_qkv % 2 == 0 && pair(a->qkv) && pair(a->q_out) && pair(a->k_cache) && pair(a->v_cache) && pair(a->q_norm_weight) && pair(a->k_norm_weight);
  using namespace xpool::rope;
  if (a->head_dim == 128 && wide)
    xpool::pdl::launch(rope_kv_kernel<128, true>, grid, 256, 0, s, 1, *a, step);
  else if (a->head_dim == 128)
    xpool::pdl::launch(rope_kv_kernel<128, false>, grid, 256, 0, s, 1, *a, step);
  else if (a->head_dim == 64)
    xpool::pdl::launch(rope_kv_kernel<64, true>, grid, 256, 0, s, 1, *a, step);
  else
    return -10;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}
