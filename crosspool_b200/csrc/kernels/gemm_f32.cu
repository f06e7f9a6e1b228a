// Plain fp32 matrix product y = x w^T (+ bias) for models served in 32-bit: FFMA only, no reduced-precision tensor mode.
//
// Two forms, both with K cut between the warps of a CTA and folded in a fixed order:
//   gemv_f32  up to 8 rows whose operands start on 16-byte boundaries. Bound by reading w once: a warp streams 16 bytes a lane of
//             four weight rows, two steps at a time, and multiplies them with every row of x from registers; nothing is staged.
//             The products of a decode step of 8 layers of width 1024 (3 rows, LM head of 152k features among them) went from
//             263 us a launch (one 64 x 64 tile a CTA, 4-byte loads, nothing in flight while it computes) to 7.9 us.
//   tile_f32  a tile of 8 TM rows x 64 features per 128 threads, 32-deep slices copied by cp.async one slice ahead; up to
//             four such groups of a CTA share a tile and take every fourth slice, because a few hundred rows give fewer tiles
//             than the SMs have schedulers. A thread owns TM x 4 outputs and reads both operands as 16-byte runs along K
//             (12 wide shared loads per 128 FMAs at TM = 8; pitch 36 floats: eight neighbouring rows fall into different banks).
//             106 us a launch at 317 rows, bound by FFMA issue and the partial last wave.
#include <cuda_runtime.h>
#include <stdint.h>

#include "xpool/mixer_api.h"

namespace {

constexpr int kBN = 64, kBK = 32, kPitch = kBK + 4;
constexpr int kGroupedRows = 64;       // rows of a tile of the grouped form's table
constexpr int kGroup = 128;            // threads that share a slice

__device__ __forceinline__ float finish(float acc, float scale, const float* bias, int c, int silu_cols) {
  const float v = fmaf(acc, scale, bias != nullptr ? bias[c] : 0.f);
  return c < silu_cols ? v / (1.f + expf(-v)) : v;
}

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {   // the rest of the 16 bytes becomes zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int TM>
constexpr int tile_smem(int groups) {
  return groups * 2 * (8 * TM + kBN) * kPitch * 4;
}

// Rows r0 .. and features n0 .. of one product; rows and n bound both. VEC: rows of both operands start on 16-byte boundaries.
template <int TM, bool VEC>
__device__ __forceinline__ void tile_f32(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                                         float* __restrict__ out, int r0, int n0, int rows, int n, int k, int ldx, int ldw, int ldo, float scale,
                                         int silu_cols) {
  extern __shared__ __align__(16) float smem_f32[];
  constexpr int kBM = 8 * TM, kStage = (kBM + kBN) * kPitch;
  const int groups = blockDim.x / kGroup, group = threadIdx.x / kGroup, t = threadIdx.x % kGroup;
  const int tr = t & 7, tc = t >> 3;
  float* mine = smem_f32 + group * 2 * kStage;
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
  const int slices = (k + kBK - 1) / kBK;
  auto load = [&](int slice, int stage) {
    const int k0 = slice * kBK;
    if constexpr (VEC) {
      constexpr int kUnits = kBK / 4;
#pragma unroll 8
      for (int i = t; i < (kBM + kBN) * kUnits; i += kGroup) {
        const int m = i / kUnits, c = k0 + i % kUnits * 4;
        const bool of_x = m < kBM;
        const int row = of_x ? r0 + m : n0 + m - kBM;
        const bool in = row < (of_x ? rows : n) && c < k;
        const float* src = of_x ? x : w;
        if (in) src += static_cast<int64_t>(row) * (of_x ? ldx : ldw) + c;
        copy16(base + (stage * kStage + m * kPitch + i % kUnits * 4) * 4, src, in ? min(4, k - c) * 4 : 0);
      }
    } else {
      // an element a copy, so the instructions around it count: a thread keeps its column and steps from row to row of one operand
      // (2048 rows x 1001 features x 999: 209 us with both operands' rows worked out for every copy)
      static_assert(kBK == 32 && kGroup % 32 == 0, "a warp copies a row's slice");
      constexpr int kStep = kGroup / 32;
      const int c = k0 + (t & 31), m0 = t >> 5;
      auto rows_of = [&](const float* src, int ld, int first, int end, int count, int at) {
        const float* p = src + static_cast<int64_t>(first + m0) * ld + c;
        uint32_t dst = base + (stage * kStage + (at + m0) * kPitch + (t & 31)) * 4;
        int left = c < k ? end - first - m0 : 0;
#pragma unroll 8
        for (int j = 0; j < count / kStep; ++j, left -= kStep, p += static_cast<int64_t>(kStep) * ld, dst += kStep * kPitch * 4)
          copy4(dst, left > 0 ? p : src, left > 0 ? 4 : 0);
      };
      rows_of(x, ldx, r0, rows, kBM, 0);
      rows_of(w, ldw, n0, n, kBN, kBM);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][4] = {};
  if (group < slices) load(group, 0);
  int stage = 0;
  for (int s = group; s < slices; s += groups, stage ^= 1) {
    if (s + groups < slices) {
      load(s + groups, stage ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kGroup) : "memory");
    const float* xs = mine + stage * kStage + tr * kPitch;
    const float* ws = mine + stage * kStage + (kBM + tc) * kPitch;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * 16 * kPitch + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(xs + i * 8 * kPitch + kk);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, acc[i][j]))));
      }
    }
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kGroup) : "memory");
  }
  if (groups > 1) {
    __syncthreads();                    // slices are consumed: their space holds the partial sums
    if (group > 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) smem_f32[((group - 1) * TM * 4 + i * 4 + j) * kGroup + t] = acc[i][j];
    }
    __syncthreads();
    if (group > 0) return;
    for (int g = 1; g < groups; ++g)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += smem_f32[((g - 1) * TM * 4 + i * 4 + j) * kGroup + t];
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = r0 + tr + 8 * i;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tc + 16 * j;
      if (c < n) out[static_cast<int64_t>(r) * ldo + c] = finish(acc[i][j], scale, bias, c, silu_cols);
    }
  }
}

template <int TM, bool VEC>
__global__ void __launch_bounds__(4 * kGroup)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ out,
                int rows, int n, int k, int ldx, int ldw, int ldo, int64_t sx, int64_t sw, int64_t so, float scale, int silu_cols) {
  tile_f32<TM, VEC>(x + blockIdx.z * sx, w + blockIdx.z * sw, bias, out + blockIdx.z * so, blockIdx.y * 8 * TM, blockIdx.x * kBN, rows, n, k, ldx,
                    ldw, ldo, scale, silu_cols);
}

// Grouped form: tiles {group, first feature of 128, first row, row end} of at most 64 rows from a device table; a CTA takes
// one half of a tile's features, with the row tile that its rows fill.
template <bool VEC>
__global__ void __launch_bounds__(4 * kGroup)
gemm_f32_grouped_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, const int4* __restrict__ tiles,
                        const int* __restrict__ n_tiles, int n, int k, int ldx, int ldw, int ldo, int w_rows_per_group) {
  if (static_cast<int>(blockIdx.x) >= *n_tiles) return;
  const int4 t = tiles[blockIdx.x];
  const int n0 = t.y + blockIdx.y * kBN;
  if (n0 >= n) return;
  const float* wg = w + static_cast<int64_t>(t.x) * w_rows_per_group * ldw;
  const int end = min(t.w, t.z + kGroupedRows);
  if (end - t.z <= 16) tile_f32<2, VEC>(x, wg, nullptr, out, t.z, n0, end, n, k, ldx, ldw, ldo, 1.f, 0);
  else tile_f32<8, VEC>(x, wg, nullptr, out, t.z, n0, end, n, k, ldx, ldw, ldo, 1.f, 0);
}

// ------------------------------------------------------------------------------------------ few rows
constexpr int kGemvWarps = 8, kGemvFeatures = 4;       // features per warp

// R: rows of x held per pass (rows <= R; those beyond repeat the first and are not stored). k_parts warps share four features.
template <int R>
__global__ void __launch_bounds__(kGemvWarps * 32)
gemv_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ out,
                int rows, int n, int k, int ldx, int ldw, int ldo, int64_t sx, int64_t sw, int64_t so, float scale, int silu_cols, int k_parts) {
  constexpr int F = kGemvFeatures, V = F * R;
  __shared__ float red[kGemvWarps][V];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_cta = kGemvWarps / k_parts * F;
  const int f0 = blockIdx.x * per_cta + warp / k_parts * F, part = warp % k_parts;
  const float* wp[F];
  const float* xp[R];
#pragma unroll
  for (int f = 0; f < F; ++f) wp[f] = w + blockIdx.z * sw + static_cast<int64_t>(f0 + f < n ? f0 + f : n - 1) * ldw;
#pragma unroll
  for (int r = 0; r < R; ++r) xp[r] = x + blockIdx.z * sx + static_cast<int64_t>(r < rows ? r : 0) * ldx;
  float acc[V] = {};
  const int step = 128 * k_parts;
  int c = part * 128 + lane * 4;
  auto add = [&](const float4 (&a)[F], int at) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 b = *reinterpret_cast<const float4*>(xp[r] + at);
#pragma unroll
      for (int f = 0; f < F; ++f)
        acc[f * R + r] = fmaf(a[f].w, b.w, fmaf(a[f].z, b.z, fmaf(a[f].y, b.y, fmaf(a[f].x, b.x, acc[f * R + r]))));
    }
  };
  for (; c + step < k; c += 2 * step) {            // k is a multiple of 4: a lane's four elements are inside or outside together
    float4 a0[F], a1[F];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      a0[f] = __ldcs(reinterpret_cast<const float4*>(wp[f] + c));
      a1[f] = __ldcs(reinterpret_cast<const float4*>(wp[f] + c + step));
    }
    add(a0, c);
    add(a1, c + step);
  }
  if (c < k) {
    float4 a0[F];
#pragma unroll
    for (int f = 0; f < F; ++f) a0[f] = __ldcs(reinterpret_cast<const float4*>(wp[f] + c));
    add(a0, c);
  }
  // sums over the lanes: each exchange halves the values a lane is responsible for, then plain butterflies
  int mine = 0;
#pragma unroll
  for (int off = 16, m = V / 2; off > 0; off >>= 1, m >>= 1) {
    if (m >= 1) {
      const bool upper = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < (m > 0 ? m : 1); ++i) {
        const float send = upper ? acc[i] : acc[i + m], keep = upper ? acc[i + m] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
      mine += upper ? m : 0;
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    }
  }
  red[warp][mine] = acc[0];                       // lanes with the same value hold the same sum
  __syncthreads();
  for (int i = threadIdx.x; i < kGemvWarps / k_parts * V; i += kGemvWarps * 32) {
    const int set = i / V, v = i % V, r = v % R, col = blockIdx.x * per_cta + set * F + v / R;
    float s = red[set * k_parts][v];
    for (int q = 1; q < k_parts; ++q) s += red[set * k_parts + q][v];
    if (r < rows && col < n) out[blockIdx.z * so + static_cast<int64_t>(r) * ldo + col] = finish(s, scale, bias, col, silu_cols);
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Groups of threads that share a tile: 16 warps per SM want work, and every group needs slices of its own.
int groups_for(int64_t ctas, int k) {
  int g = ctas >= 148 * 4 ? 1 : ctas >= 148 * 2 ? 2 : 4;
  while (g > 1 && (k + kBK - 1) / kBK < 2 * g) g >>= 1;
  return g;
}

struct Product {
  const float *x, *w, *bias;
  float* out;
  int rows, n, k, ldx, ldw, ldo, batch;
  int64_t sx, sw, so;
  float scale;
  int silu_cols;
};

template <int TM, bool VEC>
int launch_tiles(const Product& p, cudaStream_t s) {
  const dim3 grid((p.n + kBN - 1) / kBN, (p.rows + 8 * TM - 1) / (8 * TM), p.batch);
  const int groups = groups_for(static_cast<int64_t>(grid.x) * grid.y * grid.z, p.k);
  if (tile_smem<TM>(groups) > 48 * 1024 &&
      cudaFuncSetAttribute(gemm_f32_kernel<TM, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem<TM>(4)) != cudaSuccess)
    return -30;
  gemm_f32_kernel<TM, VEC><<<grid, groups * kGroup, tile_smem<TM>(groups), s>>>(p.x, p.w, p.bias, p.out, p.rows, p.n, p.k, p.ldx, p.ldw, p.ldo, p.sx,
                                                                               p.sw, p.so, p.scale, p.silu_cols);
  return 0;
}

template <int R>
void launch_gemv(const Product& p, cudaStream_t s) {
  int parts = 1;                        // enough CTAs for every SM to hold four, while a warp keeps a step of its own
  while (parts < kGemvWarps && p.k > 128 * parts && static_cast<int64_t>(p.n) * p.batch * parts < 148LL * 4 * kGemvWarps * kGemvFeatures) parts <<= 1;
  const int per_cta = kGemvWarps / parts * kGemvFeatures;
  gemv_f32_kernel<R><<<dim3((p.n + per_cta - 1) / per_cta, 1, p.batch), kGemvWarps * 32, 0, s>>>(
      p.x, p.w, p.bias, p.out, p.rows, p.n, p.k, p.ldx, p.ldw, p.ldo, p.sx, p.sw, p.so, p.scale, p.silu_cols, parts);
}

template <bool VEC>
int launch_by_rows(const Product& p, cudaStream_t s) {
  if (p.rows <= 16) return launch_tiles<2, VEC>(p, s);
  // 64-row tiles once they give every SM one; below that 32-row tiles spread the work further
  const int64_t big = static_cast<int64_t>((p.n + kBN - 1) / kBN) * ((p.rows + 63) / 64) * p.batch;
  return p.rows <= 32 || big < 148 ? launch_tiles<4, VEC>(p, s) : launch_tiles<8, VEC>(p, s);
}

}  // namespace

extern "C" int xp_gemm_f32_grouped(const float* x, const float* w, float* out, const void* tiles, const int* n_tiles, int max_tiles, int n, int k,
                                   int ldx, int ldw, int ldo, int w_rows_per_group, void* stream) {
  if (max_tiles <= 0 || n <= 0) return 0;
  if (k <= 0) return -10;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const bool vec = aligned16(x) && aligned16(w) && ldx % 4 == 0 && ldw % 4 == 0;
  auto kernel = vec ? gemm_f32_grouped_kernel<true> : gemm_f32_grouped_kernel<false>;
  const int groups = (k + kBK - 1) / kBK >= 4 ? 2 : 1;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem<8>(2)) != cudaSuccess) return -30;
  kernel<<<dim3(max_tiles, 128 / kBN), groups * kGroup, tile_smem<8>(groups), s>>>(x, w, out, static_cast<const int4*>(tiles), n_tiles, n, k, ldx, ldw,
                                                                                    ldo, w_rows_per_group);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}

extern "C" int xp_gemm_f32(const float* x, const float* w, const float* bias, float* out, int rows, int n, int k, int ldx, int ldw,
                           int ldo, int batch, int64_t sx, int64_t sw, int64_t so, float out_scale, int silu_cols, void* stream) {
  if (rows <= 0 || n <= 0 || batch <= 0) return 0;
  if (k <= 0) return -10;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const Product p{x, w, bias, out, rows, n, k, ldx, ldw, ldo, batch, sx, sw, so, out_scale == 0.f ? 1.f : out_scale, silu_cols};
  const bool vec = aligned16(x) && aligned16(w) && ldx % 4 == 0 && ldw % 4 == 0 && sx % 4 == 0 && sw % 4 == 0;
  int rc = 0;
  if (vec && rows <= 8 && k % 4 == 0) {
    if (rows == 1) launch_gemv<1>(p, s);
    else if (rows == 2) launch_gemv<2>(p, s);
    else if (rows <= 4) launch_gemv<4>(p, s);
    else launch_gemv<8>(p, s);
  } else {
    rc = vec ? launch_by_rows<true>(p, s) : launch_by_rows<false>(p, s);
  }
  if (rc != 0) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}
