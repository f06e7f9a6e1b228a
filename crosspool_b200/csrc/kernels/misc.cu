// Embedding gather and greedy sampling (row-wise argmax; ties go to the lower id,
// which is what torch.argmax returns for the first maximal element).
#include <cooperative_groups.h>
#include <math_constants.h>

#include <utility>

#include "xpool/api.h"
#include "xpool/pdl.cuh"
#include "xpool/sm100.cuh"

namespace {

__global__ void __launch_bounds__(128)
embedding_kernel(const int* ids, const uint4* table, uint4* out, int hidden8, int vocab) {
  xpool::pdl::wait();
  xpool::pdl::release_short();
  const int row = blockIdx.x;
  int id = ids[row];
  if (id < 0 || id >= vocab) id = 0;
  const uint4* src = table + static_cast<size_t>(id) * hidden8;
  uint4* dst = out + static_cast<size_t>(row) * hidden8;
  for (int i = threadIdx.x; i < hidden8; i += 128) dst[i] = src[i];
}

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Greedy sampling. A cluster of up to eight CTAs takes a row, 16 bytes a load (one 1024-thread CTA with 2-byte loads took 13.5 us for 152k
// bf16 logits, bound by the latency of a thread's 150 loads in a row); the winners meet in the first CTA's shared memory.
constexpr int kArgCluster = 8;

__device__ __forceinline__ void better(float& best, int& bi, float v, int i) {
  if (v > best || (v == best && i < bi)) best = v, bi = i;
}
__device__ __forceinline__ void warp_best(float& best, int& bi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    better(best, bi, ov, oi);
  }
}

template <typename T, int kThreads>
__global__ void __launch_bounds__(kThreads)
argmax_kernel(const T* logits, int* out, int vocab, int ld, int wide, int ranks) {
  namespace cg = cooperative_groups;
  // The first CTA's shared memory may be written once that CTA is known to have started: all arrive here and wait before the
  // stores, a row's scan later.
  auto started = cg::this_cluster().barrier_arrive();
  xpool::pdl::wait();
  xpool::pdl::release();
  constexpr int N = 16 / sizeof(T), kWarps = kThreads / 32, kSlots = kThreads == 256 ? kArgCluster * kWarps : kWarps;
  __shared__ float sv[kSlots];
  __shared__ int si[kSlots];
  const int rank = blockIdx.x % ranks, at = blockIdx.x / ranks, first = rank * kThreads + threadIdx.x, stride = ranks * kThreads;
  const T* row = logits + static_cast<size_t>(at) * ld;
  float best = -CUDART_INF_F;
  int bi = 0x7fffffff;
  const int whole = wide ? vocab / N : 0;
#pragma unroll 4
  for (int c = first; c < whole; c += stride) {
    const uint4 raw = reinterpret_cast<const uint4*>(row)[c];
    const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < N; ++j) better(best, bi, to_f<T>(v[j]), c * N + j);
  }
  for (int i = whole * N + first; i < vocab; i += stride) better(best, bi, to_f<T>(row[i]), i);
  warp_best(best, bi);
  cg::this_cluster().barrier_wait(std::move(started));
  if ((threadIdx.x & 31) == 0) {
    const int slot = rank * kWarps + (threadIdx.x >> 5);
    cg::this_cluster().map_shared_rank(sv, 0)[slot] = best;
    cg::this_cluster().map_shared_rank(si, 0)[slot] = bi;
  }
  cg::this_cluster().sync();
  if (rank != 0 || threadIdx.x >= 32) return;
  best = -CUDART_INF_F, bi = 0x7fffffff;
  for (int i = threadIdx.x; i < ranks * kWarps; i += 32) better(best, bi, sv[i], si[i]);
  warp_best(best, bi);
  if (threadIdx.x == 0) out[at] = bi;
}

// Temperature sampling by the Gumbel-max trick: argmax_i (logit_i / T + g_i) with g_i = -log(-log u_i) draws
// from softmax(logits / T) exactly, in one pass and without normalising. u_i comes from a counter-based hash
// of (row seed, token index), so a (seed, step) pair always yields the same token. T <= 0 is greedy.
__device__ __forceinline__ uint32_t hash3(uint32_t a, uint32_t b, uint32_t c) {
  uint64_t x = (static_cast<uint64_t>(a) << 32) ^ (static_cast<uint64_t>(b) * 0x9E3779B97F4A7C15ull) ^ c;
  x ^= x >> 30;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return static_cast<uint32_t>(x >> 16);
}

template <typename T>
__global__ void __launch_bounds__(1024)
sample_kernel(const T* __restrict__ logits, const float* __restrict__ temps, const uint32_t* __restrict__ seeds,
              int* __restrict__ out, int vocab, int ld) {
  __shared__ float sv[32];
  __shared__ int si[32];
  const T* row = logits + static_cast<size_t>(blockIdx.x) * ld;
  const float temp = temps[blockIdx.x];
  const float inv_t = temp > 0.f ? 1.f / temp : 1.f;
  const uint32_t seed = seeds[2 * blockIdx.x], step = seeds[2 * blockIdx.x + 1];
  float best = -CUDART_INF_F;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < vocab; i += 1024) {
    float v = to_f<T>(row[i]) * inv_t;
    if (temp > 0.f) {
      const float u = (static_cast<float>(hash3(seed, step, static_cast<uint32_t>(i)) >> 8) + 0.5f) * (1.f / 16777216.f);
      v -= __logf(-__logf(u));
    }
    if (v > best || (v == best && i < bi)) {
      best = v;
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) {
      best = ov;
      bi = oi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = best;
    si[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    best = sv[threadIdx.x];
    bi = si[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if (threadIdx.x == 0) out[blockIdx.x] = bi;
  }
}

}  // namespace

// temps [rows] fp32, seeds [rows, 2] u32 (request seed, step counter), all device memory.
extern "C" int xp_sample(const void* logits, int is_fp32, const float* temps, const uint32_t* seeds, int* out, int rows,
                         int vocab, int ld, void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (is_fp32)
    sample_kernel<float><<<rows, 1024, 0, s>>>(reinterpret_cast<const float*>(logits), temps, seeds, out, vocab, ld);
  else
    sample_kernel<__nv_bfloat16><<<rows, 1024, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(logits), temps, seeds, out, vocab, ld);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}

extern "C" int xp_embedding(const int* ids, const void* table, void* out, int rows, int hidden,
                            int vocab, void* stream) {
  if (rows <= 0) return 0;
  if (hidden % 8 != 0) return -10;
  xpool::pdl::launch(embedding_kernel, rows, 128, 0, reinterpret_cast<cudaStream_t>(stream), 1,
      ids, reinterpret_cast<const uint4*>(table), reinterpret_cast<uint4*>(out), hidden / 8, vocab);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}

extern "C" int xp_argmax(const void* logits, int is_fp32, int* out, int rows, int vocab, int ld,
                         void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int wide = (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && static_cast<size_t>(ld) * (is_fp32 ? 4 : 2) % 16 == 0;
  // Clusters while the rows leave SMs idle and every CTA has 4 KB of its row; otherwise a CTA a row, of more threads the longer it is. us,
  // clusters of eight / so: 8 rows of 151936 bf16 3.7 both; 64 rows 6.5 / 6.1; 256 rows 16.9 / 15.4; 256 rows of 32000 8.8 / 4.9, of 1000
  // 6.0 / 2.1 (one scalar 1024-thread CTA a row: 11.7, 12.0, 20.9, 6.8, 2.6).
  const size_t bytes = static_cast<size_t>(vocab) * (is_fp32 ? 4 : 2);
  int ranks = rows <= 32 ? 8 : rows <= 64 ? 4 : 1;
  while (ranks > 1 && bytes / ranks < 4096) ranks >>= 1;
  const int threads = ranks > 1 || bytes <= 8192 ? 256 : bytes <= 65536 ? 512 : 1024;
  auto go = [&](auto kernel, auto* p) { xpool::pdl::launch(kernel, static_cast<unsigned>(rows) * ranks, threads, 0, s, ranks, p, out, vocab, ld, wide, ranks); };
  if (is_fp32) {
    const float* p = reinterpret_cast<const float*>(logits);
    go(threads == 256 ? argmax_kernel<float, 256> : threads == 512 ? argmax_kernel<float, 512> : argmax_kernel<float, 1024>, p);
  } else {
    const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(logits);
    go(threads == 256 ? argmax_kernel<__nv_bfloat16, 256> : threads == 512 ? argmax_kernel<__nv_bfloat16, 512> : argmax_kernel<__nv_bfloat16, 1024>, p);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - static_cast<int>(e);
}
