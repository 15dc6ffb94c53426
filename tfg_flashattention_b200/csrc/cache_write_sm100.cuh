// New keys and values of a prompt into the K/V caches: two strided copies as one launch (the reference
// keeps no cache, src/py/model_inference.py:199-228; torch needs a copy kernel and its views for each).
//
// Bound by memory: 4 * 128 bytes move per row and head.  A thread carries 16 bytes of K and of V; eight
// threads a row, consecutive threads consecutive heads, so that reads (a fused QKV projection) and
// writes (the cache's [B, N, H, 64] rows) run along memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx_sm100.cuh"

namespace fa {

struct CacheWriteParams {
  const __nv_bfloat16 *k, *v;            // [B, N, H, 64]: strides in elements, the innermost 1
  __nv_bfloat16 *k_cache, *v_cache;      // row 0 of the new rows
  long long s_b, s_n, s_h;               // of k and v: sequence, row, head
  long long c_b, c_n, c_h;               // of the caches
  int N, H;
  long long total;                       // B * N * H * 8 vectors
};

constexpr int kCacheWriteThreads = 256;

__global__ void __launch_bounds__(kCacheWriteThreads) fa_cache_write_kernel(const CacheWriteParams p) {
  pdl_trigger();
  pdl_wait();
  const long long i = static_cast<long long>(blockIdx.x) * kCacheWriteThreads + threadIdx.x;
  if (i >= p.total) return;
  const int c = static_cast<int>(i & 7) * 8;
  const long long row = i >> 3;
  const int h = static_cast<int>(row % p.H);
  const long long bn = row / p.H;
  const int n = static_cast<int>(bn % p.N);
  const long long b = bn / p.N;
  const long long src = b * p.s_b + n * p.s_n + h * p.s_h + c, dst = b * p.c_b + n * p.c_n + h * p.c_h + c;
  const uint4 k = *reinterpret_cast<const uint4*>(p.k + src), v = *reinterpret_cast<const uint4*>(p.v + src);
  *reinterpret_cast<uint4*>(p.k_cache + dst) = k;
  *reinterpret_cast<uint4*>(p.v_cache + dst) = v;
}

}  // namespace fa
