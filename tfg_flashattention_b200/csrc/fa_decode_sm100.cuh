// Single-query ("decode") attention for sm_100a: one new token per sequence attends a K/V cache.
//
//   o[b,h,:] = softmax_j(scale * q[b,h,:] . k[b,h,j,:]) v[b,h,j,:],   j < kv_len
//
// This is the attention of autoregressive generation with a KV cache (the reference generates by
// re-running the whole prefix for every token, src/py/model_inference.py:199-228).  One query row
// gives the tensor cores nothing to do; the kernel is bound by reading K and V once from HBM
// (2 * kv_len * 128 bytes per head).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "ptx_sm100.cuh"

namespace fa {

constexpr int kDecodePartial = 66;           // floats per partial: m, l, o[64]
constexpr int kDecodeClusterMax = 16;        // CTAs per cluster (above 8: opt-in)
constexpr int kDecodeMinRows = 48;           // rows of a CTA, at least, where a head has several

struct DecodeParams {
  const __nv_bfloat16* q;      // [B, H, 64]
  const __nv_bfloat16* k;      // [B, H, kv_len.., 64] with strides below
  const __nv_bfloat16* v;
  __nv_bfloat16* o;            // [B, H, 64]
  float* lse;                  // [B, H] or null
  long long q_sb, q_sh;        // element strides of q and o: batch, head
  long long o_sb, o_sh;
  long long k_sb, k_sh, k_sn;  // element strides of the caches: batch, head, row
  long long v_sb, v_sh, v_sn;
  int B, H, kv_len;
  int cluster_log2;            // CTAs per head
  float scale_log2;            // softmax_scale * log2(e)
  // when set: the newest row (index length - 1) is taken from these [B, H, 64] buffers instead of
  // the caches and written into the caches by the CTA that owns it (the cache append of a
  // generation step, folded into the attention kernel)
  const __nv_bfloat16* k_new = nullptr;
  const __nv_bfloat16* v_new = nullptr;
  long long new_sb = 0, new_sh = 0;
  const int* kv_len_ptr = nullptr;   // when set: the current length lives in device memory (read
                                     // at run time, clamped to [1, kv_len]); kv_len is the bound
                                     // the launch was sized for
};

// grid B*H*ctas in clusters of ctas: a head is a cluster of 1, 2, 4, 8 or 16 CTAs, each with
// an equal share of the rows that are there when the kernel runs; the partials meet in the first CTA's
// shared memory (distributed shared memory, one cluster barrier), so there is one launch and no
// scratch buffer.  Lane group g = tid / 8 owns rows g, g + kGroups, ... of the share; lane c = tid % 8
// owns columns 8c .. 8c+7.  Four rows of K and of V per lane group are in flight, their scores and
// maxima are handled together (one rescale per four rows).
//
// What bounds it: HBM, as long as enough loads are open and the SMs keep up with what arrives.  A CTA
// of 128 threads has 16 KB of loads open and nothing to do while they fly; seven per SM fit (72
// registers).  All arithmetic is on packed pairs: in scalar form, a row at a time, the issue slots
// were the limit (B=32 H=25 kv 2000: 77.6 us; 63.7 us now, the floor at the copy rate is 63.5).
// With too few heads for that even as clusters of 16, CTAs have 256 or 512 threads.  The choice is
// decode_shape's (fa_b200_api.cu).  H = 25, us: B=1 kv 1001 7.2 -> 4.0, B=8 kv 1001 20.5 -> 12.0, B=8
// kv 4000 60 -> 36, B=4 kv 16384 83 -> 70 (65); before: one wide CTA per head, or chunks with a
// second launch to merge them.
template <int kThreads, int kCtasPerSm, bool kCluster>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) fa_decode_kernel(const DecodeParams p) {
  constexpr int kWarps = kThreads / 32, kGroups = kThreads / 8, kUnroll = 4;
  __shared__ float sm_w[kWarps][kDecodePartial];                              // this CTA's warps
  __shared__ float sm_c[kCluster ? kDecodeClusterMax : 1][kDecodePartial];    // rank 0: the cluster's CTAs
  const int ctas = kCluster ? 1 << p.cluster_log2 : 1;
  const int rank = kCluster ? blockIdx.x & (ctas - 1) : 0, bh = kCluster ? blockIdx.x >> p.cluster_log2 : blockIdx.x;
  const int b = bh / p.H, h = bh - b * p.H;
  const int tid = threadIdx.x, g = tid >> 3, c = tid & 7;
  // every CTA of the cluster has started before anyone writes to rank 0's shared memory
  if (kCluster) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  pdl_trigger();
  pdl_wait();
  // (an ordinary load: the kernel in front may still be writing it when this one has started)
  const int kv_len = p.kv_len_ptr ? max(1, min(*static_cast<const volatile int*>(p.kv_len_ptr), p.kv_len)) : p.kv_len;
  const int r0 = kCluster ? static_cast<int>(static_cast<long long>(rank) * kv_len / ctas) : 0;
  const int r1 = kCluster ? static_cast<int>(static_cast<long long>(rank + 1) * kv_len / ctas) : kv_len;
  const __nv_bfloat16* kp = p.k + b * p.k_sb + h * p.k_sh + (r0 + g) * p.k_sn + 8 * c;    // row r0 + g
  const __nv_bfloat16* vp = p.v + b * p.v_sb + h * p.v_sh + (r0 + g) * p.v_sn + 8 * c;
  const long long k_step = kGroups * p.k_sn, v_step = kGroups * p.v_sn;
  if (p.k_new != nullptr && r1 == kv_len && (r1 - 1 - r0) % kGroups == g) {
    // the row being appended: into the caches first, the loop then reads it back (same thread)
    const long long at = (r1 - 1 - r0 - g), src = b * p.new_sb + h * p.new_sh + 8 * c;
    const uint4 kn = *reinterpret_cast<const uint4*>(p.k_new + src), vn = *reinterpret_cast<const uint4*>(p.v_new + src);
    *reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(kp) + at * p.k_sn) = kn;
    *reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(vp) + at * p.v_sn) = vn;
  }
  uint64_t q2[4], acc[4] = {0ull, 0ull, 0ull, 0ull};
  {
    const uint4 raw = *reinterpret_cast<const uint4*>(p.q + b * p.q_sb + h * p.q_sh + 8 * c);
    const uint64_t sc = pack_f32x2(p.scale_log2, p.scale_log2);
    q2[0] = mul_f32x2(bf16x2_to_f32x2(raw.x), sc);
    q2[1] = mul_f32x2(bf16x2_to_f32x2(raw.y), sc);
    q2[2] = mul_f32x2(bf16x2_to_f32x2(raw.z), sc);
    q2[3] = mul_f32x2(bf16x2_to_f32x2(raw.w), sc);
  }
  float m = kNoScore, l = 0.f;                       // finite: a group without rows weighs nothing
#pragma unroll 1
  for (int left = r1 - r0; left > 0; left -= kGroups * kUnroll) {
    uint4 kraw[kUnroll], vraw[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      kraw[u] = vraw[u] = make_uint4(0u, 0u, 0u, 0u);
      if (g + u * kGroups < left) {
        kraw[u] = __ldcs(reinterpret_cast<const uint4*>(kp));      // streaming: every byte is read once
        vraw[u] = __ldcs(reinterpret_cast<const uint4*>(vp));
      }
      kp += k_step;
      vp += v_step;
    }
    float s[kUnroll], m_new = m;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      uint64_t t = mul_f32x2(q2[0], bf16x2_to_f32x2(kraw[u].x));
      t = fma_f32x2(q2[1], bf16x2_to_f32x2(kraw[u].y), t);
      t = fma_f32x2(q2[2], bf16x2_to_f32x2(kraw[u].z), t);
      t = fma_f32x2(q2[3], bf16x2_to_f32x2(kraw[u].w), t);
      float lo, hi;
      unpack_f32x2(t, lo, hi);
      s[u] = lo + hi;
    }
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) {
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (g + u * kGroups >= left) s[u] = -CUDART_INF_F;
      m_new = fmaxf(m_new, s[u]);
    }
    const float f = exp2f(m - m_new);
    const uint64_t f2 = pack_f32x2(f, f);
    l *= f;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = mul_f32x2(acc[i], f2);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const float pr = exp2f(s[u] - m_new);
      const uint64_t p2 = pack_f32x2(pr, pr);
      l += pr;
      acc[0] = fma_f32x2(p2, bf16x2_to_f32x2(vraw[u].x), acc[0]);
      acc[1] = fma_f32x2(p2, bf16x2_to_f32x2(vraw[u].y), acc[1]);
      acc[2] = fma_f32x2(p2, bf16x2_to_f32x2(vraw[u].z), acc[2]);
      acc[3] = fma_f32x2(p2, bf16x2_to_f32x2(vraw[u].w), acc[3]);
    }
    m = m_new;
  }
  float o[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) unpack_f32x2(acc[i], o[2 * i], o[2 * i + 1]);
#pragma unroll
  for (int off = 8; off <= 16; off <<= 1) {        // the warp's four lane groups
    const float m_o = __shfl_xor_sync(0xffffffffu, m, off), l_o = __shfl_xor_sync(0xffffffffu, l, off);
    const float m_n = fmaxf(m, m_o), fa = exp2f(m - m_n), fb = exp2f(m_o - m_n);
    l = l * fa + l_o * fb;
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = o[i] * fa + __shfl_xor_sync(0xffffffffu, o[i], off) * fb;
    m = m_n;
  }
  if ((tid & 31) < 8) {
    float* w = sm_w[tid >> 5];
    if (c == 0) { w[0] = m; w[1] = l; }
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(w + 2 + 8 * c + 2 * i) = make_float2(o[2 * i], o[2 * i + 1]);
  }
  __syncthreads();
  if (kCluster) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  float mm = kNoScore, ll = 0.f, oo = 0.f;
  if (tid < 64) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, sm_w[w][0]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = exp2f(sm_w[w][0] - mm);
      ll = fmaf(sm_w[w][1], f, ll);
      oo = fmaf(sm_w[w][2 + tid], f, oo);
    }
  }
  if (kCluster) {
    if (tid < 64) {
      uint32_t dst;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst) : "r"(smem_u32(sm_c[rank])));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + 4 * (2 + tid)), "f"(oo) : "memory");
      if (tid == 0) {
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(mm) : "memory");
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + 4), "f"(ll) : "memory");
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank != 0) return;
    if (tid < 64) {
      mm = kNoScore; ll = 0.f; oo = 0.f;
      for (int k = 0; k < ctas; ++k) mm = fmaxf(mm, sm_c[k][0]);
      for (int k = 0; k < ctas; ++k) {
        const float f = exp2f(sm_c[k][0] - mm);
        ll = fmaf(sm_c[k][1], f, ll);
        oo = fmaf(sm_c[k][2 + tid], f, oo);
      }
    }
  }
  if (tid < 64) {
    p.o[b * p.o_sb + h * p.o_sh + tid] = __float2bfloat16_rn(oo / ll);
    if (tid == 0 && p.lse != nullptr) p.lse[bh] = 0.6931471805599453f * (mm + log2f(ll));
  }
}

}  // namespace fa
