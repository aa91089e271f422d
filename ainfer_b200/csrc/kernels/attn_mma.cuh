// Attention on the tensor cores with mma.sync: tiles of 64 keys (or values) in shared memory as rows of
// DP + 8 bf16 values, fragments of 16 rows per warp, fp32 scores and sums. Shared by the attention
// kernels of the models with bf16 caches.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace ainfer {

constexpr int kCmKeys = 64;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ uint32_t cm_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}
__device__ __forceinline__ void cpa16(uint32_t dst, const void *src, bool in) {   // out of range: zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 64 keys [slot, slot + 64) of one key head into a tile of rows of DP + 8 values.
template <int DP, int THREADS>
__device__ __forceinline__ void load_keys(uint32_t dst, const uint16_t *K, int slot, int KW, int D) {
  constexpr int P = DP / 8;
  for (int i = threadIdx.x; i < kCmKeys * P; i += THREADS) {
    const int r = i / P, c = i % P;
    const bool in = c * 8 < D;
    cpa16(dst + (uint32_t)(r * (DP + 8) + c * 8) * 2, K + (size_t)(slot + r) * KW + (in ? c * 8 : 0), in);
  }
}

// One warp, 16 rows against NK keys of a tile at `kt`: s[n] = products with keys 8n .. 8n+7.
template <int DP, int NK>
__device__ __forceinline__ void scores(float (&s)[NK / 8][4], const uint32_t (&q)[DP / 16][4], uint32_t kt, int lane) {
#pragma unroll
  for (int n = 0; n < NK / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) s[n][i] = 0.0f;
  const uint32_t a = kt + (uint32_t)(((lane & 7) + ((lane >> 4) & 1) * 8) * (DP + 8) + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
  for (int kk = 0; kk < DP / 16; ++kk)
#pragma unroll
    for (int n = 0; n < NK / 16; ++n) {
      uint32_t b[4];
      ldm4(b, a + (uint32_t)(n * 16 * (DP + 8) + kk * 16) * 2);
      mma16816(s[2 * n], q[kk], b[0], b[1]);
      mma16816(s[2 * n + 1], q[kk], b[2], b[3]);
    }
}
// The same with the query fragments read from shared memory (qa: this lane's address in the warp's 16 rows).
template <int DP, int NK>
__device__ __forceinline__ void scores_smem(float (&s)[NK / 8][4], uint32_t qa, uint32_t kt, int lane) {
#pragma unroll
  for (int n = 0; n < NK / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) s[n][i] = 0.0f;
  const uint32_t a = kt + (uint32_t)(((lane & 7) + ((lane >> 4) & 1) * 8) * (DP + 8) + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
  for (int kk = 0; kk < DP / 16; ++kk) {
    uint32_t q[4];
    ldm4(q, qa + (uint32_t)(kk * 32));
#pragma unroll
    for (int n = 0; n < NK / 16; ++n) {
      uint32_t b[4];
      ldm4(b, a + (uint32_t)(n * 16 * (DP + 8) + kk * 16) * 2);
      mma16816(s[2 * n], q, b[0], b[1]);
      mma16816(s[2 * n + 1], q, b[2], b[3]);
    }
  }
}
// o += weights (as the score fragments hold them) . keys of the tile
template <int DP, int NK>
__device__ __forceinline__ void values(float (&o)[DP / 8][4], const float (&p)[NK / 8][4], uint32_t kt, int lane) {
  const uint32_t a = kt + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * (DP + 8) + ((lane >> 4) & 1) * 8) * 2;
#pragma unroll
  for (int j = 0; j < NK / 16; ++j) {
    const uint32_t w[4] = {pack2(p[2 * j][0], p[2 * j][1]), pack2(p[2 * j][2], p[2 * j][3]), pack2(p[2 * j + 1][0], p[2 * j + 1][1]),
                           pack2(p[2 * j + 1][2], p[2 * j + 1][3])};
#pragma unroll
    for (int d = 0; d < DP / 16; ++d) {
      uint32_t b[4];
      ldm4t(b, a + (uint32_t)(j * 16 * (DP + 8) + d * 16) * 2);
      mma16816(o[2 * d], w, b[0], b[1]);
      mma16816(o[2 * d + 1], w, b[2], b[3]);
    }
  }
}
__device__ __forceinline__ float fast_exp2(float x) {   // one instruction, 2 ulp, small results flushed to zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(kFull, v, 1));
  return fmaxf(v, __shfl_xor_sync(kFull, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v = v + __shfl_xor_sync(kFull, v, 1);
  return v + __shfl_xor_sync(kFull, v, 2);
}

// ---- the end of a decode step's attention: a block's warps, then the blocks of a (sequence, key head) ----
// Four warps hold sums o of up to 16 heads (a thread's heads lane / 4 and 8 more) with maxima m and sums of weights l (not yet over
// the quad). Blocks leave their share in part, sums [splits][heads][E], then (maximum, sum of weights) [splits][heads]; the last of
// `active` to come ends the heads: a share's factor exp2(m_s - M) / L first, then the shares times their factors, in their order
// (outputs travel through the layers that follow in 16 bits, so the order is part of the result). A chain of latencies, so: four
// dimensions a thread; rows of os padded, the quads of a warp store to different banks; one release and acquire, by the
// thread that counts, between two barriers, and the shares are read past L1 (fences of all threads took 1600 cycles with the
// counting and 2300 after it); the shares and what before(head, dimension) loads are under way while the factors are made. us of a step: 16
// sequences of Sinepel, four layers of 2048, at 600 280 -> 272, 64 of Robopel at 700 441 -> 434, one of Sinepel at 1500 238 -> 231.
// sink(head, the maximum): more weight in the sum. end(head, dimension, four values, what before gave).
constexpr int kStepMaxSplits = 16;
__device__ __forceinline__ uint32_t count_up(uint32_t *p) {   // release and acquire on the GPU
  uint32_t n;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(n) : "l"(p) : "memory");
  return n;
}
template <int DP, typename Sink, typename Before, typename End>
__device__ __forceinline__ void step_merge(float *os, const float (&o)[DP / 8][4], const float (&m)[2], float (&l)[2], int heads, int E, float *part,
                                           uint32_t *count, int split, int splits, int active, const Sink &sink, const Before &before, const End &end) {
  constexpr int LO = DP + 8;   // os: [4][16][LO]
  __shared__ float wm[4][16], wl[4][16];
  __shared__ int s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quads = E >> 2;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int r = (lane >> 2) + 8 * x;
    l[x] = quad_sum(l[x]);
    if ((lane & 3) == 0) { wm[warp][r] = m[x]; wl[warp][r] = l[x]; }
    if (r < heads)
#pragma unroll
      for (int d = 0; d < DP / 8; ++d) *reinterpret_cast<float2 *>(os + (warp * 16 + r) * LO + d * 8 + (lane & 3) * 2) = make_float2(o[d][2 * x], o[d][2 * x + 1]);
  }
  __syncthreads();
  float2 *part_m = reinterpret_cast<float2 *>(part + (size_t)splits * heads * E);
#pragma unroll 1
  for (int i = tid; i < heads * quads; i += 128) {
    const int hh = i / quads, d = (i - hh * quads) * 4;
    const float M = fmaxf(fmaxf(wm[0][hh], wm[1][hh]), fmaxf(wm[2][hh], wm[3][hh]));
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float L = 0.0f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = fast_exp2(wm[w][hh] - M);
      const float4 x = *reinterpret_cast<const float4 *>(os + (w * 16 + hh) * LO + d);
      v.x = fmaf(x.x, f, v.x); v.y = fmaf(x.y, f, v.y); v.z = fmaf(x.z, f, v.z); v.w = fmaf(x.w, f, v.w);
      L = fmaf(wl[w][hh], f, L);
    }
    if (active == 1) {
      const auto with = before(hh, d);
      L += sink(hh, M);
      end(hh, d, make_float4(v.x / L, v.y / L, v.z / L, v.w / L), with);
    } else {
      __stcg(reinterpret_cast<float4 *>(part + ((size_t)split * heads + hh) * E + d), v);
      if (d == 0) __stcg(part_m + split * heads + hh, make_float2(M, L));
    }
  }
  if (active == 1) return;
  __syncthreads();
  if (tid == 0) {
    s_last = count_up(count) + 1 == (uint32_t)active;
    if (s_last) *count = 0;
  }
  __syncthreads();
  if (!s_last) return;
  static_assert(16 * kStepMaxSplits <= 4 * 16 * LO, "the factors lie in the sums' place");
  float *fac = os;   // [16][kStepMaxSplits]
  const int n = heads * quads;
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += 128) {
    const int i = min(i0 + tid, n - 1), hh = i / quads, d = (i - hh * quads) * 4;
    const auto with = before(hh, d);
    float4 x[kStepMaxSplits], v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int s = 0; s < kStepMaxSplits; ++s) x[s] = __ldcg(reinterpret_cast<const float4 *>(part + ((size_t)min(s, active - 1) * heads + hh) * E + d));
    if (i0 == 0) {   // a lane a share, a warp every fourth head
      float2 ml[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = warp + 4 * u;
        ml[u] = r < heads && lane < active ? __ldcg(part_m + lane * heads + r) : make_float2(-INFINITY, 0.0f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = warp + 4 * u;
        if (r >= heads) break;
        const float M = warp_max(ml[u].x), f = fast_exp2(ml[u].x - M), L = warp_tree_sum(ml[u].y * f) + sink(r, M);
        if (lane < kStepMaxSplits) fac[r * kStepMaxSplits + lane] = lane < active ? f / L : 0.0f;
      }
      __syncthreads();
    }
    const float *f = fac + hh * kStepMaxSplits;
#pragma unroll
    for (int s = 0; s < kStepMaxSplits; ++s) {
      const float w = f[s];
      v.x = fmaf(x[s].x, w, v.x); v.y = fmaf(x[s].y, w, v.y); v.z = fmaf(x[s].z, w, v.z); v.w = fmaf(x[s].w, w, v.w);
    }
    if (i0 + tid < n) end(hh, d, v, with);
  }
}

}  // namespace ainfer
