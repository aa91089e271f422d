// Dense layers with bf16 weights W [N][ldw] (rows padded with zeros to a multiple of 8 values).
//
//   LinearRows*       fp32 activations, fp32 sums on the CUDA cores (the 32-bit form)
//   StreamGemv        one fp32 row, weights streamed once: y = act(W x + bias)
//   HyperStreamGemv   the same, x made in the kernel from the residual streams: stream update of the
//                     previous sublayer, weighted read, RMS norm, optional token shift (every block
//                     makes the row for itself; block 0 stores the updated streams and the shift row)
// act: 0 none, 1 relu squared, 2 cap tanh(v / cap).
#include "hyper_core.cuh"
#include "linear_rows.cuh"
#include "stream_gemv.cuh"

namespace ainfer {

// ---------------------------------------------------------- LinearRows ---
struct LinearRowsArgs {
  const float *X;        // [rows][ldx]
  const uint16_t *W;     // [N][ldw]
  const float *Bias;     // [N] or null
  float *Y;              // [rows][ldy]
  int32_t rows, N, K, ldx, ldw, ldy, act;
  float cap;
};
// Tiles of BM rows and BN outputs; the CL blocks of a cluster share a tile, each a part of K (whole steps of 16),
// and add their sums up in rank order through shared memory, each for its share of the tile's rows.
// 64 x 128 tiles for rows in plenty, 64 x 64 where those are too few, 16 x 128 for up to 16 rows: a tile of 64 would multiply
// zeros mostly. A thread's 8 x 8 sums take four 16-byte reads of shared memory a column of K for 32 packed multiply-adds, which
// keeps the reads as busy as the multipliers; 8 x 16 takes six for 64 (777 rows x 4096 x 1024: 192 / 163 us).
template <int BM, int BN, int CL>
__device__ __forceinline__ void linear_rows_body(const LinearRowsArgs &a) {
  using Tile = LinearRowsTile<BM, BN>;
  __shared__ __align__(16) union { typename Tile::Shared tiles; float sums[BM][BN]; } sh;
  const int nt = (a.N + BN - 1) / BN, t = blockIdx.x / CL, rank = CL > 1 ? blockIdx.x % CL : 0;
  const int n0 = t % nt * BN, r0 = t / nt * BM, nr = min(BM, a.rows - r0);
  pdl_launch_dependents();
  pdl_wait();
  const int steps = (a.K + kLrK - 1) / kLrK, per = (steps + CL - 1) / CL;
  Tile c;
  if (nr > 0)
    c.run(sh.tiles, a.X + (size_t)r0 * a.ldx, a.ldx, nr, a.W + (size_t)n0 * a.ldw, a.ldw, a.N - n0, min(a.K, rank * per * kLrK),
          min(a.K, (rank + 1) * per * kLrK));
  auto put = [&](int r, int n, const float (&v)[4]) {   // four outputs of a row
    if (r >= nr) return;
    float *y = a.Y + (size_t)(r0 + r) * a.ldy;
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = n + j < a.N ? apply_act(v[j] + (a.Bias ? a.Bias[n + j] : 0.0f), a.act, a.cap) : 0.0f;
    if (n + 3 < a.N && ((a.ldy & 3) == 0 && ((uintptr_t)a.Y & 15) == 0)) {
      *reinterpret_cast<float4 *>(y + n) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < a.N) y[n + j] = o[j];
    }
  };
  if constexpr (CL == 1) {
#pragma unroll
    for (int i = 0; i < Tile::TM; ++i)
#pragma unroll
      for (int j = 0; j < Tile::TN; j += 4) {
        const float v[4] = {c.acc[i][j], c.acc[i][j + 1], c.acc[i][j + 2], c.acc[i][j + 3]};
        put(Tile::row(i), n0 + Tile::col(j), v);
      }
  } else {
    __syncthreads();   // the last step's readers are done
#pragma unroll
    for (int i = 0; i < Tile::TM; ++i)
#pragma unroll
      for (int j = 0; j < Tile::TN; j += 4)
        *reinterpret_cast<float4 *>(&sh.sums[Tile::row(i)][Tile::col(j)]) = make_float4(c.acc[i][j], c.acc[i][j + 1], c.acc[i][j + 2], c.acc[i][j + 3]);
    cluster_sync_all();
    for (int i = threadIdx.x; i < BM * BN / CL / 4; i += kLrThreads) {
      const int r = rank * (BM / CL) + i / (BN / 4), n = i % (BN / 4) * 4;
      uint32_t at = smem_addr(&sh.sums[r][n]);
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int s = 0; s < CL; ++s) {
        uint32_t peer;
        float p[4];
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(s));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p[0]), "=f"(p[1]), "=f"(p[2]), "=f"(p[3]) : "r"(peer) : "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += p[j];
      }
      put(r, n0 + n, v);
    }
    cluster_sync_all();   // a block's sums stay until every reader is done
  }
}
#define F(f) AINFER_ARG(LinearRowsArgs, f)
#define LR_FIELDS F(X), F(W), F(Bias), F(Y), F(rows), F(N), F(K), F(ldx), F(ldw), F(ldy), F(act), F(cap)
#define LR_KERNEL(NAME, BM, BN, CL)                                                                                                        \
  __global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(kLrThreads) NAME(const LinearRowsArgs a) { linear_rows_body<BM, BN, CL>(a); } \
  AINFER_REGISTER(NAME, LinearRowsArgs, kLrThreads, 0, 0, nullptr, LR_FIELDS)
__global__ void __launch_bounds__(kLrThreads) LinearRows(const LinearRowsArgs a) { linear_rows_body<64, 64, 1>(a); }
AINFER_REGISTER(LinearRows, LinearRowsArgs, kLrThreads, 0, 0, nullptr, LR_FIELDS);
__global__ void __launch_bounds__(kLrThreads) LinearRowsFew(const LinearRowsArgs a) { linear_rows_body<16, 128, 1>(a); }
AINFER_REGISTER(LinearRowsFew, LinearRowsArgs, kLrThreads, 0, 0, nullptr, LR_FIELDS);
AINFER_EARLY_LAUNCH(LinearRowsFew);
__global__ void __launch_bounds__(kLrThreads) LinearRowsWide(const LinearRowsArgs a) { linear_rows_body<64, 128, 1>(a); }
AINFER_REGISTER(LinearRowsWide, LinearRowsArgs, kLrThreads, 0, 0, nullptr, LR_FIELDS);
LR_KERNEL(LinearRowsWideSplit2, 64, 128, 2);
LR_KERNEL(LinearRowsWideSplit4, 64, 128, 4);
LR_KERNEL(LinearRowsWideSplit8, 64, 128, 8);
LR_KERNEL(LinearRowsSplit2, 64, 64, 2);
LR_KERNEL(LinearRowsSplit4, 64, 64, 4);
LR_KERNEL(LinearRowsSplit8, 64, 64, 8);
LR_KERNEL(LinearRowsFewSplit2, 16, 128, 2);
LR_KERNEL(LinearRowsFewSplit4, 16, 128, 4);
LR_KERNEL(LinearRowsFewSplit8, 16, 128, 8);
// The 64 x 64 tiles do not come up early: the blocks would gather on the SMs that the predecessor leaves first, and
// a launch of a few blocks an SM lasts as long as the fullest one (777-token prompt 1720 us, with early blocks 1860).
AINFER_EARLY_LAUNCH(LinearRowsFewSplit2);
AINFER_EARLY_LAUNCH(LinearRowsFewSplit4);
AINFER_EARLY_LAUNCH(LinearRowsFewSplit8);
#undef F

// ---------------------------------------------------------- StreamGemv ---
struct StreamGemvArgs {
  const float *X;        // [K]
  const uint16_t *W;
  const float *Bias;     // [N] or null
  float *Y;              // [N]
  int32_t N, K, ldw, rows_pb, act;
  float cap;
};
__global__ void __launch_bounds__(kSgThreads, 4) StreamGemv(const StreamGemvArgs a) {
  __shared__ GemvShared sh;
  pdl_launch_dependents();
  const GemvDims d = gemv_dims(a.ldw);
  const GemvShape c{a.W, a.Bias, a.Y, a.N, a.ldw, a.rows_pb, a.act, a.cap};
  float *lo = reinterpret_cast<float *>(sg_smem + d.nst * d.stage_bytes), *hi = lo + a.ldw / 2, *part = hi + a.ldw / 2;
  gemv_init(&sh, d.nst);
  if (threadIdx.x >= kSgWarps * 32) {
    gemv_produce(c, d, &sh, sg_smem);
  } else {
    pdl_wait();
    sg_row(lo, hi, a.X, a.K, a.ldw, threadIdx.x, kSgWarps * 32);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    gemv_consume(c, d, &sh, sg_smem, lo, hi, part);
  }
  __syncthreads();
  gemv_store(c, d, part);
}
static uint32_t stream_gemv_smem(const void *args) {
  const StreamGemvArgs *a = (const StreamGemvArgs *)args;
  return gemv_smem(a->ldw, a->rows_pb, 0);
}
#define F(f) AINFER_ARG(StreamGemvArgs, f)
AINFER_REGISTER(StreamGemv, StreamGemvArgs, kSgThreads, 0, 0, stream_gemv_smem, F(X), F(W), F(Bias), F(Y), F(N), F(K), F(ldw), F(rows_pb),
                F(act), F(cap));
#undef F

struct HyperStreamGemvArgs {
  const float *Xin;        // [S][K] streams
  const float *Yp;         // [K] output of the sublayer whose update is pending; null: none
  const float *Mix, *Out;  // of that sublayer
  float *Xout;             // [S][K] (another buffer than Xin); null: not stored
  const float *In;         // [S]; null: plain sum
  const float *NormW;      // [K]
  const float *Shift;      // [K] or null
  float *State;            // [2][K] shift rows by position parity
  const int32_t *Ctrl;
  const uint16_t *W;
  const float *Bias;
  float *Y;
  int32_t S, N, K, ldw, rows_pb, act;
  float eps, cap;
  int32_t ahead;           // LaunchAhead
};
// The row of up to 2048 elements in whole quads and four streams: everything that does not come from the sublayer
// before (norm weights, shift, the last position's row in a list of one step) is in registers before the dependency wait, the streams
// and the sublayer's output are one round of loads after it. In loops (as below) every element's norm weight,
// shift and last row were one more round each. (One number of streams only: every other one is as much code again.)
constexpr int kHgQuads = 2;
template <int ST>
__device__ __forceinline__ void hyper_row_ahead(const HyperStreamGemvArgs &a, const StreamCoef &coef, float *lo, float *hi, float *red) {
  const int K = a.K, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = kSgWarps * 32;
  if (!(a.ahead & AHEAD_STATE)) pdl_wait();
  const int pos = a.Shift ? a.Ctrl[CTRL_POS] : 0;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float4 nw[kHgQuads], sf[kHgQuads], pv[kHgQuads];
#pragma unroll
  for (int q = 0; q < kHgQuads; ++q) {
    const int k = (q * nth + tid) * 4;
    nw[q] = k < K ? ld_val4(a.NormW + k) : zero;
    sf[q] = a.Shift && k < K ? ld_val4(a.Shift + k) : zero;
    pv[q] = a.Shift && pos > 0 && k < K ? ld_val4(a.State + (size_t)((pos - 1) & 1) * K + k) : zero;   // of the step before
  }
  pdl_wait();
  const bool update = a.Yp != nullptr;
  float4 x[kHgQuads][ST], y[kHgQuads];
#pragma unroll
  for (int q = 0; q < kHgQuads; ++q) {
    const int k = (q * nth + tid) * 4;
#pragma unroll
    for (int s = 0; s < ST; ++s) x[q][s] = k < K ? ld_val4(a.Xin + (size_t)s * K + k) : zero;
    y[q] = update && k < K ? ld_val4(a.Yp + k) : zero;
  }
  float *dst = blockIdx.x == 0 ? a.Xout : nullptr;
  float u[kHgQuads][4], ss = 0.0f;
#pragma unroll
  for (int q = 0; q < kHgQuads; ++q) {
    const int k = (q * nth + tid) * 4;
    stream_update<ST>(x[q], y[q], dst && k < K ? dst + k : nullptr, coef, K, update, u[q]);
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = fmaf(u[q][i], u[q][i], ss);
  }
  ss = warp_tree_sum(ss);
  if (lane == 0) red[warp] = ss;
  asm volatile("bar.sync 1, 256;" ::: "memory");
  ss = warp_tree_sum(lane < kSgWarps ? red[lane] : 0.0f);
  const float inv = 1.0f / sqrtf(ss / (float)K + a.eps);
  float *next = a.Shift && blockIdx.x == 0 ? a.State + (size_t)(pos & 1) * K : nullptr;
#pragma unroll
  for (int q = 0; q < kHgQuads; ++q) {
    const int k = (q * nth + tid) * 4;
    float4 v = make_float4(u[q][0] * inv * nw[q].x, u[q][1] * inv * nw[q].y, u[q][2] * inv * nw[q].z, u[q][3] * inv * nw[q].w);
    if (next && k < K) st_val4(next + k, v);
    if (a.Shift) {
      v.x = fmaf(pv[q].x - v.x, sf[q].x, v.x); v.y = fmaf(pv[q].y - v.y, sf[q].y, v.y);
      v.z = fmaf(pv[q].z - v.z, sf[q].z, v.z); v.w = fmaf(pv[q].w - v.w, sf[q].w, v.w);
    }
    if (k < a.ldw) st_val4(((k & 4) ? hi : lo) + (k >> 3) * 4, v);   // zeros between K and ldw
  }
}
__global__ void __launch_bounds__(kSgThreads, 3) HyperStreamGemv(const HyperStreamGemvArgs a) {
  __shared__ GemvShared sh;
  __shared__ StreamCoef coef;
  __shared__ float red[33];
  pdl_launch_dependents();
  const GemvDims d = gemv_dims(a.ldw);
  const GemvShape c{a.W, a.Bias, a.Y, a.N, a.ldw, a.rows_pb, a.act, a.cap};
  const int K = a.K, tid = threadIdx.x, nth = kSgWarps * 32;
  float *lo = reinterpret_cast<float *>(sg_smem + d.nst * d.stage_bytes), *hi = lo + a.ldw / 2, *us = hi + a.ldw / 2,
        *part = us + ((K + 3) & ~3);
  load_stream_coef(coef, a.Mix, a.Out, a.In, a.S);
  gemv_init(&sh, d.nst);
  if (tid >= nth) {
    gemv_produce(c, d, &sh, sg_smem);
  } else {
    if (a.S == 4 && stream_vec(a.S, K) && K <= kHgQuads * nth * 4 && on_quads(a.NormW, a.Shift, a.State)) {
      hyper_row_ahead<4>(a, coef, lo, hi, red);
    } else {
      const int lane = tid & 31, warp = tid >> 5;
      pdl_wait();
      float ss = stream_row_any(a.Xin, a.Yp, blockIdx.x == 0 ? a.Xout : nullptr, coef, a.S, K, a.Yp != nullptr, us, tid, nth);
      ss = warp_tree_sum(ss);
      if (lane == 0) red[warp] = ss;
      asm volatile("bar.sync 1, 256;" ::: "memory");   // also: every thread's u is visible
      ss = warp_tree_sum(lane < kSgWarps ? red[lane] : 0.0f);
      const float inv = 1.0f / sqrtf(ss / (float)K + a.eps);
      const int pos = a.Shift ? a.Ctrl[CTRL_POS] : 0;
      const float *prev = a.Shift ? a.State + (size_t)((pos - 1) & 1) * K : nullptr;
      float *next = a.Shift && blockIdx.x == 0 ? a.State + (size_t)(pos & 1) * K : nullptr;
      for (int k = tid; k < a.ldw; k += nth) {
        float v = 0.0f;
        if (k < K) {
          v = us[k] * inv * a.NormW[k];
          if (a.Shift) {
            const float pv = pos > 0 ? prev[k] : 0.0f;
            if (next) next[k] = v;
            v = fmaf(pv - v, a.Shift[k], v);
          }
        }
        sg_put(lo, hi, k, v);
      }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    gemv_consume(c, d, &sh, sg_smem, lo, hi, part);
  }
  __syncthreads();
  gemv_store(c, d, part);
}
static uint32_t hyper_gemv_smem(const void *args) {
  const HyperStreamGemvArgs *a = (const HyperStreamGemvArgs *)args;
  return gemv_smem(a->ldw, a->rows_pb, (a->K + 3) & ~3);
}
#define F(f) AINFER_ARG(HyperStreamGemvArgs, f)
AINFER_REGISTER(HyperStreamGemv, HyperStreamGemvArgs, kSgThreads, 0, 0, hyper_gemv_smem, F(Xin), F(Yp), F(Mix), F(Out), F(Xout), F(In),
                F(NormW), F(Shift), F(State), F(Ctrl), F(W), F(Bias), F(Y), F(S), F(N), F(K), F(ldw), F(rows_pb), F(act), F(eps), F(cap));
#undef F

// Copies [N][K] bf16 rows to rows of ld values, zero padded.
struct PackRowsBf16Args {
  uint16_t *Dst;
  const uint16_t *Src;
  int32_t N, K, ld;
};
__global__ void __launch_bounds__(256) PackRowsBf16(const PackRowsBf16Args a) {
  for (int n = blockIdx.x; n < a.N; n += gridDim.x)
    for (int k = threadIdx.x; k < a.ld; k += 256) a.Dst[(size_t)n * a.ld + k] = k < a.K ? a.Src[(size_t)n * a.K + k] : (uint16_t)0;
}
#define F(f) AINFER_ARG(PackRowsBf16Args, f)
AINFER_REGISTER(PackRowsBf16, PackRowsBf16Args, 256, 0, 0, nullptr, F(Dst), F(Src), F(N), F(K), F(ld));
#undef F

AINFER_EARLY_LAUNCH(StreamGemv);
AINFER_EARLY_LAUNCH_AHEAD(HyperStreamGemv, HyperStreamGemvArgs);

}  // namespace ainfer
