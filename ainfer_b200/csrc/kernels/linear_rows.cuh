// A tile of Y = X W^T on the CUDA cores: fp32 activations, bf16 weights, fp32 fused multiply-adds. What the
// 32-bit products of rows share (LinearRows*, LinearRowsGrouped).
//
// Bound by the fused multiply-add rate, so the tile is held in registers: a thread owns TM x TN sums and meets
// every k with TM + TN values that it reads as 16-byte pieces from shared memory (8 x 8: four reads for 64
// multiply-adds; 4 x 4 with single loads spent as many cycles on reads as on sums). The next 16 columns of both
// operands are on their way to registers while the present ones are multiplied; two shared buffers, one barrier
// a step. 64 threads a block: several blocks an SM keep the schedulers fed, and small matrices still give every SM
// one. Two neighbouring columns' sums are one packed multiply-add: half the instructions to issue beside the reads. 777 rows x 4096
// outputs x 1024: 349 us with 4 x 4 sums, 209 with 8 x 8, 192 packed (34 TFLOP/s); x 1024 x 4096 (K in four parts):
// 607, 208, 197; one row x 32000 x 1024 (16 x 128 tiles): 256, 60, 59.
#pragma once
#include "row_types.cuh"

namespace ainfer {

constexpr int kLrThreads = 64, kLrK = 16;

template <int BM, int BN>
struct LinearRowsShared {
  float x[2][kLrK][BM], w[2][kLrK][BN];
};

template <int BM, int BN>
struct LinearRowsTile {
  static constexpr int TM = BM == 64 ? 8 : 4, TN = BM == 64 ? BN / 8 : 8, TX = BN / TN;
  static_assert(BM / TM * TX == kLrThreads && TM % 4 == 0, "64 threads own the tile");
  static constexpr int XP = BM * kLrK / kLrThreads, XR = kLrThreads / BM;   // values of a thread, threads of a row
  static constexpr int WN = BN / kLrThreads;                                // weight rows of a thread
  using Shared = LinearRowsShared<BM, BN>;

  float acc[TM][TN];
  float xr[XP];
  uint4 wr[WN][2];

  // Rows and columns of the thread's sums: quads, spread evenly over the tile.
  __device__ static int row(int i) { return (i >> 2) * (BM / (TM / 4)) + (int)threadIdx.x / TX * 4 + (i & 3); }
  __device__ static int col(int j) { return (j >> 2) * (BN / (TN / 4)) + (int)threadIdx.x % TX * 4 + (j & 3); }

  // Columns [k0, k0 + 16) of `rows` rows of X and `cols` rows of W: zeros beyond K; rows and columns past the last repeat
  // it (their sums are not stored).
  __device__ __forceinline__ void fetch(const float *X, int ldx, int rows, const uint16_t *W, int ldw, int cols, int k0, int K, bool vec) {
    const int tid = threadIdx.x, r = tid % BM, kx = tid / BM * XP;
    const bool whole = vec && k0 + kLrK <= K;
    const float *px = X + (size_t)min(r, rows - 1) * ldx + k0 + kx;
    if (whole) {
#pragma unroll
      for (int i = 0; i < XP; i += 4) *reinterpret_cast<float4 *>(xr + i) = *reinterpret_cast<const float4 *>(px + i);
    } else {
#pragma unroll
      for (int i = 0; i < XP; ++i) xr[i] = k0 + kx + i < K ? px[i] : 0.0f;
    }
#pragma unroll
    for (int n = 0; n < WN; ++n) {
      const uint16_t *pw = W + (size_t)min(tid + n * kLrThreads, cols - 1) * ldw + k0;
      if (whole) {
        wr[n][0] = __ldg(reinterpret_cast<const uint4 *>(pw));
        wr[n][1] = __ldg(reinterpret_cast<const uint4 *>(pw + 8));
      } else {
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t a = k0 + 2 * i < K ? pw[2 * i] : 0u, b = k0 + 2 * i + 1 < K ? pw[2 * i + 1] : 0u;
          v[i] = a | (b << 16);
        }
        wr[n][0] = make_uint4(v[0], v[1], v[2], v[3]);
        wr[n][1] = make_uint4(v[4], v[5], v[6], v[7]);
      }
    }
  }
  // The lanes of a warp store consecutive rows of one column: no bank is met twice.
  __device__ __forceinline__ void store(Shared &sh, int b) {
    const int tid = threadIdx.x, r = tid % BM, kx = tid / BM * XP;
#pragma unroll
    for (int i = 0; i < XP; ++i) sh.x[b][kx + i][r] = xr[i];
#pragma unroll
    for (int n = 0; n < WN; ++n) {
      const uint32_t v[8] = {wr[n][0].x, wr[n][0].y, wr[n][0].z, wr[n][0].w, wr[n][1].x, wr[n][1].y, wr[n][1].z, wr[n][1].w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        sh.w[b][2 * i][tid + n * kLrThreads] = u2f(v[i] << 16);
        sh.w[b][2 * i + 1][tid + n * kLrThreads] = u2f(v[i] & 0xFFFF0000u);
      }
    }
  }
  // acc = the tile's sums over columns [k_lo, k_hi), in ascending order. X and W point at the tile's first rows.
  // All threads; the shared buffers are free again only after the caller's next barrier.
  __device__ __forceinline__ void run(Shared &sh, const float *X, int ldx, int rows, const uint16_t *W, int ldw, int cols, int k_lo, int k_hi) {
    const bool vec = (((uintptr_t)X | (uintptr_t)W) & 15) == 0 && (ldx & 3) == 0 && (ldw & 7) == 0;   // k_lo is a multiple of 16
    uint64_t sums[TM][TN / 2];   // of neighbouring columns in pairs
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) sums[i][j] = 0;
    unpack(sums);
    const int tx = threadIdx.x % TX * 4, ty = threadIdx.x / TX * 4;
    if (k_lo >= k_hi) return;
    fetch(X, ldx, rows, W, ldw, cols, k_lo, k_hi, vec);
    store(sh, 0);
    __syncthreads();
    int b = 0;
    for (int k0 = k_lo; k0 < k_hi; k0 += kLrK, b ^= 1) {
      const bool more = k0 + kLrK < k_hi;
      if (more) fetch(X, ldx, rows, W, ldw, cols, k0 + kLrK, k_hi, vec);
#pragma unroll
      for (int k = 0; k < kLrK; ++k) {
        float xv[TM];
        ulonglong2 wv[TN / 4];
#pragma unroll
        for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4 *>(xv + i) = *reinterpret_cast<const float4 *>(&sh.x[b][k][i / 4 * (BM / (TM / 4)) + ty]);
#pragma unroll
        for (int j = 0; j < TN; j += 4) wv[j / 4] = *reinterpret_cast<const ulonglong2 *>(&sh.w[b][k][j / 4 * (BN / (TN / 4)) + tx]);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const uint64_t x2 = pair2(xv[i], xv[i]);
#pragma unroll
          for (int j = 0; j < TN / 4; ++j) {
            sums[i][2 * j] = fma2(x2, wv[j].x, sums[i][2 * j]);
            sums[i][2 * j + 1] = fma2(x2, wv[j].y, sums[i][2 * j + 1]);
          }
        }
      }
      if (more) {
        store(sh, b ^ 1);   // its readers passed the barrier of the step before
        __syncthreads();
      }
    }
    unpack(sums);
  }
  __device__ __forceinline__ void unpack(const uint64_t (&sums)[TM][TN / 2]) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const float2 v = unpair2(sums[i][j]);
        acc[i][2 * j] = v.x;
        acc[i][2 * j + 1] = v.y;
      }
  }
};

}  // namespace ainfer
