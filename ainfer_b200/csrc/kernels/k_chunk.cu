// Chunk path of the Gated DeltaNet layer: M consecutive tokens per launch, with the conv history
// and the recurrent state carried from row to row on the chip and across launches in memory.
// Replaces ChunkSsmConv and ChunkSsmRecur of the reference (tools/cmdlist/kernels.cpp:896-917,
// 919-999; host mirror tools/cmdlist/chunkssm_replay.cpp:220-255). Like the reference's, the
// chunk kernels run the sequential recurrence (row m + 1 sees the state row m left), so a chunk
// of M rows is bit-identical to M decode steps; what changes is where the state lives: a block
// owns 32 columns of one head's 128x128 state in registers for the whole chunk, reads it once
// and writes it once, instead of once per token.
#include "deltanet_core.cuh"

namespace ainfer {

// ---- ChunkConvSilu: depthwise conv (k = 4) + SiLU over M rows, history chained through the chunk ----
struct ChunkConvSiluArgs {
  float *Mx;          // [M][C] conv outputs (SiLU applied)
  const float *QKV;   // [M][C] projections
  float *CS;          // [C][3] history, updated
  const float *CW;    // [C][4] taps
  int32_t C, M;
  float *Snap;        // optional: the history [C][3] after row m at Snap + m * snap_stride (to roll a speculative chunk back); null: none
  int64_t snap_stride;
};
// Launched with ceil(C / 256) x (any number of) blocks: the rows are cut into at most that many runs, since a
// row needs the three before it and not their results. (One run for all rows was a chain of loads: 109 us for
// 192 rows of 8192 channels; runs of 16 rows 12 us.) No run but the last is shorter than the history's three
// rows, so that only the first one's threads read the history, and they are the ones that replace it.
// With more than one run Mx and QKV are different buffers.
__global__ void __launch_bounds__(256) ChunkConvSilu(const ChunkConvSiluArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int cb = (a.C + 255) / 256, runs = max(1, (int)gridDim.x / cb), run = blockIdx.x / cb;
  const int c = (blockIdx.x % cb) * 256 + threadIdx.x;
  const int per = max(3, (a.M + runs - 1) / runs), m0 = run * per, m1 = min(m0 + per, a.M);
  if (c >= a.C || run >= runs || (m0 >= m1 && run > 0)) return;
  // rows before the first come from the history, oldest first
  auto row = [&](int m) { return m >= 0 ? a.QKV[(size_t)m * a.C + c] : a.CS[c * 3 + 3 + m]; };
  float h0 = row(m0 - 3), h1 = row(m0 - 2), h2 = row(m0 - 1);
  if (run == 0) {
    const float n0 = row(a.M - 3), n1 = row(a.M - 2), n2 = row(a.M - 1);
    a.CS[c * 3 + 0] = n0; a.CS[c * 3 + 1] = n1; a.CS[c * 3 + 2] = n2;
  }
  const float4 w = __ldg(reinterpret_cast<const float4 *>(a.CW) + c);
#pragma unroll 4
  for (int m = m0; m < m1; ++m) {
    const float x = a.QKV[(size_t)m * a.C + c];
    float acc = h0 * w.x;
    acc = acc + h1 * w.y;
    acc = acc + h2 * w.z;
    acc = acc + x * w.w;
    a.Mx[(size_t)m * a.C + c] = acc / (1.0f + det_expf(-acc));
    h0 = h1; h1 = h2; h2 = x;
    if (a.Snap) {
      float *sn = a.Snap + (size_t)m * a.snap_stride + (size_t)c * 3;
      sn[0] = h0; sn[1] = h1; sn[2] = h2;
    }
  }
}

// ---- ChunkBetaDecay: beta = sigmoid(b), g = -exp(A_log) * softplus(a + dt_bias) for M rows ----
// (BetaG, tools/cmdlist/kernels.cpp:606-617; the arithmetic of the decode GEMV's epilogues.)
struct ChunkBetaDecayArgs {
  const float *B;        // [M][nV] in_proj_b outputs
  const float *A;        // [M][nV] in_proj_a outputs
  const float *ALog;     // [nV]
  const float *DtBias;   // [nV]
  float *Bt;             // [M][nV]
  float *Gt;             // [M][nV]
  int32_t nV, count;     // count = M * nV
};
__global__ void __launch_bounds__(256) ChunkBetaDecay(const ChunkBetaDecayArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= a.count) return;
  const int h = i % a.nV;
  a.Bt[i] = 1.0f / (1.0f + det_expf(-a.B[i]));
  const float sa = a.A[i] + a.DtBias[h];
  const float soft = sa > 20.0f ? sa : det_logf(1.0f + det_expf(sa));
  a.Gt[i] = (-det_expf(a.ALog[h])) * soft;
}

// ---- ChunkDeltaNet: the gated delta rule over M rows ----
struct ChunkDeltaNetArgs {
  float *Out;        // [M][nV][128] head outputs
  const float *Mx;   // [M][C] conv outputs, a row = [q: nK*128 | k: nK*128 | v: nV*128]
  float *S;          // [nV][128][128] state, row-major [k][v], updated
  const float *Bt;   // [M][nV] beta
  const float *Gt;   // [M][nV] log decay
  int32_t nK, nV, M;
  float *Snap;       // optional: the state [nV][128][128] after row m at Snap + m * snap_stride (to roll a speculative chunk back); null: none
  int64_t snap_stride;
};
constexpr int kChunkRows = 32;      // rows whose normalised q / k are staged at a time (two buffers)
constexpr int kChunkWarps = 4, kChunkHelpers = 8, kChunkThreads = (kChunkWarps + kChunkHelpers) * 32;
constexpr int kChunkRow = 4 * 36;   // floats of a staged row: four quarters of 32, apart so that a warp's reads of them meet different banks
constexpr int kChunkBuffer = kChunkRows * (2 * kChunkRow + 32);   // floats: q, k, the slice's values

extern __shared__ __align__(16) float chunk_smem[];

// One block per (head, 32-column slice); grid = nV * 4. Per row the arithmetic of deltanet_step_body:
// S *= exp(g); kv = tree8 of 16-row fma chains; d = (v - kv) * beta; S += k d; o = tree8 of fma chains
// with q. A warp holds eight columns, a lane two of a column's eight segments of 16 rows (two chains side by
// side, one packed instruction for both), so that the tree is one addition and two exchanges inside the warp and the rows of a
// chunk need no barrier; a row's output is summed beside the next row's kv. Eight more warps normalise the next chunk's
// q and k meanwhile and fetch its values. Bound by the chain of a row. (Segments in different warps, two
// block barriers a row: 130 us for 192 rows of 32 heads; this form 58. 701 rows: 199 us with scalar, 193 with packed instructions;
// output and next row's kv in one pass over the state 215, and with one segment of two columns a lane 226: what a pass more costs in
// reads of shared memory or in exchanges is more than the chain it shortens.)
__global__ void __launch_bounds__(kChunkThreads) ChunkDeltaNet(const ChunkDeltaNetArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int D = 128, SEG = kDnSeg;
  __shared__ float s_beta[2][kChunkRows], s_gt[2][kChunkRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x / kDnSlices, slice = blockIdx.x % kDnSlices;
  if (h >= a.nV) return;
  const int kh = h / (a.nV / a.nK);
  const int C = 2 * a.nK * D + a.nV * D;
  const int chunks = (a.M + kChunkRows - 1) / kChunkRows;
  auto stage = [&](int ch) {   // l2norm of the rows' q and k (a warp per (row, which)), values, beta and decay of the rows
    float *qs = chunk_smem + (ch & 1) * kChunkBuffer, *ks = qs + kChunkRows * kChunkRow, *vs = ks + kChunkRows * kChunkRow;
    const int m0 = ch * kChunkRows, rows = min(kChunkRows, a.M - m0), hw = warp - kChunkWarps;
    const int which = hw & 1;
    const float *base = a.Mx + (size_t)m0 * C;
    const float *src = base + (which == 0 ? (size_t)kh * D : (size_t)a.nK * D + (size_t)kh * D) + lane;
    for (int m = hw >> 1; m < rows; m += 2 * kChunkHelpers) {   // four rows' loads in flight
      float x[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float *r = src + (size_t)min(m + u * (kChunkHelpers / 2), rows - 1) * C;
#pragma unroll
        for (int i = 0; i < 4; ++i) x[u][i] = r[32 * i];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int mm = m + u * (kChunkHelpers / 2);
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) ss = fmaf(x[u][i], x[u][i], ss);
        ss = warp_tree_sum(ss);
        const float inv = 1.0f / sqrtf(ss + 1e-6f);
        const float f = inv * (which == 0 ? 0.0883883476483184405f : 1.0f);  // 128^-1/2 for q
        float *dst = (which == 0 ? qs : ks) + mm * kChunkRow;
        if (mm < rows) {
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[36 * i + 2 * (lane & 15) + (lane >> 4)] = x[u][i] * f;   // the two segments of a quarter take turns
        }
      }
    }
    float v[kChunkRows / kChunkHelpers];
#pragma unroll
    for (int u = 0; u < kChunkRows / kChunkHelpers; ++u)
      v[u] = base[(size_t)min(hw + u * kChunkHelpers, rows - 1) * C + (size_t)2 * a.nK * D + (size_t)h * D + slice * 32 + lane];
#pragma unroll
    for (int u = 0; u < kChunkRows / kChunkHelpers; ++u) vs[(hw + u * kChunkHelpers) * 32 + lane] = v[u];
    const int m = (int)threadIdx.x - kChunkWarps * 32;
    if (m < rows) {
      s_beta[ch & 1][m] = a.Bt[(size_t)(m0 + m) * a.nV + h];
      s_gt[ch & 1][m] = det_expf(a.Gt[(size_t)(m0 + m) * a.nV + h]);
    }
  };
  const bool helper = warp >= kChunkWarps;
  const int quarter = lane & 3, wcol = warp * 8 + (lane >> 2), col = slice * 32 + wcol;   // a lane's segments: 2 quarter, 2 quarter + 1
  float *Sh = a.S + (size_t)h * D * D + (size_t)quarter * (2 * SEG) * D + col;
  uint64_t s[SEG];   // row r of the lane's two segments
  float po = 0.0f;
  float *out = a.Out + (size_t)h * D + col;   // of the last row begun
  if (helper) {
    if (chunks > 0) stage(0);
  } else {
#pragma unroll
    for (int r = 0; r < SEG; ++r) s[r] = pair2(Sh[(size_t)r * D], Sh[(size_t)(SEG + r) * D]);
  }
  __syncthreads();
  for (int ch = 0; ch < chunks; ++ch) {
    if (helper) {
      if (ch + 1 < chunks) stage(ch + 1);
    } else {
      const float *qs = chunk_smem + (ch & 1) * kChunkBuffer, *ks = qs + kChunkRows * kChunkRow, *vs = ks + kChunkRows * kChunkRow + wcol;
      const int m0 = ch * kChunkRows, rows = min(kChunkRows, a.M - m0);
      qs += quarter * 36;
      ks += quarter * 36;
#pragma unroll 1
      for (int m = 0; m < rows; ++m) {
        const float gt = s_gt[ch & 1][m], beta = s_beta[ch & 1][m], val = vs[m * 32];
        uint64_t k[SEG], q[SEG];
#pragma unroll
        for (int i = 0; i < SEG / 2; ++i) {
          const ulonglong2 k2 = *reinterpret_cast<const ulonglong2 *>(ks + m * kChunkRow + 4 * i);
          k[2 * i] = k2.x; k[2 * i + 1] = k2.y;
        }
#pragma unroll
        for (int i = 0; i < SEG / 2; ++i) {
          const ulonglong2 q2 = *reinterpret_cast<const ulonglong2 *>(qs + m * kChunkRow + 4 * i);
          q[2 * i] = q2.x; q[2 * i + 1] = q2.y;
        }
        const uint64_t gt2 = pair2(gt, gt);
        uint64_t c = 0;   // two zeros
#pragma unroll
        for (int r = 0; r < SEG; ++r) {
          s[r] = mul2(s[r], gt2);
          c = fma2(s[r], k[r], c);
        }
        float kv = sum2(c), o = po;   // the tree's first level; then this row's kv beside the last row's output
        kv = kv + __shfl_xor_sync(kFull, kv, 1);
        o = o + __shfl_xor_sync(kFull, o, 1);
        kv = kv + __shfl_xor_sync(kFull, kv, 2);
        o = o + __shfl_xor_sync(kFull, o, 2);
        if (quarter == 0 && m0 + m > 0) out[(size_t)(m0 + m - 1) * a.nV * D] = o;
        const float dl = (val - kv) * beta;
        const uint64_t dl2 = pair2(dl, dl);
        c = 0;
#pragma unroll
        for (int r = 0; r < SEG; ++r) {
          s[r] = fma2(k[r], dl2, s[r]);
          c = fma2(s[r], q[r], c);
        }
        po = sum2(c);
        if (a.Snap) {
          float *sn = a.Snap + (size_t)(m0 + m) * a.snap_stride + (size_t)h * D * D + (size_t)quarter * (2 * SEG) * D + col;
#pragma unroll
          for (int r = 0; r < SEG; ++r) {
            const float2 v = unpair2(s[r]);
            sn[(size_t)r * D] = v.x;
            sn[(size_t)(SEG + r) * D] = v.y;
          }
        }
      }
    }
    __syncthreads();   // the next chunk is staged, this one is read
  }
  if (!helper) {
    float o = po + __shfl_xor_sync(kFull, po, 1);
    o = o + __shfl_xor_sync(kFull, o, 2);
    if (quarter == 0 && a.M > 0) out[(size_t)(a.M - 1) * a.nV * D] = o;
#pragma unroll
    for (int r = 0; r < SEG; ++r) {
      const float2 v = unpair2(s[r]);
      Sh[(size_t)r * D] = v.x;
      Sh[(size_t)(SEG + r) * D] = v.y;
    }
  }
}

static uint32_t chunk_dn_smem_fn(const void *) { return 2u * kChunkBuffer * 4u; }

#define F(f) AINFER_ARG(ChunkConvSiluArgs, f)
AINFER_REGISTER(ChunkConvSilu, ChunkConvSiluArgs, 256, 256, 0, nullptr, F(Mx), F(QKV), F(CS), F(CW), F(C), F(M), F(Snap), F(snap_stride));
#undef F
#define F(f) AINFER_ARG(ChunkBetaDecayArgs, f)
AINFER_REGISTER(ChunkBetaDecay, ChunkBetaDecayArgs, 256, 256, 0, nullptr, F(B), F(A), F(ALog), F(DtBias), F(Bt), F(Gt), F(nV), F(count));
#undef F
#define F(f) AINFER_ARG(ChunkDeltaNetArgs, f)
AINFER_REGISTER(ChunkDeltaNet, ChunkDeltaNetArgs, kChunkThreads, 1, 0, chunk_dn_smem_fn, F(Out), F(Mx), F(S), F(Bt), F(Gt), F(nK), F(nV), F(M), F(Snap), F(snap_stride));
#undef F

AINFER_EARLY_LAUNCH(ChunkConvSilu);
AINFER_EARLY_LAUNCH(ChunkBetaDecay);
AINFER_EARLY_LAUNCH(ChunkDeltaNet);

}  // namespace ainfer
