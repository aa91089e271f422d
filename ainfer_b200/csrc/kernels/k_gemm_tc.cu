// Int4GemmA8Tc / Int4GemmA8TcGrouped: W4A8 group-128 GEMM for batches of activation rows on the
// tensor cores. This is the batched form of the reference's Int4Gemv (tools/cmdlist/kernels.cpp:148-193;
// sweep protocol tools/gemv/gemv.cpp:503-601): per output row and batch entry, the exact int32 sum of
// the 128 nibble x int8 products of a group, then acc = acc + ((float)sum * weight_scale) *
// activation_scale[g] in ascending group order. The integer sums are exact on any hardware and the
// fp32 order is the reference's, so every batch entry is bit-identical to the one-row GEMV.
//
// The grouped form runs a list of problems of the same shape (N, K) in one launch: problem i has
// its own weight matrix and its own range of activation rows (an expert and the tokens routed to
// it). The list and its length live in device memory, so routing never goes through the host.
//
// A block of eight warps walks units of 128 weight rows x up to NT batch entries; a warp owns 16 rows.
// A stage is two groups of 128 weights: 128 bytes of every row (a whole line), the entries' activations
// and both scales, copied by cp.async three to five stages deep, two blocks per SM, one block barrier a
// stage. A lane of mma.sync.m16n8k32 (s8) takes sixteen packed bytes of a row: 32 consecutive weights,
// widened in registers (a nibble at the top of its byte is the signed byte 16 v: no sign fix-up) and
// put back into order, are its share of four products; the same 32 activations of an entry are the
// other operand. The accumulators start at the bits of 1.5 x 2^23, so that a sum IS a float a
// subtraction away (exact: 16 times a sum is below 2^22).
//
// Why not tcgen05 here: the fp32 rescale of every group takes the sums out of the accumulators every four
// products, and the weights must be widened first. Both are register work: from registers to shared
// memory, tensor memory and back costs more than the products. A form with tcgen05.mma kind::i8 and
// warps for copying, widening, issuing and rescaling took 0.7 us a group of a 128 x 16 unit and 2.1 us
// of 128 x 96 (each hand-over is a fence and a barrier's latency); at 2048 multiply-adds a cycle and SM
// mma.sync needs 0.07 us per 16 entries, and the weight stream 0.1 us.
// Bound by the weight stream up to about 24 entries a unit, above by mma.sync.
// Measured, us (before: tcgen05 with two block barriers a group, 64 entries a launch; the experts' lists up to
// 8 rows by the dp4a form):
//   8192 x 2048, 64 / 704 entries      33.8 -> 10.4, 365 -> 68      4096 x 2048, 64   33.2 -> 9.9
//   2048 x 4096, 64                    61.8 -> 13.3                 151936 x 2048, 64  286 -> 98
//   experts of 512, gate and up, 1.25 / 3.75 / 13.7 rows on average   136 -> 107, 277 -> 148, 793 -> 174
//   the same, down                                                     85 -> 72, 173 -> 101, 430 -> 113
// Rescaling two entries in one packed instruction, and the first product of a group starting from the constant itself: experts of
// a 701-row pass 145 -> 138 us a launch on average. Several matrices over the same rows in one launch (Int4GemmA8TcMany: a hybrid
// layer's 8192 + 4096 + 32 + 32 outputs of 2048, where a matrix of 32 rows alone is 8..11 us): 701 rows 140 -> 99 us,
// 64 rows 36 -> 18. Three blocks per SM of three stages each for lists of few rows: 73 us a launch against 69.
#include "block_dot.cuh"

namespace ainfer {

struct Int4GemmA8TcArgs {
  const uint8_t *P;    // packed nibbles [N][K/2]
  const uint16_t *S;   // bf16 scales [N][K/128]
  const int8_t *XQ;    // [M][K] activations
  const float *SQ;     // [M][K/128] activation group scales
  float *Y;            // [M][ldy]
  int32_t N, K, M, ldy;
  int32_t ahead;       // LaunchAhead
};
// One to four matrices of the same K over the same rows; an output's row stride is its matrix's N.
struct Int4GemmA8TcManyArgs {
  const int8_t *XQ;
  const float *SQ;
  int32_t K, M, count;
  const uint8_t *P0; const uint16_t *S0; float *Y0; int32_t N0;
  const uint8_t *P1; const uint16_t *S1; float *Y1; int32_t N1;
  const uint8_t *P2; const uint16_t *S2; float *Y2; int32_t N2;
  const uint8_t *P3; const uint16_t *S3; float *Y3; int32_t N3;
  int32_t ahead;       // LaunchAhead
};

// One problem of a grouped launch: Y[x_row0 + m][y_col + n] = sum_k W[n][k] * X[x_row0 + m][k].
struct TcGroup {
  const uint8_t *P;    // packed nibbles [N][K/2]
  const uint16_t *S;   // bf16 scales [N][K/128]
  int32_t x_row0;      // first activation / output row
  int32_t M;           // rows (1..max_m)
  int32_t y_col;       // first output column
  int32_t pad;
};
static_assert(sizeof(TcGroup) == 32, "two 16-byte loads");
struct Int4GemmA8TcGroupedArgs {
  const TcGroup *Groups;       // [*NGroups] problems
  const int32_t *NGroups;      // device word: number of problems (0 allowed)
  const int8_t *XQ;            // [rows][K]
  const float *SQ;             // [rows][K/128]
  float *Y;                    // [rows][ldy]
  int32_t N, K, max_m, ldy;    // max_m: upper bound of every problem's M, at most 64
};

constexpr int kTcRows = 128;               // weight rows per unit
constexpr int kTcThreads = 256;
constexpr int kTcSms = 148;
constexpr uint32_t kTcWBytes = kTcRows * 128;   // a stage's packed weights: two groups
constexpr uint32_t kTcXPitch = 272;             // bytes between entries of a stage: 256 + 16, so that reads down the entries meet all banks

__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The first product of a chain: d = a b + start in all four.
__device__ __forceinline__ void mma_s8_from(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int start) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(start));
}
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst_smem), "l"(src) : "memory");
}

extern __shared__ __align__(128) unsigned char tc_smem[];

// Stages that two blocks per SM have room for. A stage: weights | activations | activation scales [2][NT] | weight scales [128][2].
__host__ __device__ constexpr int tc_stages(int nt) { return nt == 16 ? 5 : nt == 32 ? 4 : 3; }
__host__ __device__ constexpr uint32_t tc_stage_bytes(int nt) { return kTcWBytes + (uint32_t)nt * kTcXPitch + (uint32_t)nt * 8u + kTcRows * 4u; }
// Entries per unit of one problem: what finishes first over whole rounds of units on the SMs. A stage costs
// the products of its entries, and the widening and copying whatever their number.
__host__ __device__ inline int tc_entries(int tiles, int M) {
  int best = 16;
  long cost = -1;
  for (int nt = 16; nt <= 64; nt *= 2) {
    const long rounds = ((long)tiles * ((M + nt - 1) / nt) + 2 * kTcSms - 1) / (2 * kTcSms), c = rounds * (nt + 12);
    if (cost < 0 || c < cost) { cost = c; best = nt; }
    if (nt >= M) break;
  }
  return best;
}
__host__ __device__ inline int tc_entries_grouped(int max_m) { return max_m <= 16 ? 16 : max_m <= 32 ? 32 : 64; }

struct TcMat {
  const uint8_t *P;
  const uint16_t *S;
  float *Y;
  int32_t N, ldy;
};
struct TcShape {
  const TcGroup *groups;   // null: the matrices `mats` over rows 0..M
  const int32_t *ngroups;
  TcMat mats[4];
  int32_t ends[4];         // row tiles of mats[0..i]
  int32_t M;
  const int8_t *XQ;
  const float *SQ;
  float *Y;
  int32_t N, K, ldy;       // of the groups
  bool ahead;              // the matrices' weights may travel before the dependency wait
};
struct TcUnit {
  const uint8_t *P;        // of the problem's row 0
  const uint16_t *S;
  float *Y;                // of its first column and entry 0
  int32_t x0, M, row0, N, ldy, pad;
};

// One block of eight entries: the four products of a group, then rescale and add.
__device__ __forceinline__ void tc_products(int (&d)[4], const uint32_t (&a)[4][4], const uint4 &x0, const uint4 &x1) {
  mma_s8_from(d, a[0], x0.x, x0.y, 0x4B400000);   // 1.5 x 2^23 as a float
  mma_s8(d, a[1], x0.z, x0.w);
  mma_s8(d, a[2], x1.x, x1.y);
  mma_s8(d, a[3], x1.z, x1.w);
}
// Both entries of a row in one packed instruction each, but for the last addition: a packed product and a packed sum
// are fused by the assembler (found by the bits of a row), which rounds once where the sum's order asks for two.
__device__ __forceinline__ void tc_finish(float (&acc)[4], const int (&d)[4], const uint64_t (&r)[2], float2 q) {
  const uint64_t bias = pair2(-12582912.0f, -12582912.0f), q2 = pair2(q.x, q.y);
  const float2 t0 = unpair2(mul2(mul2(add2(pair2(__int_as_float(d[0]), __int_as_float(d[1])), bias), r[0]), q2)),
               t1 = unpair2(mul2(mul2(add2(pair2(__int_as_float(d[2]), __int_as_float(d[3])), bias), r[1]), q2));
  acc[0] = acc[0] + t0.x;
  acc[1] = acc[1] + t0.y;
  acc[2] = acc[2] + t1.x;
  acc[3] = acc[3] + t1.y;
}

template <int NT>
__device__ __forceinline__ void tc_body(const TcShape &c) {
  constexpr int ST = tc_stages(NT);
  constexpr uint32_t SB = tc_stage_bytes(NT), XO = kTcWBytes, QO = XO + NT * kTcXPitch, CO = QO + NT * 8;
  __shared__ TcUnit ring[8];   // units between the copies and the products (at most ST - 1 apart)
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int K = c.K, G = K >> 7;
  const size_t row_bytes = (size_t)(K >> 1);
  const int tpg = (c.N + kTcRows - 1) / kTcRows;      // row tiles per problem
  const int nrb = (c.M + NT - 1) / NT;                // blocks of entries of the matrices
  const int stride = (int)gridDim.x;
  const uint32_t base = smem_addr(tc_smem);
  if (!c.ahead) pdl_wait();
  const int units = c.groups ? __ldcg(c.ngroups) * tpg : c.ends[3] * nrb;
  // ---- copies: this thread's sources of the next stage; rows and entries that do not exist keep what is there (never stored) ----
  const bool pair_scales = (G & 1) == 0;
  const int wr = warp * 16 + (lane >> 3), wpc = lane & 7;   // weights: eight neighbours copy a row's line, four rows apart
  const int xm = tid >> 4, xpc = tid & 15;                  // activations: sixteen neighbours copy an entry's 256 bytes
  const uint32_t wdst = (uint32_t)wr * 128u + (uint32_t)((wpc ^ ((wr & 1) << 2)) << 4);   // odd rows' halves change places (bank-conflict free reads)
  const uint32_t xdst = XO + (uint32_t)xm * kTcXPitch + (uint32_t)xpc * 16u;
  const uint8_t *wp = nullptr;
  const int8_t *xp = nullptr;
  const char *sp_src = nullptr;                             // of a scale (activation: threads below 2 NT, weight pairs: from 128 on)
  uint32_t wmask = 0, xmask = 0, smask = 0, sdst = 0;
  int lu = blockIdx.x, lg = 0, ls = 0, lk = 0;              // unit, first group, buffer, units begun
  uint4 rec[2];
  auto load_rec = [&](int u) {
    if (c.groups && u < units) {
      const uint4 *p = reinterpret_cast<const uint4 *>(c.groups + u / tpg);
      rec[0] = __ldcg(p); rec[1] = __ldcg(p + 1);
    }
  };
  auto begin_unit = [&]() {   // lu < units; its record is in rec
    TcUnit n;
    if (c.groups) {
      union { uint4 q[2]; TcGroup g; } r;
      r.q[0] = rec[0]; r.q[1] = rec[1];
      n.P = r.g.P; n.S = r.g.S; n.x0 = r.g.x_row0; n.M = min(r.g.M, NT); n.row0 = (lu % tpg) * kTcRows;
      n.Y = c.Y + r.g.y_col; n.N = c.N; n.ldy = c.ldy;
    } else {
      const int rb = lu % nrb, tile = lu / nrb, i = (tile >= c.ends[0]) + (tile >= c.ends[1]) + (tile >= c.ends[2]);
      const TcMat m = i == 0 ? c.mats[0] : i == 1 ? c.mats[1] : i == 2 ? c.mats[2] : c.mats[3];
      const int before = i == 0 ? 0 : i == 1 ? c.ends[0] : i == 2 ? c.ends[1] : c.ends[2];
      n.P = m.P; n.S = m.S; n.x0 = rb * NT; n.M = min(NT, c.M - n.x0); n.row0 = (tile - before) * kTcRows;
      n.Y = m.Y; n.N = m.N; n.ldy = m.ldy;
    }
    if (tid == 0) ring[lk & 7] = n;
    ++lk;
    const int rows = n.N - n.row0;
    wp = n.P + (size_t)(n.row0 + wr) * row_bytes + wpc * 16;
    xp = c.XQ + (size_t)(n.x0 + xm) * K + xpc * 16;
    wmask = xmask = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) wmask |= (wr + 4 * i < rows ? 1u : 0u) << i;
#pragma unroll
    for (int i = 0; i < NT / 16; ++i) xmask |= (xm + 16 * i < n.M ? 1u : 0u) << i;
    smask = 0;
    if (tid < 2 * NT) {
      const int m = tid >> 1, k = tid & 1;
      sp_src = reinterpret_cast<const char *>(c.SQ + (size_t)(n.x0 + m) * G + k);
      sdst = QO + (uint32_t)(k * NT + m) * 4u;
      smask = m < n.M ? 1u + (uint32_t)k : 0u;
    } else if (tid >= 128 && pair_scales) {
      const int r = tid - 128;
      sp_src = reinterpret_cast<const char *>(n.S + (size_t)(n.row0 + r) * G);
      sdst = CO + (uint32_t)r * 4u;
      smask = r < rows ? 1u : 0u;
    }
    load_rec(lu + stride);
  };
  auto copy_w = [&]() {
    if (wpc < 4 * (G - lg)) {
      const uint32_t dst = base + (uint32_t)ls * SB + wdst;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (wmask >> i & 1u) cp_async16(dst + (uint32_t)i * 512u, wp + (size_t)(4 * i) * row_bytes);
    }
  };
  auto copy_x = [&]() {
    const uint32_t dst = base + (uint32_t)ls * SB;
    if (xpc < 8 * (G - lg)) {
#pragma unroll
      for (int i = 0; i < NT / 16; ++i)
        if (xmask >> i & 1u) cp_async16(dst + xdst + (uint32_t)(16 * i) * kTcXPitch, xp + (size_t)(16 * i) * K);
    }
    if (smask && (int)smask <= G - lg) cp_async4(dst + sdst, sp_src);
  };
  auto advance = [&]() {
    wp += 128;
    xp += 256;
    sp_src += tid < 2 * NT ? 8 : 4;
    ls = ls == ST - 1 ? 0 : ls + 1;
    if ((lg += 2) >= G) {
      lg = 0;
      lu += stride;
      if (lu < units) begin_unit();
    }
  };
  auto commit = []() { asm volatile("cp.async.commit_group;" ::: "memory"); };
  load_rec(lu);
  if (lu < units) begin_unit();
  if (c.groups) {
#pragma unroll 1
    for (int i = 0; i < ST - 1; ++i) {
      if (lu < units) { copy_w(); copy_x(); advance(); }
      commit();
    }
  } else {   // the one problem's weights travel before the predecessor is done, where none writes weights
#pragma unroll 1
    for (int i = 0; i < ST - 1 && lu < units; ++i) { copy_w(); advance(); }
    pdl_wait();
    lu = blockIdx.x; lg = 0; ls = 0; lk = 0;
    if (lu < units) begin_unit();
#pragma unroll 1
    for (int i = 0; i < ST - 1; ++i) {
      if (lu < units) { copy_x(); advance(); }
      commit();
    }
  }
  // ---- products ----
  float acc[NT / 8][4];
#pragma unroll
  for (int j = 0; j < NT / 8; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[j][q] = 0.0f;
  const int r0 = warp * 16 + g;
  int cs = 0, ck = 0;
#pragma unroll 1
  for (int u = blockIdx.x; u < units; u += stride, ++ck) {
    int nb = 0;
#pragma unroll 1
    for (int g0 = 0; g0 < G; g0 += 2) {
      asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
      __syncthreads();   // every thread's copies of this stage have landed; the last stage's readers are done
      if (lu < units) { copy_w(); copy_x(); advance(); }
      commit();
      const TcUnit &n = ring[ck & 7];
      if (g0 == 0) nb = (n.M + 7) >> 3;
      const uint32_t sb = base + (uint32_t)cs * SB;
      const unsigned char *sp = tc_smem + (uint32_t)cs * SB;
      uint32_t s0, s1;   // scales of rows r0 and r0 + 8 (two groups each)
      const int ng = min(2, G - g0);
      if (pair_scales) {
        s0 = *reinterpret_cast<const uint32_t *>(sp + CO + r0 * 4);
        s1 = *reinterpret_cast<const uint32_t *>(sp + CO + (r0 + 8) * 4);
      } else {
        const uint16_t *w0 = n.S + (size_t)min(n.row0 + r0, n.N - 1) * G + g0, *w1 = n.S + (size_t)min(n.row0 + r0 + 8, n.N - 1) * G + g0;
        s0 = __ldg(w0) | (uint32_t)__ldg(w0 + ng - 1) << 16;
        s1 = __ldg(w1) | (uint32_t)__ldg(w1 + ng - 1) << 16;
      }
#pragma unroll
      for (int gl = 0; gl < 2; ++gl) {
        if (gl >= ng) break;
        uint32_t a[4][4];   // of product s: row r0, row r0 + 8, then their next four weights
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 p = lds128(sb + (uint32_t)(r0 + 8 * h) * 128u + (uint32_t)(((gl * 4 + t) ^ ((g & 1) << 2)) << 4));
          const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
          for (int s = 0; s < 4; ++s) {   // low and high nibbles alternate
            const uint32_t lo = (w[s] << 4) & 0xF0F0F0F0u, hi = w[s] & 0xF0F0F0F0u;
            a[s][h] = __byte_perm(lo, hi, 0x5140);
            a[s][2 + h] = __byte_perm(lo, hi, 0x7362);
          }
        }
        // a sixteenth of the weight scales of the lane's rows
        const float f0 = __uint_as_float(gl ? s0 & 0xFFFF0000u : s0 << 16) * 0.0625f, f1 = __uint_as_float(gl ? s1 & 0xFFFF0000u : s1 << 16) * 0.0625f;
        const uint64_t sc[2] = {pair2(f0, f0), pair2(f1, f1)};
        const uint32_t xb = sb + XO + (uint32_t)g * kTcXPitch + (uint32_t)(gl * 128 + t * 32);
        const float *sq = reinterpret_cast<const float *>(sp + QO) + gl * NT + 2 * t;
#pragma unroll
        for (int j = 0; j < NT / 8; j += 2) {
          if (j + 1 < nb) {   // two blocks side by side: their products are chains of four
            const uint32_t xj = xb + (uint32_t)j * 8u * kTcXPitch;
            const uint4 x0 = lds128(xj), x1 = lds128(xj + 16u), x2 = lds128(xj + 8u * kTcXPitch), x3 = lds128(xj + 8u * kTcXPitch + 16u);
            const float2 q0 = *reinterpret_cast<const float2 *>(sq + 8 * j), q1 = *reinterpret_cast<const float2 *>(sq + 8 * j + 8);
            int d0[4], d1[4];
            tc_products(d0, a, x0, x1);
            tc_products(d1, a, x2, x3);
            tc_finish(acc[j], d0, sc, q0);
            tc_finish(acc[j + 1], d1, sc, q1);
          } else if (j < nb) {
            const uint32_t xj = xb + (uint32_t)j * 8u * kTcXPitch;
            const uint4 x0 = lds128(xj), x1 = lds128(xj + 16u);
            const float2 q0 = *reinterpret_cast<const float2 *>(sq + 8 * j);
            int d0[4];
            tc_products(d0, a, x0, x1);
            tc_finish(acc[j], d0, sc, q0);
          }
        }
      }
      cs = cs == ST - 1 ? 0 : cs + 1;
    }
    const TcUnit &n = ring[ck & 7];
    float *y = n.Y + (size_t)n.x0 * n.ldy + n.row0 + r0;
    const bool in0 = n.row0 + r0 < n.N, in1 = n.row0 + r0 + 8 < n.N;
    const int M = n.M, ldy = n.ldy;
#pragma unroll
    for (int j = 0; j < NT / 8; ++j) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int m = 8 * j + 2 * t + (q & 1);
        if (m < M && (q < 2 ? in0 : in1)) y[(size_t)m * ldy + (q < 2 ? 0 : 8)] = acc[j][q];
        acc[j][q] = 0.0f;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void tc_dispatch(const TcShape &c, int nt) {
  if (nt == 16) tc_body<16>(c);
  else if (nt == 32) tc_body<32>(c);
  else tc_body<64>(c);
}
__host__ __device__ inline int tc_tiles(int N) { return (N + kTcRows - 1) / kTcRows; }
__host__ __device__ inline int tc_tiles(const Int4GemmA8TcManyArgs &a) {
  return tc_tiles(a.N0) + (a.count > 1 ? tc_tiles(a.N1) : 0) + (a.count > 2 ? tc_tiles(a.N2) : 0) + (a.count > 3 ? tc_tiles(a.N3) : 0);
}
__global__ void __launch_bounds__(kTcThreads, 2) Int4GemmA8TcMany(const Int4GemmA8TcManyArgs a) {
  TcShape c;
  c.groups = nullptr;
  c.ngroups = nullptr;
  c.mats[0] = TcMat{a.P0, a.S0, a.Y0, a.N0, a.N0};
  c.mats[1] = TcMat{a.P1, a.S1, a.Y1, a.N1, a.N1};
  c.mats[2] = TcMat{a.P2, a.S2, a.Y2, a.N2, a.N2};
  c.mats[3] = TcMat{a.P3, a.S3, a.Y3, a.N3, a.N3};
  c.ends[0] = tc_tiles(a.N0);
  c.ends[1] = c.ends[0] + (a.count > 1 ? tc_tiles(a.N1) : 0);
  c.ends[2] = c.ends[1] + (a.count > 2 ? tc_tiles(a.N2) : 0);
  c.ends[3] = c.ends[2] + (a.count > 3 ? tc_tiles(a.N3) : 0);
  c.M = a.M;
  c.XQ = a.XQ; c.SQ = a.SQ; c.Y = nullptr;
  c.N = 0; c.K = a.K; c.ldy = 0;
  c.ahead = (a.ahead & AHEAD_WEIGHTS) != 0;
  tc_dispatch(c, tc_entries(c.ends[3], a.M));
}
__global__ void __launch_bounds__(kTcThreads, 2) Int4GemmA8Tc(const Int4GemmA8TcArgs a) {
  TcShape c;
  c.groups = nullptr;
  c.ngroups = nullptr;
  c.mats[0] = c.mats[1] = c.mats[2] = c.mats[3] = TcMat{a.P, a.S, a.Y, a.N, a.ldy};
  c.ends[0] = c.ends[1] = c.ends[2] = c.ends[3] = tc_tiles(a.N);
  c.M = a.M;
  c.XQ = a.XQ; c.SQ = a.SQ; c.Y = nullptr;
  c.N = 0; c.K = a.K; c.ldy = 0;
  c.ahead = (a.ahead & AHEAD_WEIGHTS) != 0;
  tc_dispatch(c, tc_entries(c.ends[3], a.M));
}

__device__ __forceinline__ TcShape tc_groups(const Int4GemmA8TcGroupedArgs &a) {
  TcShape c;
  c.groups = a.Groups;
  c.ngroups = a.NGroups;
  c.ends[3] = c.M = 0;
  c.XQ = a.XQ; c.SQ = a.SQ; c.Y = a.Y;
  c.N = a.N; c.K = a.K; c.ldy = a.ldy;
  c.ahead = false;
  return c;
}
__global__ void __launch_bounds__(kTcThreads, 2) Int4GemmA8TcGrouped(const Int4GemmA8TcGroupedArgs a) {
  tc_dispatch(tc_groups(a), tc_entries_grouped(a.max_m));
}
static uint32_t tc_smem_bytes(int nt) { return (uint32_t)tc_stages(nt) * tc_stage_bytes(nt); }
static uint32_t tc_smem_fn(const void *args) {
  const Int4GemmA8TcArgs *a = (const Int4GemmA8TcArgs *)args;
  return tc_smem_bytes(tc_entries(tc_tiles(a->N), a->M));
}
static uint32_t tc_many_smem_fn(const void *args) {
  const Int4GemmA8TcManyArgs *a = (const Int4GemmA8TcManyArgs *)args;
  return tc_smem_bytes(tc_entries(tc_tiles(*a), a->M));
}
static uint32_t tc_grouped_smem_fn(const void *args) { return tc_smem_bytes(tc_entries_grouped(((const Int4GemmA8TcGroupedArgs *)args)->max_m)); }

#define F(f) AINFER_ARG(Int4GemmA8TcArgs, f)
AINFER_REGISTER(Int4GemmA8Tc, Int4GemmA8TcArgs, kTcThreads, 0, 0, tc_smem_fn, F(P), F(S), F(XQ), F(SQ), F(Y), F(N), F(K), F(M), F(ldy));
#undef F
#define F(f) AINFER_ARG(Int4GemmA8TcManyArgs, f)
AINFER_REGISTER(Int4GemmA8TcMany, Int4GemmA8TcManyArgs, kTcThreads, 0, 0, tc_many_smem_fn, F(XQ), F(SQ), F(K), F(M), F(count), F(P0), F(S0), F(Y0),
                F(N0), F(P1), F(S1), F(Y1), F(N1), F(P2), F(S2), F(Y2), F(N2), F(P3), F(S3), F(Y3), F(N3));
#undef F
#define F(f) AINFER_ARG(Int4GemmA8TcGroupedArgs, f)
AINFER_REGISTER(Int4GemmA8TcGrouped, Int4GemmA8TcGroupedArgs, kTcThreads, 0, 0, tc_grouped_smem_fn, F(Groups), F(NGroups), F(XQ), F(SQ),
                F(Y), F(N), F(K), F(max_m), F(ldy));
#undef F

AINFER_EARLY_LAUNCH_AHEAD(Int4GemmA8Tc, Int4GemmA8TcArgs);
AINFER_EARLY_LAUNCH_AHEAD(Int4GemmA8TcMany, Int4GemmA8TcManyArgs);
AINFER_EARLY_LAUNCH(Int4GemmA8TcGrouped);

}  // namespace ainfer
