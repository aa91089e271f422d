// Kernels of the expert-parallel mixture-of-experts block for a decode batch: batched router,
// the dispatch plan and permute (pack (token, slot) items per destination rank), the grouping of
// received items by expert for the grouped tensor-core GEMM, the SiLU-multiply + activation
// quantiser between the two expert GEMMs, the un-permute back to the senders' order and the
// slot-ordered combine. The reference decodes one token on one device and has no counterpart
// (its MLP is dense: tools/decode/decode_l0.cpp:666-674); the arithmetic of every piece is the
// single-token kernels' (moe_core.cuh), so a token's result does not depend on the batch it is
// in nor on how many ranks share the experts.
//
// Exchange buffers. A dispatch buffer has one slot per peer rank:
//   [16 B header: item count][cap x 16 B records {expert, token, slot, 0}][cap x item bytes payload]
// where the payload of an item is the token's quantised hidden vector (H int8) and its group
// scales (H/128 fp32, padded to 16 bytes), and cap = owned tokens x top-k is the most one rank can send to another.
// A return buffer has one slot of cap x H fp32 per peer: the un-weighted expert outputs, in the
// order the items were sent. Slots are exchanged whole (fixed size), so the host never needs the
// counts.
#define AINFER_BLOCK_DOT_INLINE 1

#include "direct_dot.cuh"

namespace ainfer {

__host__ __device__ inline int ep_item_bytes(int H) { return H + ((H / 128 * 4 + 15) & ~15); }

// ---- batched router: logits of every owned token, then one block per token selects ----
struct RouterLogitsRowsArgs {
  const uint16_t *Wr;    // [E][H] bf16 router
  const uint16_t *Wsg;   // [H] bf16 shared-expert gate row (null: none)
  const float *Hn;       // [rows][H] normalised activations
  const float *Bias;     // optional [E]: added to the routed experts' logits (load generators); null: none
  float *Logits;         // [rows][E+1]
  int32_t E, H, rows;
  int32_t tokens_per_block;   // a unit takes 16 tokens where this is 16 or more, else 8; blocks walk the units, any number of them
};
// Every sum is RouterTopK's: a lane's chain over its eight values of every 256, then the lane tree. A warp
// sums four router rows against all of the block's tokens, so that a weight is fetched once per block of
// tokens and an activation is read from shared memory once per four rows: 512 multiply-adds per lane and
// chunk for 32 16-byte reads of activations at 16 tokens, which the shared memory serves in the time of the
// multiply-adds. Activations are staged 1024 columns at a time, a lane's two quarters of its eight values
// apart (side by side they meet the same banks). (One router row per warp and four tokens: bound by those
// reads, 74 us for 192 tokens of 513 x 2048; this form 25.) Tokens go in pairs, one packed multiply-add for both, so
// they lie in turns in shared memory: 701 tokens 76 us with scalar instructions, 64 packed.
constexpr int kRlRows = 32, kRlCols = 1024, kRlChunks = kRlCols / 256;
__host__ __device__ inline int rl_tokens(int tokens_per_block) { return tokens_per_block >= 16 ? 16 : 8; }
template <int TT>
__device__ __forceinline__ void router_logits_rows_unit(const RouterLogitsRowsArgs &a, int unit) {
  extern __shared__ __align__(16) float rl_smem[];   // [TT / 2][kRlChunks][4][32 lanes][2 columns][2 tokens]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nrows = a.E + (a.Wsg ? 1 : 0), n = a.H / 256;
  const int nrb = (a.E + 1 + kRlRows - 1) / kRlRows, e0 = (unit % nrb) * kRlRows + warp * 4, t0 = (unit / nrb) * TT;
  const uint4 *w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {   // past the last row: that row again, not stored
    const int e = min(e0 + j, nrows - 1);
    w[j] = reinterpret_cast<const uint4 *>(e < a.E ? a.Wr + (size_t)e * a.H : a.Wsg) + lane;
  }
  uint64_t acc[TT / 2][4];   // two tokens' sums
#pragma unroll
  for (int u = 0; u < TT / 2; ++u)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[u][j] = 0;
  for (int i0 = 0; i0 < n; i0 += kRlChunks) {
    const int nc = min(kRlChunks, n - i0);
    __syncthreads();   // the last columns' readers are done
    for (int i = threadIdx.x; i < TT / 2 * nc * 64; i += 256) {
      const int u = i / (nc * 64), f = i % (nc * 64), c = f >> 6, q = f & 63;   // pair of tokens (past the end: the last one, not stored), chunk, quarter
      const float *h = a.Hn + (size_t)(i0 + c) * 256 + q * 4;
      const float4 v0 = __ldcg(reinterpret_cast<const float4 *>(h + (size_t)min(t0 + 2 * u, a.rows - 1) * a.H)),
                   v1 = __ldcg(reinterpret_cast<const float4 *>(h + (size_t)min(t0 + 2 * u + 1, a.rows - 1) * a.H));
      float4 *d = reinterpret_cast<float4 *>(rl_smem) + ((u * kRlChunks + c) * 4 + 2 * (q & 1)) * 32 + (q >> 1);
      d[0] = make_float4(v0.x, v1.x, v0.y, v1.y);
      d[32] = make_float4(v0.z, v1.z, v0.w, v1.w);
    }
    __syncthreads();
    uint4 wv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) wv[j] = __ldg(w[j] + (size_t)i0 * 32);
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
      uint4 wn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) wn[j] = __ldg(w[j] + (size_t)min(i0 + c + 1, n - 1) * 32);
      const ulonglong2 *x = reinterpret_cast<const ulonglong2 *>(rl_smem) + c * 128 + lane;
#pragma unroll
      for (int p = 0; p < 4; ++p) {   // columns 2 p and 2 p + 1 of the lane's eight
        uint64_t f0[4], f1[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t v = p == 0 ? wv[j].x : p == 1 ? wv[j].y : p == 2 ? wv[j].z : wv[j].w;
          const float lo = u2f(v << 16), hi = u2f(v & 0xFFFF0000u);
          f0[j] = pair2(lo, lo);
          f1[j] = pair2(hi, hi);
        }
#pragma unroll
        for (int u = 0; u < TT / 2; ++u) {
          const ulonglong2 xv = x[(u * kRlChunks * 4 + p) * 32];
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[u][j] = fma2(f0[j], xv.x, acc[u][j]);
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[u][j] = fma2(f1[j], xv.y, acc[u][j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = wn[j];
    }
  }
  const int own = warp_tree_owner<8>(lane);   // of eight sums (two tokens x four rows), the one this lane ends with
#pragma unroll
  for (int u = 0; u < TT; u += 2) {
    const float2 s0 = unpair2(acc[u / 2][0]), s1 = unpair2(acc[u / 2][1]), s2 = unpair2(acc[u / 2][2]), s3 = unpair2(acc[u / 2][3]);
    const float v[8] = {s0.x, s1.x, s2.x, s3.x, s0.y, s1.y, s2.y, s3.y};
    const float sum = warp_tree_sum_multi<8>(v, lane);
    const int t = t0 + u + (own >> 2), e = e0 + (own & 3);
    if ((lane & 3) == 0 && t < a.rows && e < nrows)
      a.Logits[(size_t)t * (a.E + 1) + e] = a.Bias && e < a.E ? sum + __ldg(a.Bias + e) : a.Bias ? sum + 0.0f : sum;
  }
}
__global__ void __launch_bounds__(256, 2) RouterLogitsRows(const RouterLogitsRowsArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int tt = rl_tokens(a.tokens_per_block), units = (a.E + 1 + kRlRows - 1) / kRlRows * ((a.rows + tt - 1) / tt);
#pragma unroll 1
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    if (tt == 16) router_logits_rows_unit<16>(a, u);
    else router_logits_rows_unit<8>(a, u);
  }
}
static uint32_t router_rows_smem(const void *args) { return (uint32_t)rl_tokens(((const RouterLogitsRowsArgs *)args)->tokens_per_block) * kRlCols * 4u; }
struct RouterSelectRowsArgs {
  const float *Logits;   // [rows][E+1]
  int32_t *SelIdx;       // [rows][k+1]
  float *SelW;           // [rows][k+1]
  float *NearGap;        // [rows]
  int32_t E, k, has_shared;
};
__global__ void __launch_bounds__(256) RouterSelectRows(const RouterSelectRowsArgs a) {
  __shared__ float sp[1024 + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  router_select(a.Logits + (size_t)t * (a.E + 1), a.E, a.k, a.has_shared != 0, sp, a.SelIdx + (size_t)t * (a.k + 1),
                a.SelW + (size_t)t * (a.k + 1), a.NearGap + t);
}

// ---- dispatch plan: destination rank and position of every (token, slot) item ----
constexpr int kEpMaxItems = 2048;   // owned tokens x top-k, and items a rank can receive
struct EpItemRec { int32_t expert, token, slot, pad; };
struct EpPlanArgs {
  const int32_t *SelIdx;   // [n][k+1]
  unsigned char *Send;     // dispatch buffer (R slots)
  int32_t *ItemDest;       // [n*k]: dest << 16 | position in the destination's slot
  int32_t n, k, experts_per_rank, world, cap;
  uint32_t slot_bytes;
};
// One block. Item i = token * k + slot goes to the rank that holds its expert; its position there
// is the number of earlier items with the same destination (so slots are filled in item order).
__global__ void __launch_bounds__(1024) EpPlan(const EpPlanArgs a) {
  __shared__ unsigned char dest[kEpMaxItems];
  const int items = a.n * a.k;
  for (int i = threadIdx.x; i < items; i += blockDim.x)
    dest[i] = (unsigned char)(a.SelIdx[(size_t)(i / a.k) * (a.k + 1) + i % a.k] / a.experts_per_rank);
  __syncthreads();
  for (int i = threadIdx.x; i < items; i += blockDim.x) {
    const int d = dest[i];
    int pos = 0;
    for (int j = 0; j < i; ++j) pos += dest[j] == d;
    a.ItemDest[i] = (d << 16) | pos;
    EpItemRec rec{a.SelIdx[(size_t)(i / a.k) * (a.k + 1) + i % a.k], i / a.k, i % a.k, 0};
    *reinterpret_cast<EpItemRec *>(a.Send + (size_t)d * a.slot_bytes + 16 + (size_t)pos * 16) = rec;
  }
  for (int d = threadIdx.x; d < a.world; d += blockDim.x) {
    int c = 0;
    for (int j = 0; j < items; ++j) c += dest[j] == d;
    *reinterpret_cast<int4 *>(a.Send + (size_t)d * a.slot_bytes) = make_int4(c, 0, 0, 0);
  }
}
// ---- permute: one block per item copies the token's quantised vector and scales ----
struct EpPackArgs {
  const int8_t *Q8;        // [n][H]
  const float *SQ;         // [n][H/128]
  const int32_t *ItemDest; // [n*k]
  unsigned char *Send;
  int32_t k, H, cap;
  uint32_t slot_bytes;
};
__global__ void __launch_bounds__(128) EpPack(const EpPackArgs a) {
  const int i = blockIdx.x, t = i / a.k;
  const int dp = a.ItemDest[i], d = dp >> 16, pos = dp & 0xFFFF;
  const int item_bytes = ep_item_bytes(a.H);
  unsigned char *dst = a.Send + (size_t)d * a.slot_bytes + 16 + (size_t)a.cap * 16 + (size_t)pos * item_bytes;
  const uint4 *q = reinterpret_cast<const uint4 *>(a.Q8 + (size_t)t * a.H);
  for (int j = threadIdx.x; j < a.H / 16; j += blockDim.x) reinterpret_cast<uint4 *>(dst)[j] = q[j];
  const float *s = a.SQ + (size_t)t * (a.H / 128);
  for (int j = threadIdx.x; j < a.H / 128; j += blockDim.x) reinterpret_cast<float *>(dst + a.H)[j] = s[j];
}

// ---- grouping of the received items by expert, and the problem lists of the grouped GEMMs ----
struct EpTcGroup {           // = TcGroup of the grouped tensor-core GEMM
  const uint8_t *P;
  const uint16_t *S;
  int32_t x_row0, M, y_col, pad;
};
static_assert(sizeof(EpTcGroup) == 32, "layout of the grouped GEMM's problem record");
// Counts of a grouping: items in total; gate/up and down problems of experts with at most eight rows; the same of experts
// with more; gate/up and down problems in the lists.
constexpr int kEpFewRows = 8;
__device__ __forceinline__ void ep_store_counts(int32_t *c, int items, int few, int all) {
  reinterpret_cast<int4 *>(c)[0] = make_int4(items, 2 * few, few, 2 * (all - few));
  reinterpret_cast<int4 *>(c)[1] = make_int4(all - few, 2 * all, all, 0);
}
// The problems of one expert's rows, at most max_rows each, from index g of the lists on.
__device__ __forceinline__ void ep_problems(EpTcGroup *gate_up, EpTcGroup *down, const ExpertW &w, int row0, int rows, int max_rows, int I, int g) {
  for (int j = 0; j * max_rows < rows; ++j, ++g) {
    const int r0 = row0 + j * max_rows, mr = min(max_rows, rows - j * max_rows);
    gate_up[2 * g] = EpTcGroup{w.gP, w.gS, r0, mr, 0, 0};
    gate_up[2 * g + 1] = EpTcGroup{w.uP, w.uS, r0, mr, I, 0};
    down[g] = EpTcGroup{w.dP, w.dS, r0, mr, 0, 0};
  }
}
struct EpGroupArgs {
  const unsigned char *Recv;  // dispatch buffer received (R slots)
  const ExpertW *Experts;     // the layer's table [E+1]
  int32_t *Sorted;            // [R*cap]: src << 16 | index in the source's slot, grouped by expert
  EpTcGroup *GroupsGateUp;    // gate and up problem of every active expert and cut
  EpTcGroup *GroupsDown;
  int32_t *Counts;            // [8], see ep_store_counts
  int32_t world, rank, experts_per_rank, cap, I;
  uint32_t slot_bytes;
  // The shared expert of this rank's own rows rides in the same launches as one more problem:
  // its activations are rows [shared_row0, shared_row0 + shared_rows) of the grouped layout
  // (the owner's quantiser writes them there). shared_rows == 0: none.
  int32_t shared_row0, shared_rows, shared_expert;
  int32_t max_rows;     // an expert with more rows is cut into problems of at most this many (same weights, consecutive rows)
};
// One block. Items are numbered (source rank, index) in ascending order; an item's row in the
// grouped layout is the start of its expert's range plus the number of earlier items of the same
// expert. Experts with no item produce no problem.
__global__ void __launch_bounds__(1024) EpGroup(const EpGroupArgs a) {
  __shared__ short le[kEpMaxItems];          // local expert of every received item
  __shared__ int base[65];                   // first item number of every source
  __shared__ int hist[1024], start[1024], active[1024];   // active: index of the expert's first problem
  const int tid = threadIdx.x;
  if (tid == 0) {
    int s = 0;
    for (int r = 0; r < a.world; ++r) {
      base[r] = s;
      s += *reinterpret_cast<const int *>(a.Recv + (size_t)r * a.slot_bytes);
    }
    base[a.world] = s;
  }
  for (int e = tid; e < a.experts_per_rank; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  const int total = base[a.world] < kEpMaxItems ? base[a.world] : kEpMaxItems;
  for (int it = tid; it < total; it += blockDim.x) {
    int r = 0;
    while (it >= base[r + 1]) ++r;
    const EpItemRec rec = *reinterpret_cast<const EpItemRec *>(a.Recv + (size_t)r * a.slot_bytes + 16 + (size_t)(it - base[r]) * 16);
    const int l = rec.expert - a.rank * a.experts_per_rank;
    le[it] = (short)l;
    atomicAdd(&hist[l], 1);
  }
  __syncthreads();
  if (tid < 32) {   // exclusive scans over the experts (counts, and "has items" flags): one warp, chunks of 32
    int run = 0, all = 0, few = 0;
    for (int e0 = 0; e0 < a.experts_per_rank; e0 += 32) {
      const int e = e0 + tid;
      const int c = e < a.experts_per_rank ? hist[e] : 0, np = (c + a.max_rows - 1) / a.max_rows;
      int sc = c, sp = np;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int vc = __shfl_up_sync(kFull, sc, off), vp = __shfl_up_sync(kFull, sp, off);
        if (tid >= off) { sc += vc; sp += vp; }
      }
      if (e < a.experts_per_rank) { start[e] = run + sc - c; active[e] = all + sp - np; }
      run += __shfl_sync(kFull, sc, 31);
      all += __shfl_sync(kFull, sp, 31);
      few += __popc(__ballot_sync(kFull, c > 0 && c <= kEpFewRows));
    }
    if (tid == 0) {
      const int sh = (a.shared_rows + a.max_rows - 1) / a.max_rows;
      if (sh > 0) ep_problems(a.GroupsGateUp, a.GroupsDown, a.Experts[a.shared_expert], a.shared_row0, a.shared_rows, a.max_rows, a.I, all);
      ep_store_counts(a.Counts, total, few + (a.shared_rows > 0 && a.shared_rows <= kEpFewRows), all + sh);
    }
  }
  __syncthreads();
  for (int e = tid; e < a.experts_per_rank; e += blockDim.x)
    if (hist[e] > 0) ep_problems(a.GroupsGateUp, a.GroupsDown, a.Experts[a.rank * a.experts_per_rank + e], start[e], hist[e], a.max_rows, a.I, active[e]);
  for (int it = tid; it < total; it += blockDim.x) {
    const int l = le[it];
    int pos = start[l];
    for (int j = 0; j < it; ++j) pos += le[j] == l;
    int r = 0;
    while (it >= base[r + 1]) ++r;
    a.Sorted[pos] = (r << 16) | (it - base[r]);
  }
}
// ---- gather the received payloads into the grouped layout ----
struct EpGatherArgs {
  const unsigned char *Recv;
  const int32_t *Sorted;
  const int32_t *Counts;
  int8_t *XQ;     // [R*cap][H]
  float *SQ;      // [R*cap][H/128]
  int32_t H, cap;
  uint32_t slot_bytes;
};
__global__ void __launch_bounds__(128) EpGather(const EpGatherArgs a) {
  const int pos = blockIdx.x;
  if (pos >= __ldg(a.Counts)) return;
  const int si = a.Sorted[pos], r = si >> 16, i = si & 0xFFFF;
  const int item_bytes = ep_item_bytes(a.H);
  const unsigned char *src = a.Recv + (size_t)r * a.slot_bytes + 16 + (size_t)a.cap * 16 + (size_t)i * item_bytes;
  uint4 *q = reinterpret_cast<uint4 *>(a.XQ + (size_t)pos * a.H);
  for (int j = threadIdx.x; j < a.H / 16; j += blockDim.x) q[j] = reinterpret_cast<const uint4 *>(src)[j];
  float *s = a.SQ + (size_t)pos * (a.H / 128);
  for (int j = threadIdx.x; j < a.H / 128; j += blockDim.x) s[j] = reinterpret_cast<const float *>(src + a.H)[j];
}

// ---- one rank: its own rows need no dispatch buffers ----
// Item i = token * k + slot; its place among the rows grouped by expert goes to ItemRow (the order within
// an expert is free: a row's products do not depend on its place).
constexpr int kEpLocalItems = 8192;
struct EpGroupLocalArgs {
  const int32_t *SelIdx;      // [n][k+1]
  const ExpertW *Experts;     // the layer's table [E+1]
  int32_t *Sorted;            // [n*k]: item, grouped by expert
  int32_t *ItemRow;           // [n*k]: place of an item
  EpTcGroup *GroupsGateUp;    // gate and up problem of every active expert and cut
  EpTcGroup *GroupsDown;
  int32_t *Counts;            // [8], see ep_store_counts
  int32_t n, k, E, I;
  int32_t shared_row0, shared_rows, max_rows;
};
struct EpGroupLocalCutArgs {
  EpGroupLocalArgs g;
  int32_t *Lists;             // [2] lengths of the lists; Counts counts by 64 rows whatever max_rows is
};
// Lists: null: Counts counts by max_rows.
__device__ __forceinline__ void ep_group_local(const EpGroupLocalArgs &a, int32_t *Lists) {
  __shared__ int hist[1024], start[1024], wsum[2][33];
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, items = a.n * a.k;
  hist[tid] = 0;
  pdl_wait();
  __syncthreads();
  constexpr int kPer = kEpLocalItems / 1024;
  int ex[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = tid + q * 1024;
    ex[q] = i < items ? a.SelIdx[(size_t)(i / a.k) * (a.k + 1) + i % a.k] : -1;
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q)
    if (ex[q] >= 0) atomicAdd(&hist[ex[q]], 1);
  __syncthreads();
  const int c = hist[tid], np = (c + a.max_rows - 1) / a.max_rows;   // items and problems of expert tid
  int sc = c, sp = np;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int vc = __shfl_up_sync(kFull, sc, off), vp = __shfl_up_sync(kFull, sp, off);
    if (lane >= off) { sc += vc; sp += vp; }
  }
  if (lane == 31) { wsum[0][warp] = sc; wsum[1][warp] = sp; }
  __syncthreads();
  if (warp < 2) {
    const int own = wsum[warp][lane];
    int v = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(kFull, v, off);
      if (lane >= off) v += o;
    }
    wsum[warp][lane] = v - own;
    if (lane == 31) wsum[warp][32] = v;
  }
  __syncthreads();
  const int first = wsum[0][warp] + sc - c, g0 = wsum[1][warp] + sp - np, total = wsum[1][32];
  start[tid] = first;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; ++q)
    if (ex[q] >= 0) {
      const int i = tid + q * 1024, pos = atomicAdd(&start[ex[q]], 1);
      a.Sorted[pos] = i;
      a.ItemRow[i] = pos;
    }
  if (c > 0) ep_problems(a.GroupsGateUp, a.GroupsDown, a.Experts[tid], first, c, a.max_rows, a.I, g0);
  const int few = __syncthreads_count(c > 0 && c <= kEpFewRows);
  int counted = total, by = a.max_rows;
  if (Lists) {   // the documented counts are by 64 rows, whatever the lists' cut
    by = 64;
    counted = 0;
#pragma unroll 1
    for (int j = 0; j * 64 < a.n; ++j) counted += __syncthreads_count(c > j * 64);   // an expert has an item of a row at most once
    if (tid == 0) {
      const int lists = total + (a.shared_rows + a.max_rows - 1) / a.max_rows;
      Lists[0] = 2 * lists;
      Lists[1] = lists;
    }
  }
  if (tid == 1023) {
    if (a.shared_rows > 0) ep_problems(a.GroupsGateUp, a.GroupsDown, a.Experts[a.E], a.shared_row0, a.shared_rows, a.max_rows, a.I, total);
    ep_store_counts(a.Counts, items, few + (a.shared_rows > 0 && a.shared_rows <= kEpFewRows), counted + (a.shared_rows + by - 1) / by);
  }
}
__global__ void __launch_bounds__(1024) EpGroupLocal(const EpGroupLocalArgs a) { ep_group_local(a, nullptr); }
__global__ void __launch_bounds__(1024) EpGroupLocalCut(const EpGroupLocalCutArgs a) { ep_group_local(a.g, a.Lists); }
struct EpGatherLocalArgs {
  const int8_t *Q8;        // [n][H]
  const float *SQ;         // [n][H/128]
  const int32_t *Sorted;   // [items]
  int8_t *XQ;              // [items][H]
  float *XS;               // [items][H/128]
  int32_t H, k;
};
__global__ void __launch_bounds__(128) EpGatherLocal(const EpGatherLocalArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int pos = blockIdx.x, t = a.Sorted[pos] / a.k;
  const uint4 *q = reinterpret_cast<const uint4 *>(a.Q8 + (size_t)t * a.H);
  uint4 *d = reinterpret_cast<uint4 *>(a.XQ + (size_t)pos * a.H);
  for (int j = threadIdx.x; j < a.H / 16; j += 128) d[j] = q[j];
  const float *s = a.SQ + (size_t)t * (a.H / 128);
  for (int j = threadIdx.x; j < a.H / 128; j += 128) a.XS[(size_t)pos * (a.H / 128) + j] = s[j];
}

// ---- between the expert GEMMs: act = silu(gate) * up, then the per-128 activation quantiser ----
// (SiluMul tools/cmdlist/kernels.cpp:29-37, ScalesMax + Quantize :551-579.) One warp per group of
// 128, a lane holds four consecutive elements.
struct SiluQuantRowsArgs {
  const float *GU;         // [rows][2*I]: gate outputs, then up outputs
  const int32_t *Counts;   // optional device word: rows in use among the first always_from (null: every launched row)
  int8_t *AQ;              // [rows][I]
  float *ASQ;              // [rows][I/128]
  int32_t I;
  int32_t always_from;     // rows from this one on are always in use
  int32_t front;           // blocks below it take their own row, the others the rows from always_from on
};
__global__ void __launch_bounds__(128) SiluQuantRows(const SiluQuantRowsArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = (int)blockIdx.x < a.front ? (int)blockIdx.x : a.always_from + (int)blockIdx.x - a.front;
  // Counts is written by a kernel that this one may have started beside: not through the read-only path
  if (a.Counts && row < a.always_from && row >= __ldcg(a.Counts)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float *g = a.GU + (size_t)row * 2 * a.I, *u = g + a.I;
  for (int grp = warp; grp < a.I / 128; grp += 4) {
    const int j = grp * 128 + lane * 4;
    const float4 gv = *reinterpret_cast<const float4 *>(g + j), uv = *reinterpret_cast<const float4 *>(u + j);
    float4 y;
    y.x = silu_mul(gv.x, uv.x);
    y.y = silu_mul(gv.y, uv.y);
    y.z = silu_mul(gv.z, uv.z);
    y.w = silu_mul(gv.w, uv.w);
    float m = fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w)));
    m = warp_max(m);
    float s = m / 127.0f;
    if (s == 0.0f) s = 1.0f;
    if (lane == 0) a.ASQ[(size_t)row * (a.I / 128) + grp] = s;
    const int q0 = quant_round(y.x, s), q1 = quant_round(y.y, s), q2 = quant_round(y.z, s), q3 = quant_round(y.w, s);
    *reinterpret_cast<uint32_t *>(a.AQ + (size_t)row * a.I + j) =
        (uint32_t)(q0 & 0xFF) | ((uint32_t)(q1 & 0xFF) << 8) | ((uint32_t)(q2 & 0xFF) << 16) | ((uint32_t)(q3 & 0xFF) << 24);
  }
}

// ---- un-permute: expert outputs back into the senders' slots, in the order they were sent ----
struct EpScatterArgs {
  const float *Y;          // [R*cap][H] down-projection outputs in the grouped layout
  const int32_t *Sorted;
  const int32_t *Counts;
  unsigned char *Ret;      // return buffer (R slots of cap x H fp32)
  int32_t H;
  uint32_t slot_bytes;
};
__global__ void __launch_bounds__(128) EpScatter(const EpScatterArgs a) {
  const int pos = blockIdx.x;
  if (pos >= __ldg(a.Counts)) return;
  const int si = a.Sorted[pos], r = si >> 16, i = si & 0xFFFF;
  const float4 *src = reinterpret_cast<const float4 *>(a.Y + (size_t)pos * a.H);
  float4 *dst = reinterpret_cast<float4 *>(a.Ret + (size_t)r * a.slot_bytes + (size_t)i * a.H * 4);
  for (int j = threadIdx.x; j < a.H / 4; j += blockDim.x) dst[j] = src[j];
}

// ---- combine on the token's owner: the additions of ExpertDownCombine, in slot order ----
// X[t][n] = Res[t][n] + (sum over routed slots j in rank order of W[t][j] * Y_j[n], then
// + W[t][k] * Ysh[t][n]); products and sums unfused.
struct EpCombineArgs {
  const float *Res;         // [n][H]
  const unsigned char *Back;// return buffer received (R slots)
  const int32_t *ItemDest;  // [n*k]
  const float *SelW;        // [n][k+1]
  const float *Ysh;         // [n][H] shared expert's output (null: none)
  float *X;                 // [n][H]
  float *X2;                // a second copy (the next layer's input; may be Res)
  int32_t k, H;
  uint32_t slot_bytes;
};
// Launched with tokens x ceil(H / 256) blocks.
// A block: 256 columns of a row. The outputs of a row's items lie apart: their places and weights come first, then every
// thread fetches 16 bytes of up to three items at once into shared memory, where a column's thread adds them in slot
// order. (A thread a column that fetched item by item, place and value: 29 us for 701 rows of ten, 6.3 for 64; so 20 and 3.8.) 16-byte
// pieces need H a multiple of four and the buffer and its slots on 16 bytes; otherwise, and beyond 32 items, item by item.
constexpr int kCombineItems = 12;
__global__ void __launch_bounds__(256) EpCombine(const EpCombineArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) float ys[kCombineItems][256];
  __shared__ float ws[33];
  __shared__ int places[32];
  const int bpr = (a.H + 255) / 256, t = blockIdx.x / bpr, c0 = (blockIdx.x % bpr) * 256, tid = threadIdx.x;
  const int n = c0 + tid;
  const size_t at = (size_t)t * a.H + n;
  float acc = 0.0f, res = 0.0f, ysh = 0.0f, wsh = 0.0f;
  if (n < a.H) {
    res = a.Res[at];
    if (a.Ysh) ysh = a.Ysh[at];
  }
  if (a.Ysh) wsh = a.SelW[(size_t)t * (a.k + 1) + a.k];
  if (a.k <= 32 && (a.H & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.Back) | a.slot_bytes) & 15u) == 0) {
    if (tid < a.k) {
      places[tid] = a.ItemDest[t * a.k + tid];
      ws[tid] = a.SelW[(size_t)t * (a.k + 1) + tid];
    }
    const int part = tid >> 6, col = (tid & 63) * 4;
    __syncthreads();
    for (int j0 = 0; j0 < a.k; j0 += kCombineItems) {
      const int some = min(kCombineItems, a.k - j0);
      float4 v[kCombineItems / 4];
#pragma unroll
      for (int u = 0; u < kCombineItems / 4; ++u) {
        const int j = part + 4 * u;
        v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (j < some && c0 + col < a.H) {
          const int dp = places[j0 + j];
          v[u] = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(a.Back + (size_t)(dp >> 16) * a.slot_bytes) + (size_t)(dp & 0xFFFF) * a.H + c0 + col);
        }
      }
      if (j0) __syncthreads();   // the last items are added
#pragma unroll
      for (int u = 0; u < kCombineItems / 4; ++u) *reinterpret_cast<float4 *>(&ys[part + 4 * u][col]) = v[u];
      __syncthreads();
      for (int j = 0; j < some; ++j) acc = acc + ws[j0 + j] * ys[j][tid];
    }
  } else if (n < a.H) {
    for (int j = 0; j < a.k; ++j) {
      const int dp = a.ItemDest[t * a.k + j];
      const float y = reinterpret_cast<const float *>(a.Back + (size_t)(dp >> 16) * a.slot_bytes)[(size_t)(dp & 0xFFFF) * a.H + n];
      acc = acc + a.SelW[(size_t)t * (a.k + 1) + j] * y;
    }
  }
  if (n >= a.H) return;
  if (a.Ysh) acc = acc + wsh * ysh;
  const float x = res + acc;
  a.X[at] = x;
  a.X2[at] = x;
}

#define F(f) AINFER_ARG(RouterLogitsRowsArgs, f)
AINFER_REGISTER(RouterLogitsRows, RouterLogitsRowsArgs, 256, 0, 0, router_rows_smem, F(Wr), F(Wsg), F(Hn), F(Bias), F(Logits), F(E), F(H), F(rows),
                F(tokens_per_block));
#undef F
#define F(f) AINFER_ARG(RouterSelectRowsArgs, f)
AINFER_REGISTER(RouterSelectRows, RouterSelectRowsArgs, 256, 1, 0, nullptr, F(Logits), F(SelIdx), F(SelW), F(NearGap), F(E), F(k), F(has_shared));
#undef F
#define F(f) AINFER_ARG(EpPlanArgs, f)
AINFER_REGISTER(EpPlan, EpPlanArgs, 1024, 0, 0, nullptr, F(SelIdx), F(Send), F(ItemDest), F(n), F(k), F(experts_per_rank), F(world), F(cap),
                F(slot_bytes));
#undef F
#define F(f) AINFER_ARG(EpPackArgs, f)
AINFER_REGISTER(EpPack, EpPackArgs, 128, 1, 0, nullptr, F(Q8), F(SQ), F(ItemDest), F(Send), F(k), F(H), F(cap), F(slot_bytes));
#undef F
#define F(f) AINFER_ARG(EpGroupArgs, f)
AINFER_REGISTER(EpGroup, EpGroupArgs, 1024, 0, 0, nullptr, F(Recv), F(Experts), F(Sorted), F(GroupsGateUp), F(GroupsDown), F(Counts), F(world),
                F(rank), F(experts_per_rank), F(cap), F(I), F(slot_bytes), F(shared_row0), F(shared_rows), F(shared_expert), F(max_rows));
#undef F
#define F(f) AINFER_ARG(EpGatherArgs, f)
AINFER_REGISTER(EpGather, EpGatherArgs, 128, 1, 0, nullptr, F(Recv), F(Sorted), F(Counts), F(XQ), F(SQ), F(H), F(cap), F(slot_bytes));
#undef F
#define F(f) AINFER_ARG(EpGroupLocalArgs, f)
AINFER_REGISTER(EpGroupLocal, EpGroupLocalArgs, 1024, 0, 0, nullptr, F(SelIdx), F(Experts), F(Sorted), F(ItemRow), F(GroupsGateUp), F(GroupsDown),
                F(Counts), F(n), F(k), F(E), F(I), F(shared_row0), F(shared_rows), F(max_rows));
#undef F
#define F(f) AINFER_ARG(EpGroupLocalCutArgs, f)
AINFER_REGISTER(EpGroupLocalCut, EpGroupLocalCutArgs, 1024, 0, 0, nullptr, F(g.SelIdx), F(g.Experts), F(g.Sorted), F(g.ItemRow), F(g.GroupsGateUp),
                F(g.GroupsDown), F(g.Counts), F(g.n), F(g.k), F(g.E), F(g.I), F(g.shared_row0), F(g.shared_rows), F(g.max_rows), F(Lists));
#undef F
#define F(f) AINFER_ARG(EpGatherLocalArgs, f)
AINFER_REGISTER(EpGatherLocal, EpGatherLocalArgs, 128, 1, 0, nullptr, F(Q8), F(SQ), F(Sorted), F(XQ), F(XS), F(H), F(k));
#undef F
#define F(f) AINFER_ARG(SiluQuantRowsArgs, f)
AINFER_REGISTER(SiluQuantRows, SiluQuantRowsArgs, 128, 1, 0, nullptr, F(GU), F(Counts), F(AQ), F(ASQ), F(I), F(always_from), F(front));
#undef F
#define F(f) AINFER_ARG(EpScatterArgs, f)
AINFER_REGISTER(EpScatter, EpScatterArgs, 128, 1, 0, nullptr, F(Y), F(Sorted), F(Counts), F(Ret), F(H), F(slot_bytes));
#undef F
#define F(f) AINFER_ARG(EpCombineArgs, f)
AINFER_REGISTER(EpCombine, EpCombineArgs, 256, 0, 0, nullptr, F(Res), F(Back), F(ItemDest), F(SelW), F(Ysh), F(X), F(X2), F(k), F(H), F(slot_bytes));
#undef F

AINFER_EARLY_LAUNCH(RouterLogitsRows);
AINFER_EARLY_LAUNCH(RouterSelectRows);
AINFER_EARLY_LAUNCH(EpGroupLocal);
AINFER_EARLY_LAUNCH(EpGroupLocalCut);
AINFER_EARLY_LAUNCH(EpGatherLocal);
AINFER_EARLY_LAUNCH(SiluQuantRows);
AINFER_EARLY_LAUNCH(EpCombine);

}  // namespace ainfer
