// DecodeStep: one whole decode token in ONE persistent cooperative launch, one block per SM.
//
// The recorded list replays hundreds of small dependent launches per token and is bound by
// their latency, not by HBM. Here the blocks stay resident for the whole token and the work
// is split between two kinds of warps:
//   * one PRODUCER warp per block streams every weight byte the block will need, in the order
//     it will need it, from HBM into a ring of 16 KB shared-memory tiles with bulk
//     asynchronous copies (cp.async.bulk, completion on an mbarrier). It runs ahead of the
//     consumers across stage and layer boundaries, limited only by ring space, and stops only
//     where the addresses depend on data (the routed experts), until the consumers have
//     selected them;
//   * sixteen CONSUMER warps run the stages of a layer, separated by grid-wide hand-overs:
//     each stage takes its activations from global memory (L2), its weights from the ring,
//     and writes its outputs back to global memory for the next stage (words, see below).
// So HBM traffic is decoupled from the dependency chain: while the consumers wait for one
// another, the next stages' weights are already landing in shared memory.
//
// Stages of a Gated DeltaNet layer (tools/decode/decode_l0.cpp:610-674 in the reference):
//   1 norm + quantiser, in_proj qkv/z/b/a GEMV with conv / sigmoid / decay epilogues
//   2 gated delta rule step (state read once and written once)
//   3 gated per-head norm + quantiser, out_proj GEMV + residual
//   4 post norm + quantiser, router logits
//   5 softmax top-k (every block selects for itself), expert gate/up GEMV + SiLU-mul
//   6 quantiser, expert down GEMV, rank-ordered combine + residual
// Stages of a gated attention layer (decode_l0.cpp:560-608): 1 q/k/v GEMV, 2 head norm + RoPE
// + INT8 KV append + one 64-token chunk of attention per block, 3 ordered merge of the chunk
// partials + sigmoid gate + quantiser, 4 o_proj + residual, then 4-6 of the above.
// The tail is final norm, LM head, first-max-wins argmax and the control-block update.
//
// The arithmetic of every stage (operation order, reduction shapes) is that of the stand-alone
// kernels in this directory, so the two paths give bit-identical results.
//
// Every wait (mbarrier, arrivals, words) is bounded by a wall-clock limit: when one runs out the
// block sets the plan's sticky error word, no wait in the grid spins again, and the kernel
// terminates with garbage results that the host refuses (the error word is read after the step).
//
// What bounds it: not HBM (0.33 ms a token of the full preset) but the chain of six stages a layer, each a
// hand-over between all blocks (await, gather: about 1500 cycles), a prologue that every block repeats and rows of
// short loops. Per token, full preset, context 4096: 2.73 ms; 2.08 with shares of rows dealt once a
// launch, epilogue operands as asynchronous copies, one thread a (row, group), group scales by one
// reduction instruction, selection by ranks, silu(z) from the projection's epilogue; 1.96 with words instead of
// barriers and fences, rolled code (instruction-cache misses 0.85 -> 0.32 M a launch of the small preset) and
// attention with queries in registers. What was slower: the state of the delta rule in registers (unrolled: 2.03),
// one loop over the stages with the products inlined (2.11: its registers spill), more groups quantised side by side.
#include "../common/step_plan.h"
#include "attention_core.cuh"
#include "block_stages.cuh"
#include "deltanet_core.cuh"
#include "gemv_stage.cuh"
#include "moe_core.cuh"
#include "tail_core.cuh"

namespace ainfer {

struct DecodeStepArgs {
  const StepPlan *plan;  // device copy of the plan (the kernel keeps its own copy in shared memory)
  int32_t mode;  // 1: final norm + lm_head + argmax, control advances to the selected token
                 // 0: prompt step, control advances to ids[position + 1]
};

constexpr int kCons = 512;          // consumer threads (16 warps)
constexpr int kStepThreads = 544;   // consumers + the producer warp
constexpr int kNT = 10;             // ring tiles
constexpr int kTileStride = kTileBytes + kTileScaleBytes;
// Limit of any single wait, in SM clock cycles (about two seconds). The waits are timed with the
// SM's own cycle counter: reading the global nanosecond timer takes about a microsecond, far too
// long for a poll loop that usually succeeds within a few hundred nanoseconds.
constexpr long long kWaitCycles = 4000000000ll;

// ---- shared-memory map (all dynamic) ----
constexpr int kHdrBytes = 5120;                 // StepShared
constexpr int kActBytes = 8704;                 // staged INT8 activations (<= 8192) + group scales (<= 512)
constexpr int kFbufFloats = 8192;               // fp32 scratch: norm input, O|Z, Act, KV chunk
constexpr int kActOff = kHdrBytes;
constexpr int kFbufOff = kActOff + kActBytes;
constexpr int kTOff = kFbufOff + kFbufFloats * 4;
constexpr int kRingOff = (kTOff + kTFloats * 4 + 127) / 128 * 128;
constexpr int kStepSmemBytes = kRingOff + kNT * kTileStride;
static_assert(kStepSmemBytes <= 232448, "shared memory of one SM");

// Contiguous rows of one matrix, as the producer streams them.
struct Seg {
  const uint8_t *P;   // first row's bytes
  const uint8_t *S;   // first row's scales (null: none)
  int32_t nrows, vec, trow, pad;
};
constexpr int kMaxSegs2 = 24;

// Stages whose rows are dealt to the blocks; kRngIn and kRngOut are followed by the layer type.
enum { kRngIn = 0, kRngOut = 2, kRngRouter = 4, kRngGateUp = 5, kRngDown = 6, kRngHead = 7, kRngCount = 8 };

struct StepShared {
  // the members that are copied 16 bytes at a time come first (the struct sits at a
  // 128-byte aligned address and the sizes are multiples of 16)
  StepPlan plan;                // the plan: read from here, not from global memory, by every stage
  StepLayer ly;                 // the current layer's record
  ExpertW sew[12];              // weight pointers of the selected expert slots
  unsigned long long full[kNT], empty[kNT];
  unsigned long long sel_bar;   // consumers -> producer: this layer's routing is in sew[]
  int32_t sel_idx[12];
  float sel_w[12];
  float gap;
  float wmax[16];
  float av[16];
  int32_t ai[16];
  unsigned kmax[16];            // selection: each warp's largest key
  int32_t ncand;                // selection: candidates so far
  int2 rng[kRngCount];          // this block's rows of every stage (deal())
  volatile int32_t fail;
  int32_t nstamp[2];            // stage clock: records written so far (consumer, producer)
  Seg segs[kMaxSegs2];          // the producer warp's current segment list
  float down_recip;             // 1 / rows of the down share
};
static_assert(sizeof(StepShared) <= kHdrBytes, "header area");
static_assert(sizeof(StepPlan) % 16 == 0 && sizeof(StepLayer) % 16 == 0 && sizeof(ExpertW) % 16 == 0 &&
                  offsetof(StepShared, ly) % 16 == 0 && offsetof(StepShared, sew) % 16 == 0,
              "records copied as 16-byte words");

// The block's shared memory and the two things every stage needs from it. (Kept out of the
// per-thread context on purpose: that lives in local memory, and with 544 threads and a
// 24 KB L1 every access to it was a trip to L2.)
extern __shared__ __align__(128) unsigned char step_smem[];
#define SH (reinterpret_cast<StepShared *>(step_smem))
#define PL (reinterpret_cast<StepShared *>(step_smem)->plan)

// kClock: with the stage clock (the step without it has no trace of it).
//
// A layer runs every piece of code once, so code is fetched, not reused: straight code takes 1 cycle an
// instruction from the SM's first-level cache up to about 28 KB, 3 to 4 from the next level (to 128 KB), 64 beyond
// it, and more where it jumps. Loops are therefore rolled wherever their latency allows, and
// what two stages share (dot_tiles, norm_quant, gather, divisions) is one function that is called.
template <bool kClock>
struct Step {

static __device__ __forceinline__ void csync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
static __device__ __forceinline__ void hsync() { asm volatile("bar.sync 2, 256;" ::: "memory"); }  // threads 0..255
static __device__ __forceinline__ unsigned long long gtime_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
static __device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

static __device__ __forceinline__ void step_fail(int code) {
  SH->fail = code;
  atomicExch(PL.error, code);
}
// Bounded wait on an mbarrier phase; false when it gave up (now or earlier). The loop is out of line.
static __device__ __noinline__ bool mbar_wait_slow(uint32_t addr, uint32_t parity, int code) {
  if (SH->fail) return false;
  const long long t0 = clock64();
#pragma unroll 1
  for (unsigned i = 1;; ++i) {
    if (mbar_try_a(addr, parity)) return true;
    if ((i & 63u) == 0u) {
      if (SH->fail) return false;
      if (clock64() - t0 > kWaitCycles) {
        step_fail(code);
        return false;
      }
    }
  }
}
static __device__ __forceinline__ bool mbar_wait_b(uint32_t addr, uint32_t parity, int code) {
  return mbar_try_a(addr, parity) || mbar_wait_slow(addr, parity, code);
}

// Optional stage clock (plan->stage_stamps non-null): block 0 appends (id << 48 | %globaltimer)
// records, consumer thread 0 to the first half of the buffer, the producer thread to the second.
// Consumer ids: 1 a stage's input has arrived (a gather, or the barrier of the attention), 2 its prologue (norm /
// quantiser) is done, 3 its rows are done, 5 the experts are selected and their pointer records fetched, 20-24 inside
// the attention stage (heads prepared, scores, softmax, values). Producer ids: 10-11 the tiles of the first projections
// and the output projection are issued, 12 those of the router, 13 the selection arrived, 14 / 15 the gate/up and the
// down tiles are issued. A record costs about a hundred nanoseconds.
static __device__ __forceinline__ void stamp(int id) {
  if (kClock) stamp_now(id);
}
static __device__ __noinline__ void stamp_now(int id) {
  if (PL.stage_stamps && blockIdx.x == 0 && (threadIdx.x == 0 || threadIdx.x == kCons)) {
    const int who = threadIdx.x == 0 ? 0 : 1, half = PL.stage_stamp_cap / 2;
    const int n = SH->nstamp[who];
    if (n < half)
      PL.stage_stamps[who * half + n] = ((unsigned long long)id << 48) | (gtime_ns() & 0xFFFFFFFFFFFFull);
    SH->nstamp[who] = n + 1;
  }
}

// Rows [lo, hi) of `total` for block blk of nblk, cut at multiples of `unit` rows.
static __device__ __forceinline__ void deal(int total, int unit, int blk, int nblk, int &lo, int &hi) {
  const long units = (total + unit - 1) / unit;
  lo = (int)(units * blk / nblk) * unit;
  hi = (int)(units * (blk + 1) / nblk) * unit;
  if (hi > total) hi = total;
  if (lo > total) lo = total;
}
// Row unit that keeps a block's share of the bf16 group scales 16-byte aligned (2*K/128 bytes per row).
static __device__ __forceinline__ int row_unit(int K) {
  const int G = K >> 7;
  return G >= 8 ? 1 : 8 / G;
}
// Shares of all stages, once per launch: the divisions cost about a thousand cycles, and the shares
// depend on the shapes alone.
static __device__ __forceinline__ void deal_all(int i) {
  const StepPlan &P = PL;
  int total, unit;
  if (i < kRngOut) { total = P.in_rows[i - kRngIn]; unit = row_unit(P.H); }
  else if (i < kRngRouter) { total = P.H; unit = row_unit(i == kRngOut ? P.nV * 128 : P.nQ * 256); }
  else if (i == kRngRouter) { total = P.E + P.slots - P.topk; unit = 1; }
  else if (i == kRngGateUp) { total = P.slots * P.I; unit = row_unit(P.H); }
  else if (i == kRngDown) { total = P.H; unit = row_unit(P.I); }
  else { total = P.vocab; unit = row_unit(P.H); }
  int lo, hi;
  deal(total, unit, (int)blockIdx.x, (int)gridDim.x, lo, hi);
  SH->rng[i] = make_int2(lo, hi);
  if (i == kRngDown) SH->down_recip = hi > lo ? 1.0f / (float)(hi - lo) : 0.0f;
}

// ---------------------------------------------------------------- arrivals ---
// Every block counts itself once at the end of every stage. The count runs on from launch to launch.
// Ordered: a grid barrier; not ordered: only a sign that the other blocks' words are (about to be) there.
template <bool kOrdered>
static __device__ __forceinline__ void arrive() {
  csync();
  if (threadIdx.x == 0) {
    if (kOrdered) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(PL.sync + STEP_BAR) : "memory");
    else asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(PL.sync + STEP_BAR) : "memory");
  }
}
// After 64 polls in vain, and every 64th from then on. t0: clock at the 64th; returns it, or -1 when the wait
// is over (error word set). By value: a variable whose address is taken lives in memory.
static __device__ __noinline__ long long poll_late(unsigned n, long long t0) {
  const long long now = clock64();
  if (n == 64u) t0 = now;
  if (!SH->fail) {
    if (*(volatile int *)PL.error != 0) SH->fail = 1;
    else if (now - t0 > kWaitCycles) step_fail(1);
  }
  return SH->fail ? -1 : t0;
}
// Until the count has reached `target`. One thread polls: the words themselves, polled by every thread
// of every block, keep their own writers out (a router's 513 words took 5.5 us to arrive, against 1.1). A block that has
// no item of the recurrence or of the attention counts itself in for that stage without waiting for the one before, so there the
// count may be met early and the words are polled by all threads after all; a barrier (arrive<true>) is still one, as no
// block can count more often than it has ended stages.
static __device__ __noinline__ void await(unsigned target) {
  if (threadIdx.x == 0) {
    long long t0 = 0;
#pragma unroll 1
    for (unsigned i = 1; (int)(ld_acquire_u32(PL.sync + STEP_BAR) - target) < 0; ++i)
      if ((i & 63u) == 0u && (t0 = poll_late(i, t0)) < 0) break;
  }
  csync();
}

// ====================================================================== producer ===

// Streams the rows of the segment list in shared memory (SH->segs), laid end to end, through
// the ring in tiles of 16 KB. Called by the whole producer warp: lane l (l < kNT) owns ring slot
// l and issues the tiles whose running index is l modulo kNT, so up to kNT tiles are prepared and
// issued at once. Tile j of the call holds rows [j * rpt, (j + 1) * rpt) of the list, so the
// consumers know what every tile holds without being told. The group scales of a piece travel
// by bulk copy when source, size and offset are 16-byte aligned; otherwise (small matrices) the
// lane copies them itself before it completes the tile. `tile` is the running index of the
// call's first tile; returns the index after its last.
// total: rows of the list.
static __device__ __forceinline__ uint32_t prod_emit(uint32_t tile, int nseg, int row_bytes, int sc_row_bytes, int total) {
  const Seg *segs = SH->segs;
  const int lrpt = __ffs(kTileBytes) - __ffs(row_bytes), rpt = 1 << lrpt;   // both powers of two
  const int ntiles = (total + rpt - 1) >> lrpt;
  const uint32_t base = tile;
  const int lane = threadIdx.x & 31;
  if (lane < kNT && ntiles > 0) {
    unsigned char *ring = step_smem + kRingOff;
    int j = (int)(((uint32_t)lane + kNT - base % kNT) % kNT);  // first tile of this call that lands in slot `lane`
#pragma unroll 1
    for (; j < ntiles; j += kNT) {
      const uint32_t g = base + (uint32_t)j, slot = (uint32_t)lane, use = g / kNT;
      if (use > 0 && !mbar_wait_b(smem_addr(&SH->empty[slot]), (use - 1u) & 1u, 3)) break;
      unsigned char *dst = ring + slot * kTileStride;
      unsigned long long *bar = &SH->full[slot];
      const int f0 = j * rpt, f1 = f0 + rpt < total ? f0 + rpt : total;
      int row0 = 0;  // flat row of the current segment's first row
#pragma unroll 1
      for (int si = 0; si < nseg && row0 < f1; ++si) {
        const Seg sg = segs[si];
        const int a = row0 > f0 ? row0 : f0, b = row0 + sg.nrows < f1 ? row0 + sg.nrows : f1;
        if (a < b) {
          const int sr = a - row0, take = b - a, rows = a - f0;
          const uint8_t *src = sg.P + (size_t)sr * row_bytes;
          const uint8_t *ssrc = sg.S ? sg.S + (size_t)sr * sc_row_bytes : nullptr;
          const uint32_t wb = (uint32_t)(take * row_bytes), sb = (uint32_t)(take * sc_row_bytes);
          const bool sc_bulk = ssrc != nullptr &&
                               ((reinterpret_cast<uintptr_t>(ssrc) | sb | (uint32_t)(rows * sc_row_bytes)) & 15u) == 0;
          if (ssrc != nullptr && !sc_bulk) {
            const uint16_t *s16 = reinterpret_cast<const uint16_t *>(ssrc);
            uint16_t *d16 = reinterpret_cast<uint16_t *>(dst + kTileBytes + (size_t)rows * sc_row_bytes);
#pragma unroll 1
            for (uint32_t i = 0; i < sb / 2; ++i) d16[i] = __ldg(s16 + i);
          }
          if (reinterpret_cast<uintptr_t>(src) & 15u) {  // cannot be copied in bulk: report, skip
            if (g_stream_fault_word) *reinterpret_cast<volatile unsigned int *>(g_stream_fault_word) = 2;
          } else {
            mbar_expect_tx(bar, wb + (sc_bulk ? sb : 0u));
            bulk_g2s(dst + (size_t)rows * row_bytes, src, wb, bar);
            if (sc_bulk) bulk_g2s(dst + kTileBytes + (size_t)rows * sc_row_bytes, ssrc, sb, bar);
          }
        }
        row0 += sg.nrows;
      }
      mbar_arrive(bar);  // releases this lane's own stores and completes the phase once the bytes have landed
    }
  }
  __syncwarp();  // the list may be rewritten once every lane is done with it
  return base + (uint32_t)ntiles;
}

// The producer warp's whole token: the lists of a layer's five streams one after the other, a lane a
// segment. Returns the number of tiles issued.
static __device__ __noinline__ uint32_t producer_main(int mode) {
  const StepPlan &P = PL;
  const int H = P.H, I = P.I, lane = threadIdx.x & 31, lgI = __ffs(I) - 1;
  uint32_t tile = 0;
#pragma unroll 1
  for (int L = 0; L < P.layers + (mode != 0 ? 1 : 0); ++L) {
    const StepLayer &ly = P.L[L];
#pragma unroll 1
    for (int job = 0; job < 5; ++job) {
      const bool head = L == P.layers;
      // first projections (or LM head) | output projection | router and shared-expert gate | gate and up | down
      const int type = head ? 0 : ly.type;
      const int2 rows = SH->rng[head ? kRngHead : job == 0 ? kRngIn + type : job == 1 ? kRngOut + type : kRngRouter + job - 2];
      const int lo = rows.x, hi = rows.y;
      int K = H, nseg = 0, total = hi - lo;
      Seg sg = Seg{nullptr, nullptr, 0, 0, 0, 0};
      if (job < 2) {
        const GemvMat *m = head ? &P.lm_head : &ly.m[job * 4];
        nseg = job == 1 || head ? 1 : type == 0 ? 4 : 3;
        if (job == 1) K = type == 0 ? P.nV * 128 : P.nQ * 256;
        if (lane < nseg) {
          int rs = 0;
          for (int i = 0; i < lane; ++i) rs += m[i].N;
          const int N = m[lane].N, a = lo > rs ? lo : rs, b = hi < rs + N ? hi : rs + N;
          if (a < b) sg = Seg{m[lane].P + (size_t)(a - rs) * (K >> 1), reinterpret_cast<const uint8_t *>(m[lane].S + (size_t)(a - rs) * (K >> 7)), b - a, 0, 0, 0};
        }
      } else if (job == 2) {   // bf16 rows
        nseg = 2;
        const int b = hi < P.E ? hi : P.E;
        if (lane == 0 && lo < b) sg = Seg{reinterpret_cast<const uint8_t *>(ly.router + (size_t)lo * H), nullptr, b - lo, 0, 0, 0};
        if (lane == 1 && hi > P.E) sg = Seg{reinterpret_cast<const uint8_t *>(ly.shared_gate), nullptr, 1, 0, 0, 0};
      } else if (job == 3) {   // pair rows [lo, hi) over slots x I: a slot's gate rows, then its up rows
        stamp(12);
        // the expert weights depend on the routing: wait for the consumers' selection
        if (!mbar_wait_b(smem_addr(&SH->sel_bar), (uint32_t)L & 1u, 4)) return tile;
        stamp(13);
        total = 2 * (hi - lo);
        if (lo < hi) {
          const int s0 = lo >> lgI, s = s0 + (lane >> 1);
          nseg = 2 * (((hi - 1) >> lgI) - s0 + 1);
          if (lane < nseg) {
            const int a = lo > s * I ? lo : s * I, b = hi < (s + 1) * I ? hi : (s + 1) * I;
            const ExpertW &ew = SH->sew[s];
            const size_t r0 = (size_t)(a - s * I);
            sg = Seg{((lane & 1) ? ew.uP : ew.gP) + r0 * (H >> 1), reinterpret_cast<const uint8_t *>(((lane & 1) ? ew.uS : ew.gS) + r0 * (H >> 7)), b - a, 0, 0, 0};
          }
        }
      } else {   // down rows [lo, hi) of every slot
        K = I;
        nseg = P.slots;
        total = P.slots * (hi - lo);
        if (lane < nseg) {
          const ExpertW &ew = SH->sew[lane];
          sg = Seg{ew.dP + (size_t)lo * (I >> 1), reinterpret_cast<const uint8_t *>(ew.dS + (size_t)lo * (I >> 7)), hi - lo, 0, 0, 0};
        }
      }
      if (lane < nseg) SH->segs[lane] = sg;
      __syncwarp();
      tile = prod_emit(tile, nseg, job == 2 ? H * 2 : K >> 1, job == 2 ? 0 : (K >> 7) * 2, total);
      stamp(job < 2 ? 10 + job : 11 + job);
      if (head) break;
    }
  }
  return tile;
}

// ======================================================== words between blocks ===
// What one stage hands to the next crosses the grid as 64-bit words of a value and a flag (the
// launch's and layer's number). A word is one access, so the value is there when the flag is, and the
// writer needs no fence in front of its arrival. Nothing else is ordered, and no
// stage reads anything of another block in any other way (the chunk partials of the attention, too many
// for words of twice their size, keep a barrier). Words alternate between two sets by layer: a
// block writes layer L + 2's only after it has read words that depend on every block's rows of layer L + 1's first
// stage (the host deals at least one to each), which a block computes after its last read of layer L.
static __device__ __forceinline__ void put(unsigned long long *p, float v, unsigned flag) {
  asm volatile("{\n\t.reg .b64 w;\n\tmov.b64 w, {%1, %2};\n\tst.relaxed.gpu.global.b64 [%0], w;\n\t}" ::"l"(p),
               "r"(__float_as_uint(v)), "r"(flag)
               : "memory");
}
// One word.
static __device__ __forceinline__ float take(const unsigned long long *p, unsigned flag) {
  unsigned v, f, n = 0;
  long long t0 = 0;
#pragma unroll 1
  while (true) {
    asm volatile("{\n\t.reg .b64 w;\n\tld.relaxed.gpu.global.b64 w, [%2];\n\tmov.b64 {%0, %1}, w;\n\t}" : "=r"(v), "=r"(f) : "l"(p) : "memory");
    if (f == flag) break;
    if ((++n & 63u) == 0u && (t0 = poll_late(n, t0)) < 0) break;
  }
  return __uint_as_float(v);
}
// Eight words 32 apart, all in flight together.
static __device__ __forceinline__ void take8(float (&x)[8], const unsigned long long *p, unsigned flag) {
  unsigned n = 0;
  long long t0 = 0;
#pragma unroll 1
  while (true) {
    unsigned f[8];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      asm volatile("{\n\t.reg .b64 w;\n\tld.relaxed.gpu.global.b64 w, [%2];\n\tmov.b64 {%0, %1}, w;\n\t}"
                   : "=f"(x[i]), "=r"(f[i])
                   : "l"(p + 32 * i)
                   : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) ok = ok && f[i] == flag;
    if (ok || ((++n & 63u) == 0u && (t0 = poll_late(n, t0)) < 0)) break;
  }
}
// n consecutive words (16-byte aligned) into shared memory, by the whole consumer group: two pairs
// (four words) a thread in flight. The caller synchronises.
static __device__ __noinline__ void gather(float *dst, const unsigned long long *src, int n, unsigned flag) {
  unsigned tries = 0;
  long long t0 = 0;
#pragma unroll 1
  for (int w = 2 * (int)threadIdx.x; w < n; w += 4 * kCons) {
    unsigned v0[2], f0[2], v1[2], f1[2];
#pragma unroll 1
    while (true) {
      bool ok = true;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        f0[u] = f1[u] = flag;
        if (w + 2 * kCons * u < n)
          asm volatile("{\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.v2.b64 {a, b}, [%4];\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
                       : "=r"(v0[u]), "=r"(f0[u]), "=r"(v1[u]), "=r"(f1[u])
                       : "l"(src + w + 2 * kCons * u)
                       : "memory");
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) ok = ok && f0[u] == flag && (f1[u] == flag || w + 2 * kCons * u + 1 >= n);
      if (ok) break;
      if ((++tries & 63u) == 0u && (t0 = poll_late(tries, t0)) < 0) break;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (w + 2 * kCons * u < n) *reinterpret_cast<uint2 *>(dst + w + 2 * kCons * u) = make_uint2(v0[u], v1[u]);
  }
}

// num / (1 + exp(arg)) and 1 / sqrt(x): one copy each, see Step.
static __device__ __noinline__ float over_exp(float num, float arg) { return num / (1.0f + det_expf(arg)); }
static __device__ __noinline__ float inv_sqrt(float x) { return 1.0f / sqrtf(x); }

// ====================================================================== consumers ===
// Group terms of a stage's rows: t[row][g], 4-term pieces in an order that turns with the row, so that
// the thread that adds a row's terms reads them four at a time.
static __device__ __forceinline__ int term_index(int row, int g, int lg) {
  return lg >= 2 ? (row << lg) + ((((g >> 2) ^ row) & ((1 << (lg - 2)) - 1)) << 2) + (g & 3) : (row << lg) + g;
}
// Sum of one row's group terms in ascending group order.
static __device__ __forceinline__ float row_terms(const float *T, int row, int lg) {
  float acc = 0.0f;
  if (lg >= 2) {
    const float4 *t = reinterpret_cast<const float4 *>(T + (row << lg));
    const int n = 1 << (lg - 2);
    float4 v = t[row & (n - 1)];
#pragma unroll 1
    for (int i = 1; i <= n; ++i) {
      const float4 c = v;
      if (i < n) v = t[(i ^ row) & (n - 1)];
      acc = acc + c.x;
      acc = acc + c.y;
      acc = acc + c.z;
      acc = acc + c.w;
    }
  } else {
#pragma unroll 1
    for (int g = 0; g < 1 << lg; ++g) acc = acc + T[(row << lg) + g];
  }
  return acc;
}

// Dots the next tiles of a stage with staged activations: nrows rows in the order the producer
// streams them (tile j of the call holds rows [j * rpt, (j + 1) * rpt)). Row f is dotted with
// activation vector floor((f + 1/2) vec_recip), vec_recip = 1 / rows of a vector (f < 4096: the error, 2^-22 of the quotient,
// is far below the half row), and its group terms go to t[f][]. Starts at
// running tile index `tile`; returns the index after the last tile. A tile is 256 (row, group) tasks of
// 64 bytes, one a thread: the two halves of the consumers take alternate tiles, so that every
// wait, scale and store serves 64 bytes and two tiles are in work at once. A thread reads its 64
// bytes in a lane-rotated order that keeps every quarter-warp on distinct banks. Not inlined: see Step.
static __device__ __noinline__ uint32_t dot_tiles(uint32_t tile, int lg, int sq_off, int nrows, float vec_recip) {
  const uint4 *xa = reinterpret_cast<const uint4 *>(step_smem + kActOff);
  const float *sq = reinterpret_cast<const float *>(step_smem + kActOff + sq_off);
  float *T = reinterpret_cast<float *>(step_smem + kTOff);
  const int G = 1 << lg, rpt = 256 >> lg;
  const int t = threadIdx.x & 255, half = threadIdx.x >> 8, lane = threadIdx.x & 31;
  const int r = t >> lg, g = t & (G - 1), rot = (t >> 1) & 3;
  const uint32_t ring_a = smem_addr(step_smem + kRingOff);
  const int ntiles = (nrows + rpt - 1) >> (8 - lg);
  uint4 x[8];
  float sqg = 0.0f;
  int cvec = -1;
#pragma unroll 1
  for (int j = half; j < ntiles; j += 2) {
    const uint32_t idx = tile + (uint32_t)j, slot = idx % kNT, use = idx / kNT;
    const int f = j * rpt + r;
    const bool live = f < nrows;
    const int vec = live ? (int)(((float)f + 0.5f) * vec_recip) : 0;
    if (vec != cvec) {
      cvec = vec;
      const uint4 *xv = xa + (size_t)vec * 8 * G + g;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int q = 2 * ((s + rot) & 3);
        x[2 * s] = xv[q * G];
        x[2 * s + 1] = xv[(q + 1) * G];
      }
      sqg = sq[vec * G + g];
    }
    // a wait that gave up ends the stage for the whole warp (the results are lost anyway)
    if (!__all_sync(kFull, mbar_wait_b(smem_addr(&SH->full[slot]), use & 1u, 5))) break;
    const uint32_t tb = ring_a + slot * kTileStride, wb = tb + (uint32_t)t * 64u;
    const uint4 w0 = lds128(wb + (uint32_t)(rot << 4)), w1 = lds128(wb + (uint32_t)(((1 + rot) & 3) << 4)),
                w2 = lds128(wb + (uint32_t)(((2 + rot) & 3) << 4)), w3 = lds128(wb + (uint32_t)(((3 + rot) & 3) << 4));
    const uint32_t sraw = lds_u16(tb + kTileBytes + (uint32_t)t * 2u);
    int d0 = dot16_x16(w0, 0, x[0], 0), d1 = dot16_x16(w0, 1, x[1], 0);
    int d2 = dot16_x16(w1, 0, x[2], 0), d3 = dot16_x16(w1, 1, x[3], 0);
    d0 = dot16_x16(w2, 0, x[4], d0);
    d1 = dot16_x16(w2, 1, x[5], d1);
    d2 = dot16_x16(w3, 0, x[6], d2);
    d3 = dot16_x16(w3, 1, x[7], d3);
    __syncwarp();
    if (lane == 0) mbar_arrive_a(smem_addr(&SH->empty[slot]));
    const float v = (float)(((d0 + d1) + (d2 + d3)) >> 4) * __uint_as_float(sraw << 16);
    if (live) T[term_index(f, g, lg)] = v * sqg;
  }
  csync();
  return tile + (uint32_t)ntiles;
}

// Largest magnitude of the warp's values (one instruction; NaNs do not count, as with fmaxf).
static __device__ __forceinline__ float warp_absmax(float v) {
  float r;
  asm volatile("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
static __device__ __forceinline__ float warp_largest(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
// Quantises one group of 128 values held four a lane: (bytes, scale bits); scale s = largest / 127 (ScalesMax +
// Quantize, tools/cmdlist/kernels.cpp:551-579), the bytes quant_round()'s integers, from the
// approximate reciprocal r of s, 127 x rcp(largest), which is there before s is. With q = x/s, |q| <= 127 (1 + 2^-24):
// r is within 2^-22 of 1/s (one ulp of rcp, the product, the rounding of s), so x r within 3.8e-5 of q, rounded
// to 0.76e-5; the rounded quotient is within 0.76e-5 of q; and the addition of one half rounds to 2^-17 at
// most, twice: in all 6.1e-5. Unless |x r| + 0.5 is within 8e-5 of a whole number both truncate alike; there, and for an r that
// is not well inside the range, the division itself decides.
static __device__ __noinline__ uint2 quant_group(float4 v) {
  const float mx = warp_absmax(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(mx));
  r = r * 127.0f;
  float s = mx / 127.0f;
  if (s == 0.0f) s = 1.0f;
  const float x[4] = {v.x, v.y, v.z, v.w};
  uint32_t out = 0;
  bool sure = r > 1e-30f && r < 1e30f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float vp = x[i] * r, t = fabsf(vp) + 0.5f, w = truncf(t), f = t - w;
    sure = sure && f >= 8e-5f && f <= 0.99992f;
    int q = (int)w;
    q = q > 127 ? 127 : q;
    q = vp < 0.0f ? -q : q;
    out |= (uint32_t)(q & 0xFF) << (8 * i);
  }
  if (!sure) {
    out = 0;
#pragma unroll 1
    for (int i = 3; i >= 0; --i) {
      const float xi = i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
      out = (out << 8) | (uint32_t)(quant_round(xi, s) & 0xFF);
    }
  }
  return make_uint2(out, __float_as_uint(s));
}
// A group's bytes into the staged form (quant_group_staged()'s result).
static __device__ __forceinline__ void stage_group(uint32_t *xw, float *sqs, int G, int m, int g, const uint2 &qs) {
  const int lane = threadIdx.x & 31;
  const uint32_t own = qs.x, other = __shfl_xor_sync(kFull, own, 1);
  const int i = lane >> 1;  // 8-weight piece of the group: two lanes of 4 weights each
  uint32_t *dst = xw + ((((m * 8 + (i >> 1)) * G + g) << 2) + ((i & 1) << 1));
  if (lane & 1) dst[1] = __byte_perm(other, own, 0x7531);
  else dst[0] = __byte_perm(own, other, 0x6420);
  if (lane == 0) sqs[m * G + g] = __uint_as_float(qs.y);
}

// (1+w) RMSNorm + per-128 quantiser of one H-vector into the staged form, by the whole
// consumer group (RMSNormW + ScalesMax + Quantize, tools/cmdlist/kernels.cpp:73-114,551-579).
// Sum of squares: fp64 over 256 strided lanes (thread j < 256 adds x[j], x[j+256], ... in
// order; a square is exact in fp64, so one fused multiply-add a term), then the stride-halving
// tree, whose levels 128, 64 and 32 every warp evaluates for
// itself from the 256 partial sums in shared memory (lane l: ((p[l]+p[l+128]) + (p[l+64]+
// p[l+192])) + ((p[l+32]+p[l+160]) + (p[l+96]+p[l+224]))) and whose last five levels are the xor
// butterfly. The mean is a product: H is a power of two.
// src: the vector's words, or (emb != null) a bf16 embedding row. hn: the normalised fp32 vector,
// shared memory. Returns the input at row rows.x + thread, for the threads below rows.y - rows.x: the
// residual of a later stage.
static __device__ __noinline__ float norm_quant(unsigned target, const unsigned long long *src, unsigned flag, const uint16_t *emb,
                                                const float *w, int H, int2 rows) {
  float *xs = reinterpret_cast<float *>(step_smem + kFbufOff), *hn = xs + 4096;
  double *ps = reinterpret_cast<double *>(step_smem + kTOff);
  unsigned char *act = step_smem + kActOff;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, G = H >> 7;
  float4 wv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (warp < G) wv = __ldg(reinterpret_cast<const float4 *>(w + warp * 128) + lane);
  if (emb) {
#pragma unroll 1
    for (int j = tid; j < H; j += kCons) xs[j] = u2f((uint32_t)__ldg(emb + j) << 16);
  } else {
    await(target);
    gather(xs, src, H, flag);
  }
  csync();
  stamp(1);
  if (tid < 256) {
    double ss = 0;
#pragma unroll 1
    for (int j = tid; j < H; j += 1024) {   // four loads ahead of the chain (H >= 1024: all of them in range)
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = j + 256 * i < H ? xs[j + 256 * i] : 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) ss = fma((double)v[i], (double)v[i], ss);
    }
    ps[tid] = ss;
  }
  csync();
  double t = ((ps[lane] + ps[lane + 128]) + (ps[lane + 64] + ps[lane + 192])) +
             ((ps[lane + 32] + ps[lane + 160]) + (ps[lane + 96] + ps[lane + 224]));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) t = t + __shfl_xor_sync(kFull, t, off);
  const double rH = __hiloint2double((1023 - (__ffs(H) - 1)) << 20, 0);
  const float inv = inv_sqrt((float)(t * rH) + PL.eps);
#pragma unroll 1
  for (int g = warp; g < G; g += 16) {
    const int j = g * 128 + lane * 4;
    const float4 x = *reinterpret_cast<const float4 *>(xs + j);
    float4 y;
    y.x = (x.x * inv) * (1.0f + wv.x);
    y.y = (x.y * inv) * (1.0f + wv.y);
    y.z = (x.z * inv) * (1.0f + wv.z);
    y.w = (x.w * inv) * (1.0f + wv.w);
    if (g + 16 < G) wv = __ldg(reinterpret_cast<const float4 *>(w + (g + 16) * 128) + lane);
    *reinterpret_cast<float4 *>(hn + j) = y;
    stage_group(reinterpret_cast<uint32_t *>(act), reinterpret_cast<float *>(act + H), G, 0, g, quant_group(y));
  }
  const float res = tid < rows.y - rows.x ? xs[rows.x + tid] : 0.0f;
  csync();
  stamp(2);
  return res;
}

// Gated per-head norm + quantiser (RmsInv + NormGated + ScalesMax + Quantize,
// kernels.cpp:619-644,551-579) into the staged form (K = nV * 128 <= 4096), a warp a head. The
// words of z hold silu(z): the projection's epilogue has it from one thread a row,
// where every block would evaluate nV * 128 exponentials here. Lane l takes values l, l + 32, l + 64 and
// l + 96 of a head, the terms of its sum of squares.
static __device__ __forceinline__ void gated_norm_quant(unsigned target, const unsigned long long *O, const unsigned long long *Zs,
                                                        unsigned flag, const float *W, int nV) {
  float *os = reinterpret_cast<float *>(step_smem + kFbufOff), *zs = os + 4096;
  unsigned char *act = step_smem + kActOff;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float wn[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) wn[i] = __ldg(W + lane + 32 * i);
  gather(zs, Zs, nV * 128, flag);   // complete since the recurrence's inputs were
  await(target);
  gather(os, O, nV * 128, flag);
  csync();
  stamp(1);
  int8_t *xb = reinterpret_cast<int8_t *>(act);
  float *sqs = reinterpret_cast<float *>(act + nV * 128);
#pragma unroll 1
  for (int h = warp; h < nV; h += 16) {
    float o[4], z[4], ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[i] = os[h * 128 + lane + 32 * i];
      z[i] = zs[h * 128 + lane + 32 * i];
      ss = fmaf(o[i], o[i], ss);
    }
    ss = warp_tree_sum(ss);
    const float inv = inv_sqrt(ss * 0.0078125f + PL.eps);
    float4 y;
    y.x = ((wn[0] * o[0]) * inv) * z[0];
    y.y = ((wn[1] * o[1]) * inv) * z[1];
    y.z = ((wn[2] * o[2]) * inv) * z[2];
    y.w = ((wn[3] * o[3]) * inv) * z[3];
    const uint2 qs = quant_group(y);
    const uint32_t q = qs.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // value k of the group: piece k / 8 (two words: even and odd values), byte (k % 8) / 2 of its word
      const int k = lane + 32 * i, pc = k >> 3;
      xb[((((pc >> 1) * nV + h) << 2) + ((pc & 1) << 1) + (k & 1)) * 4 + ((k & 7) >> 1)] = (int8_t)(q >> (8 * i));
    }
    if (lane == 0) sqs[h] = __uint_as_float(qs.y);
  }
  csync();
}

// Matrix and local row of flat row `flat` of a table of matrices.
static __device__ __forceinline__ int mat_of_row(const GemvMat *m, int nm, int flat, int &n) {
  int rs = 0, i = 0;
#pragma unroll 1
  while (i < nm - 1 && flat >= rs + m[i].N) {
    rs += m[i].N;
    ++i;
  }
  n = flat - rs;
  return i;
}

// Operands of a row's epilogue that do not depend on its dot product: 32 bytes of shared memory a row,
// under way during the dot as asynchronous copies (registers that wait for them would be spilled, and the
// spill would wait): convolution taps [0..3] and history [4..6], or decay constants [4], [5]. All of
// them are read once a launch, so that no cached line is older than they are.
static __device__ __forceinline__ void cp_async4(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
static __device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
static __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
static __device__ __forceinline__ void row_operands(const GemvMat &mt, int n, float *op) {
  const int epi = mt.epi;
  if (epi == EPI_CONV_SILU) {
    const float *cs = mt.e1 + (size_t)n * 3;
    cp_async16(op, mt.e0 + (size_t)n * 4);
    cp_async4(op + 4, cs);
    cp_async4(op + 5, cs + 1);
    cp_async4(op + 6, cs + 2);
  }
  if (epi == EPI_GDECAY) {
    cp_async4(op + 4, mt.e0 + n);
    cp_async4(op + 5, mt.e2 + n);
  }
}
// gemv_epilogue()'s arithmetic; every kind of row that needs an exponential of its sum shares one.
static __device__ __forceinline__ float row_epilogue(const GemvMat &mt, int n, float acc, const float *op, float res) {
  const int epi = mt.epi;
  if (epi == EPI_STORE) return acc;
  if (epi == EPI_RESADD) return res + acc;
  float num = epi == EPI_BETA ? 1.0f : acc, arg = -acc;
  if (epi == EPI_CONV_SILU) {
    const float4 cw = *reinterpret_cast<const float4 *>(op);
    const float c1 = op[5], c2 = op[6];
    float a = op[4] * cw.x;
    a = a + c1 * cw.y;
    a = a + c2 * cw.z;
    a = a + acc * cw.w;
    num = a;
    arg = -a;
    float *cs = mt.e1 + (size_t)n * 3;
    cs[0] = c1;
    cs[1] = c2;
    cs[2] = acc;
  }
  if (epi == EPI_GDECAY) arg = acc + op[5];
  if (epi != EPI_GDECAY) return over_exp(num, arg);
  const float soft = arg > 20.0f ? arg : det_logf(1.0f + det_expf(arg));
  return (-det_expf(op[4])) * soft;
}

// One GEMV stage: this block's rows of the matrices, activations already staged; a matrix's Y is its
// rows' words. res: the residual of row `thread` of the share.
static __device__ __noinline__ uint32_t gemv_stage_run(uint32_t tile, const GemvMat *m, int nm, int K, int2 rows, unsigned flag, float res) {
  const int lo = rows.x, nr = rows.y - lo;
  const float *T = reinterpret_cast<const float *>(step_smem + kTOff);
  float *op = reinterpret_cast<float *>(step_smem + kFbufOff) + 4096 + threadIdx.x * 8;
  const int lg = 31 - __clz(K >> 7);
  int mi = 0, n = 0;
  if ((int)threadIdx.x < nr) {
    mi = mat_of_row(m, nm, lo + threadIdx.x, n);
    row_operands(m[mi], n, op);
  }
  tile = dot_tiles(tile, lg, K, nr, 0.0f);
  if ((int)threadIdx.x < nr) {   // nr <= 512
    cp_async_wait();   // the thread's own copies
    put(reinterpret_cast<unsigned long long *>(m[mi].Y) + n, row_epilogue(m[mi], n, row_terms(T, threadIdx.x, lg), op, res), flag);
  }
  stamp(3);
  return tile;
}

// Router logits of this block's rows from the ring (bf16 rows), activations hn in shared memory.
// logits[e] = sum_k bf16(W[e][k]) * hn[k]: lane l takes k = (i*32+l)*8+j, fma chain in (i, j)
// order, then the lane tree (as RouterTopK). Tiles go to alternate halves of the consumers, as in dot_tiles.
static __device__ __forceinline__ uint32_t router_stage(uint32_t tile, unsigned long long *out, unsigned flag, int H) {
  const int lo = SH->rng[kRngRouter].x, total = SH->rng[kRngRouter].y - lo;
  const float *hn = reinterpret_cast<const float *>(step_smem + kFbufOff) + 4096;
  const int warp = (threadIdx.x >> 5) & 7, half = threadIdx.x >> 8, lane = threadIdx.x & 31, n = H >> 8;
  const int lrpt = __ffs(kTileBytes) - __ffs(H * 2), rpt = 1 << lrpt, ntiles = (total + rpt - 1) >> lrpt;
  const uint32_t ring_a = smem_addr(step_smem + kRingOff);
#pragma unroll 1
  for (int j = half; j < ntiles; j += 2) {
    const uint32_t idx = tile + (uint32_t)j, slot = idx % kNT, use = idx / kNT;
    if (!__all_sync(kFull, mbar_wait_b(smem_addr(&SH->full[slot]), use & 1u, 5))) break;
    const uint32_t tb = ring_a + slot * kTileStride;
    const int nr = total - j * rpt < rpt ? total - j * rpt : rpt;
#pragma unroll 1
    for (int r = warp; r < nr; r += 8) {
      float acc = 0.0f;
      const uint32_t wb = tb + (uint32_t)r * (uint32_t)(H * 2) + (uint32_t)lane * 16u;
      const float *hb = hn + lane * 8;
      uint4 wv = lds128(wb);
      float4 a0 = *reinterpret_cast<const float4 *>(hb), a1 = *reinterpret_cast<const float4 *>(hb + 4);
#pragma unroll 1
      for (int i = 1; i <= n; ++i) {   // the next piece is on its way while this one is added
        const uint4 w = wv;
        const float4 x0 = a0, x1 = a1;
        if (i < n) {
          wv = lds128(wb + (uint32_t)i * 512u);
          a0 = *reinterpret_cast<const float4 *>(hb + i * 256);
          a1 = *reinterpret_cast<const float4 *>(hb + i * 256 + 4);
        }
        acc = fmaf(u2f(w.x << 16), x0.x, acc);
        acc = fmaf(u2f(w.x & 0xFFFF0000u), x0.y, acc);
        acc = fmaf(u2f(w.y << 16), x0.z, acc);
        acc = fmaf(u2f(w.y & 0xFFFF0000u), x0.w, acc);
        acc = fmaf(u2f(w.z << 16), x1.x, acc);
        acc = fmaf(u2f(w.z & 0xFFFF0000u), x1.y, acc);
        acc = fmaf(u2f(w.w << 16), x1.z, acc);
        acc = fmaf(u2f(w.w & 0xFFFF0000u), x1.w, acc);
      }
      acc = warp_tree_sum(acc);
      if (lane == 0) put(out + lo + j * rpt + r, acc, flag);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_a(smem_addr(&SH->empty[slot]));
  }
  return tile + (uint32_t)ntiles;
}

// Softmax over the E <= 1024 router logits, top-k by (probability desc, index asc), renormalised
// weights, shared-expert gate: the selection of RouterTopK, run by every block for itself, with the
// selected experts' pointer records fetched on the way. Order of experts: key = bits of the
// probability + 1 (it is >= 0, so the bits order like integers), then the lower index. The
// nsel-th largest of the sixteen warps' largest keys bounds the nsel-th largest of all from below,
// so the entries at or above it (about 17 of 512 for a top 10) hold the whole selection: they are
// gathered, and each one's rank is the number of candidates ahead of it. slots <= 12, so nsel <=
// 13 of the sixteen maxima. The exponentials are padded to whole runs of 512 entries with zeros.
static __device__ __forceinline__ void router_select_cons(unsigned target, const unsigned long long *logits, unsigned flag, const ExpertW *experts,
                                                          int E, int k, bool has_shared) {
  float *lg = reinterpret_cast<float *>(step_smem + kFbufOff), *sp = lg + 2048, *pr = lg + 4096;
  unsigned long long *cand = reinterpret_cast<unsigned long long *>(step_smem + kTOff);   // up to E candidates
  StepShared *sh = SH;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, runs = (E + kCons - 1) / kCons;
  await(target);
  gather(lg, logits, E + (has_shared ? 1 : 0), flag);
  if (tid == 0) sh->ncand = 0;
  csync();
  stamp(1);
  // maximum and sum keep the one-warp partition (lane l takes entries l, l+32, ... in ascending
  // order, then the xor butterfly); every warp evaluates them for itself, which gives every warp
  // the same bits and saves two block barriers and two one-warp sections
  float m = -INFINITY;
#pragma unroll 4
  for (int e = lane; e < E; e += 32) m = fmaxf(m, lg[e]);
  m = warp_largest(m);
#pragma unroll 1
  for (int u = 0; u < runs; ++u) {
    const int e = tid + kCons * u;
    sp[e] = e < E ? det_expf(lg[e] - m) : 0.0f;
  }
  csync();
  float sum = 0.0f;
#pragma unroll 1
  for (int e = lane; e < runs * kCons; e += 256) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = sp[e + 32 * i];
#pragma unroll
    for (int i = 0; i < 8; ++i) sum = sum + v[i];
  }
  sum = warp_tree_sum(sum);
  unsigned *keys = reinterpret_cast<unsigned *>(lg);   // over the logits, which every warp has read (lg[E] stays)
  unsigned wk = 0u;
#pragma unroll 1
  for (int e = tid; e < E; e += kCons) {
    const unsigned key = __float_as_uint(sp[e] / sum) + 1u;
    keys[e] = key;   // read by the same thread
    wk = key > wk ? key : wk;
  }
  wk = __reduce_max_sync(kFull, wk);
  if (lane == 0) sh->kmax[warp] = wk;
  csync();
  const int nsel = k < E ? k + 1 : k;
  const unsigned mine = lane < 16 ? sh->kmax[lane] : 0u;
  int ahead = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const unsigned o = sh->kmax[i];
    ahead += o > mine || (o == mine && i < lane);
  }
  unsigned bound = __reduce_min_sync(kFull, lane < 16 && ahead < nsel ? mine : 0xFFFFFFFFu);
  if (bound == 0u) bound = 1u;   // fewer warps than nsel hold entries: all of them are candidates
#pragma unroll 1
  for (int e = tid; e < E; e += kCons)
    if (keys[e] >= bound) cand[atomicAdd(&sh->ncand, 1)] = ((unsigned long long)keys[e] << 32) | (0xFFFFFFFFu - (unsigned)e);
  csync();
  const int nc = sh->ncand;
#pragma unroll 1
  for (int i = warp; i < nc; i += 16) {
    const unsigned long long c = cand[i];
    int rank = 0;
#pragma unroll 1
    for (int j0 = 0; j0 < nc; j0 += 32) rank += __popc(__ballot_sync(kFull, j0 + lane < nc && cand[j0 + lane] > c));
    if (rank > k) continue;
    const int e = (int)(0xFFFFFFFFu - (unsigned)c);
    if (rank < k && lane < 3)
      reinterpret_cast<uint4 *>(sh->sew + rank)[lane] = __ldg(reinterpret_cast<const uint4 *>(experts + e) + lane);
    if (lane == 0) {
      pr[rank] = __uint_as_float((unsigned)(c >> 32) - 1u);
      if (rank < k) sh->sel_idx[rank] = e;
    }
  }
  if (warp == 15) {
    if (has_shared && lane < 3)
      reinterpret_cast<uint4 *>(sh->sew + k)[lane] = __ldg(reinterpret_cast<const uint4 *>(experts + E) + lane);
    if (lane == 0) {
      sh->sel_idx[k] = E;
      sh->sel_w[k] = has_shared ? over_exp(1.0f, -lg[E]) : 0.0f;
    }
  }
  csync();
  if (tid == 0) mbar_arrive(&sh->sel_bar);  // the producer may now stream the experts
  stamp(5);
  // the weights are needed by the down projection only
  if (warp == 1) {
    float s = 0.0f;
#pragma unroll 1
    for (int j = 0; j < k && j < E; ++j) s = s + pr[j];
    if (lane < k) sh->sel_w[lane] = (lane < E ? pr[lane] : 0.0f) / s;
    if (lane == 0) {
      const float lastp = pr[k - 1];
      sh->gap = k >= E ? 1.0f : (lastp > 0.0f ? (lastp - pr[k]) / lastp : 0.0f);
    }
  }
}

// ------------------------------------------------------------ gated delta rule ---
// One (head, column slice) item per block; the arithmetic is DeltaNetStep's (deltanet_core.cuh). The
// slice of the state, 128 rows of 32 columns, comes to shared memory by asynchronous copies while the words are
// waited for: it was last written one token ago by this same block. Warp w < 8 owns segment w of the rows.
static __device__ __noinline__ void deltanet_stage(unsigned target, const StepLayer &ly, const unsigned long long *Mx,
                                                   const unsigned long long *Bt, const unsigned long long *Gt, unsigned long long *O,
                                                   unsigned flag) {
  const StepPlan &P = PL;
  constexpr int D = 128, SEG = kDnSeg;
  const int nitems = P.nV * kDnSlices, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, per_k = P.nV / P.nK;
  // q | k | value slice | beta | decay of the item, then the segments' partial sums
  float *raw = reinterpret_cast<float *>(step_smem + kTOff), *st = reinterpret_cast<float *>(step_smem + kFbufOff);
  float *part = raw + 512;
  csync();   // the first projections' terms and operands are read
#pragma unroll 1
  for (int item = (int)blockIdx.x; item < nitems; item += (int)gridDim.x) {
    const int h = item / kDnSlices, slice = item % kDnSlices, kh = h / per_k;
    float *S0 = ly.S + (size_t)h * D * D + slice * 32;
#pragma unroll 1
    for (int i = tid; i < D * 8; i += kCons) cp_async16(st + i * 4, S0 + (i >> 3) * D + (i & 7) * 4);
    if (item == (int)blockIdx.x) await(target);
    if (tid < 290) {
      const unsigned long long *w = tid < 128 ? Mx + kh * D + tid
                                    : tid < 256 ? Mx + (P.nK + kh) * D + tid - 128
                                    : tid < 288 ? Mx + (2 * P.nK + h) * D + slice * 32 + tid - 256
                                    : tid == 288 ? Bt + h : Gt + h;
      raw[tid] = take(w, flag);
    }
    cp_async_wait();
    csync();
    stamp(1);
    if (tid < 256) {
      float sq = 0.0f, sk = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float q = raw[lane + 32 * i], k = raw[D + lane + 32 * i];
        sq = fmaf(q, q, sq);
        sk = fmaf(k, k, sk);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        sq = sq + __shfl_xor_sync(kFull, sq, off);
        sk = sk + __shfl_xor_sync(kFull, sk, off);
      }
      const float fq = inv_sqrt(sq + 1e-6f) * 0.0883883476483184405f, fk = inv_sqrt(sk + 1e-6f);
      const float val = raw[256 + lane], beta = raw[288], gt = det_expf(raw[289]);
      const float *kr = raw + D + warp * SEG, *qr = raw + warp * SEG, *sr = st + warp * SEG * 32 + lane;
      float acc = 0.0f;
#pragma unroll 4
      for (int r = 0; r < SEG; ++r) acc = fmaf(sr[r * 32] * gt, kr[r] * fk, acc);
      part[tid] = acc;
      hsync();
      const float *p = part + lane;
      const float kv = ((p[0] + p[32]) + (p[64] + p[96])) + ((p[128] + p[160]) + (p[192] + p[224]));
      const float dl = (val - kv) * beta;
      float *Sh = S0 + (size_t)warp * SEG * D + lane;
      acc = 0.0f;
#pragma unroll 4
      for (int r = 0; r < SEG; ++r) {
        const float s = fmaf(kr[r] * fk, dl, sr[r * 32] * gt);
        acc = fmaf(s, qr[r] * fq, acc);
        Sh[r * D] = s;
      }
      part[256 + tid] = acc;
      hsync();
      if (warp == 0) {
        p += 256;
        const float o = ((p[0] + p[32]) + (p[64] + p[96])) + ((p[128] + p[160]) + (p[192] + p[224]));
        put(O + item * 32 + lane, o, flag);
      }
    }
    if (item + (int)gridDim.x < nitems) csync();   // the item's memory is rewritten
  }
}

// ------------------------------------------------------------------- attention ---
// One 64-token chunk of one KV head per item: head norm + RoPE of the group's query heads
// (and, in the chunk that holds the new position, of the new key; INT8 append of key and
// value), scores, chunk softmax, weighted values. Arithmetic of AttnPrep + AttnSplit
// (attention_core.cuh). K/V rows of earlier tokens are on their way while the words are waited
// for (they were written by earlier steps). Sixteen warps: in the score pass eight of every eighth token for
// each half of the heads, whose queries they hold in registers; an INT8 value becomes a float by a byte permute
// and an addition (in the mantissa of 2^23, less 2^23 + 128: exact) instead of the quarter-rate conversion.
static __device__ __forceinline__ float byte_f32(uint32_t biased, int i) {
  return __uint_as_float(__byte_perm(biased, 0x4B000000u, 0x7540 + i)) - 8388736.0f;
}
template <int GQ>
static __device__ __noinline__ void attn_stage_t(unsigned target, const StepLayer &ly, const unsigned long long *Q, const unsigned long long *K,
                                                 const unsigned long long *V, unsigned flag, int pos, int T) {
  const StepPlan &P = PL;
  constexpr int D = kHeadDim, C = kAttnChunk;
  constexpr int GH = (GQ + 1) / 2;  // query heads per half of the warps
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nKV = P.nKV;
  const int nch = (T + C - 1) / C, nitems = nch * nKV;
  unsigned char *kvs = step_smem + kFbufOff;  // K rows [C][D], then V rows [C][D]
  float *qs = reinterpret_cast<float *>(step_smem + kTOff);  // [GQ][D]
  float *sc = qs + 2048;   // [C][GQ] scores, then exponentials
  float *pw = sc + 512;    // [C][GQ] weights x value scales
  uint16_t *kss = reinterpret_cast<uint16_t *>(pw + 512), *vss = kss + C;
  const int p = pos < P.max_ctx ? pos : P.max_ctx - 1;  // clamp, kernels.cpp:456
  const float scale = 1.0f / sqrtf((float)D);
#pragma unroll 1
  for (int item = (int)blockIdx.x; item < nitems; item += (int)gridDim.x) {
    const int ch = item / nKV, kv = item % nKV, t0 = ch * C;
    const int nt = (T < t0 + C ? T : t0 + C) - t0;
    csync();   // the stage before, or the item before, is done with this memory
    {
      const size_t first = ((size_t)t0 * nKV + kv) * D, rs = (size_t)nKV * D;
#pragma unroll 1
      for (int i = tid; i < 2 * C * (D / 16); i += kCons) {
        const int which = i >> 10, row = (i & 1023) >> 4, pc = i & 15;
        if (row < nt && t0 + row != p) cp_async16(kvs + (size_t)i * 16, (which ? ly.Vc : ly.Kc) + first + row * rs + pc * 16);
      }
      if (tid < 2 * C) {
        const int row = tid & (C - 1);
        if (row < nt && t0 + row != p) (tid < C ? kss : vss)[row] = __ldcg((tid < C ? ly.Ks : ly.Vs) + (size_t)(t0 + row) * nKV + kv);
      }
    }
    if (item == (int)blockIdx.x) await(target);
    // query heads of the group: warp g. New key row: warp GQ, new value row: warp GQ+1.
    if (warp < GQ || ((warp == GQ || warp == GQ + 1) && p >= t0 && p < t0 + nt)) {
      const unsigned long long *src = warp < GQ ? Q + (size_t)(kv * GQ + warp) * 2 * D : (warp == GQ ? K : V) + (size_t)kv * D;
      float x[8];
      take8(x, src + lane, flag);
      if (warp <= GQ) {
        const float *w = warp < GQ ? ly.q_norm : ly.k_norm;
        double ss = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss = fma((double)x[i], (double)x[i], ss);
        ss = warp_tree_sum(ss);
        const float inv = inv_sqrt((float)(ss * (1.0 / D)) + P.eps);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = (x[i] * inv) * (1.0f + __ldg(w + lane + 32 * i));
        if (P.rot / 2 == 32) {
          const float cs = P.Cos[(size_t)pos * P.rot + lane], sn = P.Sin[(size_t)pos * P.rot + lane];
          const float x0 = x[0], x1 = x[1];
          x[0] = x0 * cs - x1 * sn;
          x[1] = x0 * sn + x1 * cs;
        }
      }
      if (warp < GQ) {
#pragma unroll
        for (int i = 0; i < 8; ++i) qs[warp * D + lane + 32 * i] = x[i];
      } else {
        // quantise the new row into the staged chunk, then copy it to the cache
        const bool isk = warp == GQ;
        int8_t *srow = reinterpret_cast<int8_t *>(kvs) + (isk ? 0 : C * D) + (p - t0) * D;
        uint16_t *ssc = (isk ? kss : vss) + (p - t0);
        kv_quant_store(x, lane, srow, ssc);
        __syncwarp();
        int8_t *grow = (isk ? ly.Kc : ly.Vc) + ((size_t)p * nKV + kv) * D;
        reinterpret_cast<uint2 *>(grow)[lane] = reinterpret_cast<const uint2 *>(srow)[lane];
        if (lane == 0) ((isk ? ly.Ks : ly.Vs))[(size_t)p * nKV + kv] = *ssc;
      }
    }
    cp_async_wait();
    csync();
    stamp(20);
    const int g0 = (warp >> 3) * GH;   // this half's first head
    if (g0 < GQ) {
      float q[GH][8];
#pragma unroll
      for (int g = 0; g < GH; ++g) {
        const float4 a = *reinterpret_cast<const float4 *>(qs + (g0 + g) * D + lane * 8), b = *reinterpret_cast<const float4 *>(qs + (g0 + g) * D + lane * 8 + 4);
        q[g][0] = a.x; q[g][1] = a.y; q[g][2] = a.z; q[g][3] = a.w;
        q[g][4] = b.x; q[g][5] = b.y; q[g][6] = b.z; q[g][7] = b.w;
      }
#pragma unroll 2
      for (int tt = warp & 7; tt < nt; tt += 8) {
        const uint2 kw = reinterpret_cast<const uint2 *>(kvs)[tt * (D / 8) + lane];
        const uint32_t b0 = kw.x ^ 0x80808080u, b1 = kw.y ^ 0x80808080u;
        float kf[8], part[GH];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          kf[j] = byte_f32(b0, j);
          kf[4 + j] = byte_f32(b1, j);
        }
#pragma unroll
        for (int g = 0; g < GH; ++g) {
          float acc = 0.0f;
#pragma unroll
          for (int j = 0; j < 8; ++j) acc = fmaf(q[g][j], kf[j], acc);
          part[g] = acc;
        }
        attn_store_scores<GH>(part, lane, sc + tt * GQ + g0, f16_to_f32(kss[tt]), scale);
      }
    }
    csync();
    stamp(22);
    if (warp < GQ) {   // chunk softmax of a head
      const float s0 = lane < nt ? sc[lane * GQ + warp] : -INFINITY, s1 = lane + 32 < nt ? sc[(lane + 32) * GQ + warp] : -INFINITY;
      const float mx = warp_largest(fmaxf(s0, s1));
#pragma unroll 1
      for (int u = 0; u < 2; ++u) {
        const int tt = lane + 32 * u;
        if (tt < nt) {
          const float e = det_expf((u ? s1 : s0) - mx);
          sc[tt * GQ + warp] = e;
          pw[tt * GQ + warp] = e * f16_to_f32(vss[tt]);
        }
      }
      if (lane == 0) P.Pm[(size_t)(kv * GQ + warp) * P.max_chunks + ch] = mx;
    }
    csync();
    stamp(23);
    if (warp == 15 && lane < GQ) {   // the sum of exponentials, in token order
      float se = 0.0f;
#pragma unroll 8
      for (int tt = 0; tt < nt; ++tt) se = se + sc[tt * GQ + lane];
      P.Pse[(size_t)(kv * GQ + lane) * P.max_chunks + ch] = se;
    }
    // weighted values: thread (dim, half) accumulates its dim for the heads of its half
    const int dim = tid & 255;
    float acc[GH];
#pragma unroll
    for (int g = 0; g < GH; ++g) acc[g] = 0.0f;
    const uint8_t *vs = reinterpret_cast<const uint8_t *>(kvs + C * D) + dim;
#pragma unroll 4
    for (int tt = 0; tt < nt; ++tt) {
      const float v = __uint_as_float(0x4B000000u | ((uint32_t)vs[tt * D] ^ 0x80u)) - 8388736.0f;
      if constexpr (GQ == 8) {   // four heads per half: one 16-byte read gives a token's four weights
        const float4 w = *reinterpret_cast<const float4 *>(pw + tt * GQ + g0);
        acc[0] = fmaf(w.x, v, acc[0]);
        acc[1] = fmaf(w.y, v, acc[1]);
        acc[2] = fmaf(w.z, v, acc[2]);
        acc[3] = fmaf(w.w, v, acc[3]);
      } else {
#pragma unroll
        for (int g = 0; g < GH; ++g)
          if (g0 + g < GQ) acc[g] = fmaf(pw[tt * GQ + g0 + g], v, acc[g]);
      }
    }
#pragma unroll
    for (int g = 0; g < GH; ++g)
      if (g0 + g < GQ) P.Pacc[((size_t)(kv * GQ + g0 + g) * P.max_chunks + ch) * D + dim] = acc[g];
    stamp(24);
  }
}
static __device__ __forceinline__ void attn_stage(unsigned target, const StepLayer &ly, const unsigned long long *Q, const unsigned long long *K,
                                                  const unsigned long long *V, unsigned flag, int pos, int T) {
  switch (PL.nQ / PL.nKV) {
    case 1: attn_stage_t<1>(target, ly, Q, K, V, flag, pos, T); break;
    case 2: attn_stage_t<2>(target, ly, Q, K, V, flag, pos, T); break;
    case 4: attn_stage_t<4>(target, ly, Q, K, V, flag, pos, T); break;
    case 6: attn_stage_t<6>(target, ly, Q, K, V, flag, pos, T); break;
    case 8: attn_stage_t<8>(target, ly, Q, K, V, flag, pos, T); break;
    default: break;  // rejected on the host
  }
}

// Ordered merge of the chunk partials, sigmoid gate, quantiser: AttnCombine's arithmetic
// (attention_core.cuh). An item is half a query head, the 128 dims of a quantiser group: thread d < 128 adds
// its dim over the chunks in ascending order, from 64 chunks at a time in shared memory. Its
// words: 32 of four INT8 values, and the scale.
static __device__ __noinline__ void attn_merge(unsigned target, const unsigned long long *Q, unsigned long long *q8, unsigned flag, int T) {
  const StepPlan &P = PL;
  constexpr int D = kHeadDim, C = kAttnChunk;
  float *pa = reinterpret_cast<float *>(step_smem + kFbufOff);   // [64][128] partials
  float *fs = reinterpret_cast<float *>(step_smem + kTOff), *es = fs + 64;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nch = (T + C - 1) / C;
#pragma unroll 1
  for (int it = (int)blockIdx.x; it < 2 * P.nQ; it += (int)gridDim.x) {
    const int h = it >> 1, d0 = (it & 1) * 128;
    const float *pm = P.Pm + (size_t)h * P.max_chunks, *pse = P.Pse + (size_t)h * P.max_chunks;
    const float *pacc = P.Pacc + (size_t)h * P.max_chunks * D + d0;
    const float gate = tid < 128 ? take(Q + (size_t)h * 2 * D + D + d0 + tid, flag) : 0.0f;
    float M = -INFINITY, se = 0.0f, acc = 0.0f;
    const auto fetch = [&](int c0, int nb) {
#pragma unroll 1
      for (int i = tid; i < nb * 32; i += kCons) cp_async16(pa + i * 4, pacc + (size_t)(c0 + (i >> 5)) * D + (i & 31) * 4);
    };
    if (it != (int)blockIdx.x) csync();   // the memory's last readers are done
    fetch(0, nch < 64 ? nch : 64);
#pragma unroll 1
    for (int ch = lane; ch < nch; ch += 32) M = fmaxf(M, __ldcg(pm + ch));
    M = warp_largest(M);
#pragma unroll 1
    for (int c0 = 0; c0 < nch; c0 += 64) {
      const int nb = nch - c0 < 64 ? nch - c0 : 64;
      if (c0) {
        csync();
        fetch(c0, nb);
      }
      if (tid < nb) {
        fs[tid] = det_expf(__ldcg(pm + c0 + tid) - M);
        es[tid] = __ldcg(pse + c0 + tid);
      }
      cp_async_wait();
      csync();
      if (tid < 128) {
#pragma unroll 8
        for (int c = 0; c < nb; ++c) acc = fmaf(pa[c * 128 + tid], fs[c], acc);
      } else if (tid == 128) {
#pragma unroll 8
        for (int c = 0; c < nb; ++c) se = fmaf(es[c], fs[c], se);
      }
    }
    if (tid == 128) SH->wmax[8] = se;
    csync();
    float y = 0.0f;
    if (tid < 128) {
      y = over_exp(acc / SH->wmax[8], -gate);
      const float m = warp_absmax(y);
      if (lane == 0) SH->wmax[warp] = m;
    }
    csync();
    if (tid < 128) {
      const float m = fmaxf(fmaxf(SH->wmax[0], SH->wmax[1]), fmaxf(SH->wmax[2], SH->wmax[3]));
      float s = m / 127.0f;
      if (s == 0.0f) s = 1.0f;
      uint32_t w = (uint32_t)(quant_round(y, s) & 0xFF);
      w |= __shfl_down_sync(kFull, w, 1) << 8;
      w |= __shfl_down_sync(kFull, w, 2) << 16;
      if ((tid & 3) == 0) put(q8 + it * 32 + (tid >> 2), __uint_as_float(w), flag);
      if (tid == 0) put(q8 + P.nQ * 64 + it, s, flag);
    }
  }
  // the merged vector into the staged form
  const int K = P.nQ * D, G = K >> 7;
  unsigned char *act = step_smem + kActOff;
  uint32_t *xw = reinterpret_cast<uint32_t *>(act);
  arrive<false>();
  await(target);
  gather(pa, q8, P.nQ * 66, flag);
  csync();
  stamp(1);
#pragma unroll 1
  for (int pc = tid; pc < K / 8; pc += kCons) {
    const uint2 v = reinterpret_cast<const uint2 *>(pa)[pc];
    const int g = pc >> 4, i = pc & 15;
    uint32_t *dst = xw + ((((i >> 1) * G + g) << 2) + ((i & 1) << 1));
    dst[0] = __byte_perm(v.x, v.y, 0x6420);
    dst[1] = __byte_perm(v.x, v.y, 0x7531);
  }
  if (tid < G) reinterpret_cast<float *>(act + K)[tid] = pa[P.nQ * 64 + tid];
  csync();
}

// ------------------------------------------------------------------- MoE stages ---
static __device__ __forceinline__ uint32_t gateup_stage(uint32_t tile, unsigned long long *out, unsigned flag) {
  const StepPlan &P = PL;
  const int H = P.H, lgI = __ffs(P.I) - 1, lg = 31 - __clz(H >> 7);
  const int lo = SH->rng[kRngGateUp].x, hi = SH->rng[kRngGateUp].y, np = hi - lo;
  const float *T = reinterpret_cast<const float *>(step_smem + kTOff);
  csync();   // the candidates of the selection lie where the terms go
  tile = dot_tiles(tile, lg, H, 2 * np, 0.0f);
  // the producer streams, slot by slot, the slot's gate rows and then its up rows: the pair row
  // lo + r of slot s (rows a .. a + n - 1 of the share belong to it) has its gate term at
  // 2 (a - lo) + i and its up term n rows later
#pragma unroll 1
  for (int r = threadIdx.x; r < np; r += kCons) {
    const int s = (lo + r) >> lgI;
    const int a = lo > s * P.I ? lo : s * P.I, b = hi < (s + 1) * P.I ? hi : (s + 1) * P.I;
    const int n = b - a, i = lo + r - a, fg = 2 * (a - lo) + i;
    const float g = row_terms(T, fg, lg), u = row_terms(T, fg + n, lg);
    put(out + lo + r, over_exp(g, -g) * u, flag);
  }
  return tile;
}

// Output row n: residual + sum over the slots in rank order of weight x product. One thread a (slot,
// row) adds the row's group terms, then one a row adds the slots.
static __device__ __forceinline__ uint32_t down_stage(unsigned target, uint32_t tile, const unsigned long long *in, unsigned long long *out, unsigned flag,
                                                      float res, int L) {
  const StepPlan &P = PL;
  const int H = P.H, I = P.I, lg = 31 - __clz(I >> 7), warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int lo = SH->rng[kRngDown].x, nr = SH->rng[kRngDown].y - lo, n = P.slots * nr;
  float *xs = reinterpret_cast<float *>(step_smem + kFbufOff), *ts = xs + 4096;
  const float *T = reinterpret_cast<const float *>(step_smem + kTOff);
  unsigned char *act = step_smem + kActOff;
  await(target);
  gather(xs, in, P.slots * I, flag);
  csync();
  stamp(1);
  if ((int)blockIdx.x == 0 && tid <= P.topk) {
    const StepShared *sh = SH;
    P.SelIdx[tid] = sh->sel_idx[tid];
    P.SelW[tid] = sh->sel_w[tid];
    if (tid == 0) *P.NearGap = sh->gap;
    if (P.routed) {
      P.routed[(size_t)L * (P.topk + 1) + tid] = sh->sel_idx[tid];
      if (tid == 0) P.near_gap[L] = sh->gap;
    }
  }
#pragma unroll 1
  for (int gi = warp; gi < P.slots << lg; gi += 16)
    stage_group(reinterpret_cast<uint32_t *>(act), reinterpret_cast<float *>(act + P.slots * I), 1 << lg, gi >> lg, gi & ((1 << lg) - 1),
                quant_group(*reinterpret_cast<const float4 *>(xs + gi * 128 + lane * 4)));
  csync();
  stamp(2);
  tile = dot_tiles(tile, lg, P.slots * I, n, SH->down_recip);
#pragma unroll 1
  for (int f = tid; f < n; f += kCons) ts[f] = SH->sel_w[(int)(((float)f + 0.5f) * SH->down_recip)] * row_terms(T, f, lg);
  csync();
  if (tid < nr) {
    float acc = 0.0f;
#pragma unroll 4
    for (int s = 0; s < P.slots; ++s) acc = acc + ts[s * nr + tid];
    const float x = res + acc;
    put(out + lo + tid, x, flag);
    if (L + 1 == P.layers) P.X[lo + tid] = x;
    if (P.layer_out) P.layer_out[(size_t)L * H + lo + tid] = x;
  }
  stamp(3);
  return tile;
}

// LM head in sub-blocks of 16 tiles (t[][] holds 256 rows of K = 2048), running argmax per thread.
static __device__ __noinline__ uint32_t lm_head_stage(uint32_t tile, float &bv, int &bi) {
  const StepPlan &P = PL;
  const int K = P.H, lg = 31 - __clz(K >> 7);
  const int lo = SH->rng[kRngHead].x, hi = SH->rng[kRngHead].y;
  const float *T = reinterpret_cast<const float *>(step_smem + kTOff);
  const int sub = kTCap >> lg;  // rows whose terms fit t[][]: a whole, even number of tiles
#pragma unroll 1
  for (int base = 0; base < hi - lo; base += sub) {
    const int nrows = (hi - lo) - base < sub ? (hi - lo) - base : sub;
    tile = dot_tiles(tile, lg, K, nrows, 0.0f);
#pragma unroll 1
    for (int r = threadIdx.x; r < nrows; r += kCons) {
      const float v = row_terms(T, r, lg);
      const int n = lo + base + r;
      P.Logits[n] = v;
      argmax_merge(bv, bi, v, n);
    }
    csync();
  }
  return tile;
}

// Block-wide first-max-wins argmax over the consumer threads; result valid in thread 0.
static __device__ __noinline__ void cons_argmax(float &bv, int &bi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int off = 16; off > 0; off >>= 1)
    argmax_merge(bv, bi, __shfl_xor_sync(kFull, bv, off), __shfl_xor_sync(kFull, bi, off));
  if (lane == 0) {
    SH->av[warp] = bv;
    SH->ai[warp] = bi;
  }
  csync();
  if (warp == 0) {
    bv = lane < 16 ? SH->av[lane] : -INFINITY;
    bi = lane < 16 ? SH->ai[lane] : 0x7FFFFFFF;
#pragma unroll 1
    for (int off = 16; off > 0; off >>= 1)
      argmax_merge(bv, bi, __shfl_xor_sync(kFull, bv, off), __shfl_xor_sync(kFull, bi, off));
  }
}

static __device__ __forceinline__ void consumer_main(int mode) {
  const StepPlan &P = PL;
  StepShared *sh = SH;
  const int H = P.H, tid = threadIdx.x;
  uint32_t tile = 0;   // running index of the next ring tile to consume
  const unsigned seq = __ldcg(P.sync + STEP_LAUNCHES), bar0 = __ldcg(P.sync + STEP_BAR_BASE);
  unsigned bar = bar0;   // the count of arrivals when all blocks have ended the last stage
  const int token = __ldcg(P.ctrl + CTRL_TOKEN), pos = __ldcg(P.ctrl + CTRL_POS);
  int T = __ldcg(P.ctrl + CTRL_LEN);
  if (T > P.max_ctx) T = P.max_ctx;
  const int tok = token < 0 ? 0 : (token >= P.vocab ? P.vocab - 1 : token);
  unsigned flag = seq * (unsigned)P.layers;
  float res;

#pragma unroll 1
  for (int L = 0; L < P.layers; ++L) {
    // the layer's record into shared memory (the previous layer's is no longer read: every
    // consumer has passed a block barrier behind its last use)
    if (tid < (int)(sizeof(StepLayer) / 16))
      reinterpret_cast<uint4 *>(&sh->ly)[tid] = __ldg(reinterpret_cast<const uint4 *>(P.L + L) + tid);
    csync();
    const StepLayer &ly = sh->ly;
    const bool lin = ly.type == 0;
    // words of this layer; the input's are the layer before's
    unsigned long long *W = P.words + (L & 1 ? P.words_set : 0), *Wx = P.words + (L & 1 ? 0 : P.words_set);
    // the layer's table of experts into L2, two lines a block
    {
      const int line = (int)blockIdx.x * 2 + tid;
      if (tid < 2 && line * 128 < (P.E + 1) * (int)sizeof(ExpertW))
        prefetch_l2(reinterpret_cast<const unsigned char *>(ly.experts) + line * 128);
    }
    // ---- stage 1: input norm + quantiser, first projections ----
    res = norm_quant(bar, Wx + P.wX, flag, L == 0 ? P.emb + (size_t)tok * H : nullptr, ly.in_norm, H, sh->rng[kRngOut + ly.type]);
    ++flag;
    tile = gemv_stage_run(tile, &ly.m[0], lin ? 4 : 3, H, sh->rng[kRngIn + ly.type], flag, 0.0f);
    bar += gridDim.x;
    arrive<false>();
    if (lin) {
      // ---- stage 2: gated delta rule; stage 3: gated norm, out_proj + residual ----
      deltanet_stage(bar, ly, W + P.wM, W + P.wB, W + P.wG, W + P.wO, flag);
      bar += gridDim.x;
      arrive<false>();
      gated_norm_quant(bar, W + P.wO, W + P.wZ, flag, ly.lin_norm, P.nV);
    } else {
      attn_stage(bar, ly, W + P.wQ, W + P.wK, W + P.wV, flag, pos, T);
      bar += gridDim.x;
      arrive<true>();   // the chunk partials are plain stores
      await(bar);
      stamp(1);
      bar += gridDim.x;
      attn_merge(bar, W + P.wQ, W + P.w8, flag, T);
    }
    stamp(2);
    tile = gemv_stage_run(tile, &ly.m[4], 1, lin ? P.nV * 128 : P.nQ * 256, sh->rng[kRngOut + ly.type], flag, res);
    bar += gridDim.x;
    arrive<false>();
    // ---- stage 4: post norm + quantiser (kept staged for the experts), router logits ----
    res = norm_quant(bar, W + P.wT, flag, nullptr, ly.post_norm, H, sh->rng[kRngDown]);
    tile = router_stage(tile, W + P.wR, flag, H);
    stamp(3);
    bar += gridDim.x;
    arrive<false>();
    // ---- stage 5: selection, expert gate/up ----
    router_select_cons(bar, W + P.wR, flag, ly.experts, P.E, P.topk, ly.shared_gate != nullptr);
    tile = gateup_stage(tile, W + P.wA, flag);
    stamp(3);
    bar += gridDim.x;
    arrive<false>();
    // ---- stage 6: expert down, combine, residual ----
    tile = down_stage(bar, tile, W + P.wA, W + P.wX, flag, res, L);
    bar += gridDim.x;
    arrive<false>();
  }

  const bool lead = (int)blockIdx.x == 0;
  if (mode != 0) {
    // ---- tail: final norm, LM head, first-max-wins argmax ----
    norm_quant(bar, P.words + (P.layers & 1 ? 0 : P.words_set) + P.wX, flag, nullptr, P.final_norm, H, make_int2(0, 0));
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
    tile = lm_head_stage(tile, bv, bi);
    cons_argmax(bv, bi);
    if (tid == 0) {
      P.PV[(int)blockIdx.x] = bv;
      P.PI[(int)blockIdx.x] = bi;
    }
    bar += gridDim.x;
    arrive<true>();
    if (lead) {
      await(bar);
      bv = -INFINITY;
      bi = 0x7FFFFFFF;
      for (int i = tid; i < (int)gridDim.x; i += kCons) argmax_merge(bv, bi, __ldcg(P.PV + i), __ldcg(P.PI + i));
      csync();
      cons_argmax(bv, bi);
      if (tid == 0) {
        P.out_tok[0] = bi;
        if (P.history && P.history_cap > 0) P.history[pos % P.history_cap] = bi;
        P.ctrl[CTRL_SELECTED] = bi;
        P.ctrl[CTRL_TOKEN] = bi;
      }
    }
  } else if (lead && tid == 0) {
    // prompt step: no logits; move on to the next prompt id
    if (pos + 1 < P.max_ctx) P.ctrl[CTRL_TOKEN] = P.ids[pos + 1];
    P.ctrl[CTRL_SELECTED] = -1;
  }
  // The control block and the launch's numbers for the next launch. Every block has read them: block 0 is
  // here behind words that depend on every block's rows of the last layer.
  if (lead && tid == 0) {
    P.ctrl[CTRL_POS] = pos + 1;
    P.ctrl[CTRL_LEN] = P.ctrl[CTRL_LEN] + 1;
    P.sync[STEP_BAR_BASE] = bar;
    P.sync[STEP_LAUNCHES] = seq + 1u;
  }
}
};

template <bool kClock>
__device__ __forceinline__ void decode_step(const DecodeStepArgs &args) {
  using B = Step<kClock>;
  StepShared *sh = SH;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kNT; ++i) {
      mbar_init(&sh->full[i], 1);
      mbar_init(&sh->empty[i], kCons / 64);  // one arrival per warp of the half that consumes the tile
    }
    mbar_init(&sh->sel_bar, 1);
    sh->fail = 0;
    sh->nstamp[0] = 0;
    sh->nstamp[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < sizeof(StepPlan) / 16)
    reinterpret_cast<uint4 *>(&sh->plan)[threadIdx.x] = __ldg(reinterpret_cast<const uint4 *>(args.plan) + threadIdx.x);
  __syncthreads();
  if (threadIdx.x < kRngCount) B::deal_all((int)threadIdx.x);
  __syncthreads();
  if (*(volatile int *)PL.error != 0) return;  // a previous launch failed: stay out
  if (threadIdx.x >= kCons) {
    const uint32_t issued = B::producer_main(args.mode);
    // Nothing may still be landing in this block's shared memory when it retires: every slot
    // owner waits (bounded) for the last tile it issued. In a run without faults the consumers
    // have waited for all of them already.
    const uint32_t lane = threadIdx.x & 31;
    if (lane < (uint32_t)kNT && issued > lane) {
      const uint32_t t = issued - 1u - ((issued - 1u - lane) % kNT);  // latest tile issued into slot `lane`
      const long long t0 = clock64();
      while (!mbar_try(&sh->full[lane], (t / kNT) & 1u))
        if (clock64() - t0 > kWaitCycles) break;
    }
    return;
  }
  B::consumer_main(args.mode);
}
__global__ void __launch_bounds__(kStepThreads, 1) DecodeStep(const DecodeStepArgs args) { decode_step<false>(args); }
__global__ void __launch_bounds__(kStepThreads, 1) DecodeStepClock(const DecodeStepArgs args) { decode_step<true>(args); }

// quant_group() alone, a warp a group: its bound is checked with this.
struct StepQuantGroupsArgs {
  const float *X;   // [groups][128]
  int8_t *Q;
  float *S;
  int32_t groups;
};
__global__ void __launch_bounds__(128) StepQuantGroups(const StepQuantGroupsArgs a) {
  const int g = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (g >= a.groups) return;
  const uint2 q = Step<false>::quant_group(reinterpret_cast<const float4 *>(a.X + (size_t)g * 128)[lane]);
  reinterpret_cast<uint32_t *>(a.Q + (size_t)g * 128)[lane] = q.x;
  if (lane == 0) a.S[g] = __uint_as_float(q.y);
}

static uint32_t step_smem_fn(const void *) { return (uint32_t)kStepSmemBytes; }

#define F(f) AINFER_ARG(DecodeStepArgs, f)
AINFER_REGISTER_COOP(DecodeStep, DecodeStepArgs, kStepThreads, 0, 0, step_smem_fn, F(plan), F(mode));
AINFER_REGISTER_COOP(DecodeStepClock, DecodeStepArgs, kStepThreads, 0, 0, step_smem_fn, F(plan), F(mode));
#undef F
#define F(f) AINFER_ARG(StepQuantGroupsArgs, f)
AINFER_REGISTER(StepQuantGroups, StepQuantGroupsArgs, 128, 4, 0, nullptr, F(X), F(Q), F(S), F(groups));
#undef F

}  // namespace ainfer
