// Device-side token sampler with the semantics of the reference's host sampler
// (tools/sample/sampler.h:16-62 parameters, :27-45 repetition penalty, :47-56 xorshift64* stream,
// :60-158 sample_token): greedy first-max-wins for temp <= 0; otherwise softmax in double with the
// maximum subtracted, top-k (k most probable, ties to the lower index), top-p (shortest prefix of
// the sorted distribution whose mass reaches p, ties to the lower index), renormalisation after
// each filter, and an inverse-CDF draw in index order from the same 53-bit uniform stream. The
// logits never leave the device: 4 bytes come back instead of 4 V.
//
// The row is cut into one contiguous run of tokens per thread and lies in shared memory (a thread's j-th
// token at [j][thread]: no bank conflicts), over a cluster of eight blocks (SampleTokenCluster, the
// session's form: 8192 threads hold a vocabulary of 32000 with four tokens each) or one block
// (SampleToken); vocabularies that do not fit there stay in `Work`. Selection by rank is a radix select
// over the probabilities' bit patterns, most probable first: a block counts its tokens of a digit's
// 2048 bins, adds the bins that are not empty to the first block's (32-bit counts; for top-p also the
// mass as a 62-bit fixed-point integer: integer sums do not depend on the order of the additions, so
// the cut is the same on every run), which scans them and tells the others the chosen bin. The first
// digit has 32 bins per factor of two, so that a second one usually meets a handful of tokens, and the
// select ends as soon as the bin is kept whole. Other sums are tree sums, not the host's index-order
// sums, so a draw that lands within rounding of a CDF step may pick the neighbouring token; everything
// else (support of top-k / top-p, tie rules, the stream of uniforms) is identical.
//
// Bound by latency: reductions and two barriers of the cluster per digit. A form with one block, eight
// passes of eight bits over a row in global memory and one thread that walked the 256 bins took
// 969 us at 32000 tokens (top-k 40, top-p 0.95); a step and a draw together went from 1102 to 196 us.
#include "tail_core.cuh"

namespace ainfer {

struct SampleTokenArgs {
  const float *Logits;    // [V]
  const int32_t *Seen;    // [nseen] ids for the repetition penalty (may be null when nseen == 0)
  double *Work;           // [V] scratch: probabilities
  unsigned char *Mark;    // [V] scratch
  unsigned long long *Rng;// [1] xorshift64* state, advanced by one draw when temp > 0
  int32_t *OutT;          // [1] selected token
  float *Probs;           // optional [V]: the final distribution
  int32_t *Ctrl;          // optional control block: {token, position + 1, length + 1, token}
  int32_t V, nseen;
  float temp;
  int32_t top_k;
  float top_p, rep_penalty;
};

constexpr int kSampThreads = 1024, kSampBins = 2048, kSampCluster = 8;
constexpr double kFix = 4611686018427387904.0;   // 2^62
constexpr uint32_t kSampRowBytes = 160 * 1024;   // of the row in shared memory, at most

// What the first block tells the others about a digit, and what follows from it.
struct SampPick {
  unsigned long long lo;     // probabilities are keyed by their bits' distance from 1.0's: smaller = more probable
  unsigned long long end;    // final: keys below it are kept
  unsigned long long need;   // top-k: how many of the bin's tokens are still wanted; final with ties: how many of those with key `lo`
  unsigned long long cum;    // top-p: mass before the bin
  unsigned long long shift;  // of the next digit
  unsigned long long state;  // 0: another digit, 1: final, 2: final with ties at `lo`, 3: everything is kept
};
struct SampShared {
  unsigned int hist[kSampBins], all[kSampBins];               // this block's counts; (first block) the cluster's
  unsigned long long mass[kSampBins], all_mass[kSampBins];    // the same in units of 2^-62
  unsigned long long scan_c[33], scan_m[33];
  double scan_d[33], slot_d[4][kSampCluster];                 // one value of every block: softmax sum, totals after the filters, totals of the draw
  unsigned long long slot_u[2][kSampCluster];                 // ties per block, by filter
  float slot_v[kSampCluster], sv[32];
  int slot_i[kSampCluster], si[32];
  SampPick pick;
  int chosen;
};

template <int CL>
__device__ __forceinline__ void samp_barrier() {
  if constexpr (CL == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
// The address of p in another block of the cluster (p itself in a launch without one).
template <int CL, typename T>
__device__ __forceinline__ T *samp_peer(T *p, uint32_t rank) {
  if constexpr (CL == 1) {
    return p;
  } else {
    unsigned long long q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(reinterpret_cast<unsigned long long>(p)), "r"(rank));
    return reinterpret_cast<T *>(q);
  }
}
// Exclusive scan over the block's threads; the block's total in *tot. sh: 33 values, free again after the next barrier.
template <typename T>
__device__ __forceinline__ T samp_scan(T v, T *sh, T *tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T y = __shfl_up_sync(kFull, x, off);
    if (lane >= off) x += y;
  }
  __syncthreads();
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const T mine = sh[lane];
    T z = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const T y = __shfl_up_sync(kFull, z, off);
      if (lane >= off) z += y;
    }
    const T before = __shfl_up_sync(kFull, z, 1);
    sh[lane] = lane ? before : T(0);
    if (lane == 31) sh[32] = z;
  }
  __syncthreads();
  *tot = sh[32];
  const T in_warp = __shfl_up_sync(kFull, x, 1);
  return sh[warp] + (lane ? in_warp : T(0));
}
// Sum over the cluster's threads, the same in every thread.
template <int CL>
__device__ __forceinline__ double samp_sum(double v, SampShared *s, int slot, uint32_t rank) {
  double tot;
  samp_scan<double>(v, s->scan_d, &tot);
  if (threadIdx.x < CL) *samp_peer<CL>(&s->slot_d[slot][rank], threadIdx.x) = tot;
  samp_barrier<CL>();
  double t = 0.0;
#pragma unroll
  for (int b = 0; b < CL; ++b) t += s->slot_d[slot][b];
  return t;
}
__device__ __forceinline__ unsigned long long samp_key(double p) { return 0x3FF0000000000000ull - (unsigned long long)__double_as_longlong(p); }

// First block: the bin in which the rank or the mass falls, from the cluster's counts (cleared on the way).
__device__ __forceinline__ void samp_pick(SampShared *s, bool by_count, bool first, float top_p) {
  const int b0 = 2 * threadIdx.x;
  const unsigned int c0 = s->all[b0], c1 = s->all[b0 + 1];
  const unsigned long long m0 = by_count ? 0ull : s->all_mass[b0], m1 = by_count ? 0ull : s->all_mass[b0 + 1];
  s->all[b0] = s->all[b0 + 1] = 0u;
  s->all_mass[b0] = s->all_mass[b0 + 1] = 0ull;
  const SampPick p = s->pick;
  const unsigned long long want = by_count ? p.need : (unsigned long long)((double)top_p * kFix);
  unsigned long long tot;
  unsigned long long before = by_count ? samp_scan<unsigned long long>((unsigned long long)c0 + c1, s->scan_c, &tot)
                                       : p.cum + samp_scan<unsigned long long>(m0 + m1, s->scan_m, &tot);
  const unsigned long long reached = by_count ? tot : p.cum + tot;
  // (every thread has read the old pick before the scan's barriers)
  if (reached < want) {   // rounding: the whole distribution does not reach top_p
    if (threadIdx.x == 0) s->pick.state = 3;
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const unsigned int c = q ? c1 : c0;
    const unsigned long long step = by_count ? (unsigned long long)c : (q ? m1 : m0), prev = before;
    before += step;
    // the first bin that reaches it; a bin without tokens never does
    const bool hit = by_count ? prev < want && before >= want : c != 0u && before >= want && (prev < want || (want == 0ull && prev == 0ull));
    if (!hit) continue;
    const int b = b0 + q;
    SampPick n;
    const bool clamp = first && b == kSampBins - 1;   // everything below 2^-64 in one bin: continue from there with wide digits
    n.lo = p.lo + ((unsigned long long)b << p.shift);
    n.end = n.lo + (1ull << p.shift);
    n.need = by_count ? want - prev : 0ull;
    n.cum = by_count ? 0ull : prev;
    n.shift = clamp ? 52ull : p.shift > 11 ? p.shift - 11 : 0ull;
    n.state = 0;
    if (clamp) n.end = ~0ull;
    if (by_count ? (unsigned long long)c == n.need : c == 1u) {
      n.state = 1;                                    // the bin is kept whole
    } else if (p.shift == 0) {
      n.state = 2;                                    // equal probabilities: as many of them as it takes, lower tokens first
      if (!by_count) {
        const double pt = __longlong_as_double((long long)(0x3FF0000000000000ull - n.lo));
        const double rest = (double)top_p - (double)prev / kFix;
        long long k = pt > 0.0 ? (long long)ceil(rest / pt) : 1;
        n.need = k < 1 ? 1ull : (unsigned long long)k;
      }
      n.end = n.lo;
    }
    s->pick = n;
  }
}

template <int CL>
__device__ __forceinline__ void sample_token(const SampleTokenArgs &a) {
  extern __shared__ __align__(16) unsigned char samp_smem[];
  SampShared *s = reinterpret_cast<SampShared *>(samp_smem);
  uint32_t rank = 0;
  if constexpr (CL > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int tid = threadIdx.x, V = a.V;
  const int chunk = (V + kSampThreads * CL - 1) / (kSampThreads * CL);
  const bool shared_row = (uint32_t)chunk * kSampThreads * 8u <= kSampRowBytes;
  const int lo = min(((int)rank * kSampThreads + tid) * chunk, V), n = min(chunk, V - lo);
  double *row = shared_row ? reinterpret_cast<double *>(samp_smem + sizeof(SampShared)) + tid : a.Work + lo;
  const int step = shared_row ? kSampThreads : 1;
  for (int b = tid; b < kSampBins; b += kSampThreads) { s->hist[b] = s->all[b] = 0u; s->mass[b] = s->all_mass[b] = 0ull; }
  if (tid == 0) s->chosen = V - 1;
  // ---- repetition penalty: every seen id once, by the block that holds the token ----
  const bool penal = a.rep_penalty > 1.0f && a.nseen > 0;
  if (penal) {
    const int first = min((int)rank * kSampThreads * chunk, V), last = min(first + kSampThreads * chunk, V);
    for (int i = first + tid; i < last; i += kSampThreads) a.Mark[i] = 0;
    __syncthreads();
    for (int i = tid; i < a.nseen; i += kSampThreads) {
      const int id = a.Seen[i];
      if (id >= first && id < last) a.Mark[id] = 1;
    }
    __syncthreads();
  }
  // ---- maximum (and the greedy answer) ----
  float bv = -INFINITY;
  int bi = 0x7FFFFFFF;
  for (int j = 0; j < n; ++j) {
    float l = a.Logits[lo + j];
    if (penal && a.Mark[lo + j]) l = l > 0 ? l / a.rep_penalty : l * a.rep_penalty;
    row[j * step] = (double)l;
    argmax_merge(bv, bi, l, lo + j);
  }
  block_argmax(bv, bi, s->sv, s->si);
  if (tid == 0) { s->sv[0] = bv; s->si[0] = bi; }
  __syncthreads();
  if constexpr (CL > 1) samp_barrier<CL>();   // every block of the cluster runs: its shared memory may be written
  if (tid < CL) {
    *samp_peer<CL>(&s->slot_v[rank], tid) = s->sv[0];
    *samp_peer<CL>(&s->slot_i[rank], tid) = s->si[0];
  }
  samp_barrier<CL>();
  float top = s->slot_v[0];
  int chosen = s->slot_i[0];
#pragma unroll
  for (int b = 1; b < CL; ++b) argmax_merge(top, chosen, s->slot_v[b], s->slot_i[b]);
  unsigned long long rng_next = 0;
  if (a.temp <= 0.0f) {
    if (a.Probs) for (int j = 0; j < n; ++j) a.Probs[lo + j] = lo + j == chosen ? 1.0f : 0.0f;
  } else {
    // ---- softmax in double ----
    double part = 0.0;
    for (int j = 0; j < n; ++j) {
      const double p = exp((row[j * step] - (double)top) / (double)a.temp);
      row[j * step] = p;
      part += p;
    }
    const double z = samp_sum<CL>(part, s, 0, rank);
    for (int j = 0; j < n; ++j) row[j * step] = row[j * step] / z;
    const bool valid = z > 0.0 && z < (double)INFINITY;   // else (an infinite or undefined logit): no order to filter by
    // ---- filters: keep the top_k most probable, then the shortest prefix of mass >= top_p ----
    for (int filter = 0; filter < 2 && valid; ++filter) {
      const bool by_count = filter == 0;
      if (by_count ? !(a.top_k > 0 && a.top_k < V) : !(a.top_p < 1.0f)) continue;
      __syncthreads();
      if (tid == 0) s->pick = SampPick{0ull, ~0ull, by_count ? (unsigned long long)a.top_k : 0ull, 0ull, 47ull, 0ull};
      __syncthreads();
      for (bool first = true;; first = false) {
        const SampPick p = s->pick;
        for (int j = 0; j < n; ++j) {
          const double v = row[j * step];
          const unsigned long long d = samp_key(v);
          if (d < p.lo || d >= p.end) continue;
          const unsigned long long at = (d - p.lo) >> p.shift;
          const int b = at < (unsigned long long)(kSampBins - 1) ? (int)at : kSampBins - 1;
          atomicAdd(&s->hist[b], 1u);
          if (!by_count) atomicAdd(&s->mass[b], (unsigned long long)(v * kFix));
        }
        __syncthreads();
        for (int b = tid; b < kSampBins; b += kSampThreads) {
          const unsigned int c = s->hist[b];
          if (!c) continue;
          s->hist[b] = 0u;
          atomicAdd(samp_peer<CL>(&s->all[b], 0), c);
          if (!by_count) { atomicAdd(samp_peer<CL>(&s->all_mass[b], 0), s->mass[b]); s->mass[b] = 0ull; }
        }
        samp_barrier<CL>();
        if (rank == 0) {
          samp_pick(s, by_count, first, a.top_p);
          __syncthreads();
          if (CL > 1 && tid >= 8 && tid < 8 * CL && (tid & 7) < 6)
            reinterpret_cast<unsigned long long *>(samp_peer<CL>(&s->pick, tid >> 3))[tid & 7] = reinterpret_cast<unsigned long long *>(&s->pick)[tid & 7];
        }
        samp_barrier<CL>();
        if (s->pick.state) break;
      }
      const SampPick p = s->pick;
      unsigned long long before = 0;
      if (p.state == 2) {   // tokens of equal probability are kept in index order
        unsigned long long mine = 0, tot;
        for (int j = 0; j < n; ++j) mine += samp_key(row[j * step]) == p.lo;
        before = samp_scan<unsigned long long>(mine, s->scan_c, &tot);
        if (tid < CL) *samp_peer<CL>(&s->slot_u[filter][rank], tid) = tot;
        samp_barrier<CL>();
        for (uint32_t b = 0; b < rank; ++b) before += s->slot_u[filter][b];
      }
      double part2 = 0.0;
      for (int j = 0; j < n; ++j) {
        const double v = row[j * step];
        const unsigned long long d = samp_key(v);
        bool keep = p.state == 3 || d < p.end;
        if (p.state == 2 && d == p.lo) {
          if (before < p.need) keep = true;
          ++before;
        }
        if (keep) part2 += v; else row[j * step] = 0.0;
      }
      const double total = samp_sum<CL>(part2, s, 1 + filter, rank);
      for (int j = 0; j < n; ++j) row[j * step] = row[j * step] / total;
    }
    // ---- inverse-CDF draw in index order ----
    unsigned long long x = *a.Rng;
    x ^= x >> 12; x ^= x << 25; x ^= x >> 27;
    rng_next = x;
    const double u = (double)((x * 2685821657736338717ull) >> 11) * (1.0 / 9007199254740992.0);
    double part3 = 0.0, tot;
    for (int j = 0; j < n; ++j) part3 += row[j * step];
    double acc = samp_scan<double>(part3, s->scan_d, &tot);
    if (tid < CL) *samp_peer<CL>(&s->slot_d[3][rank], tid) = tot;
    samp_barrier<CL>();
    double base = 0.0;
    for (uint32_t b = 0; b < rank; ++b) base += s->slot_d[3][b];
    acc += base;
    for (int j = 0; j < n; ++j) {
      acc += row[j * step];
      if (u < acc) { atomicMin(samp_peer<CL>(&s->chosen, 0), lo + j); break; }
    }
    if (a.Probs) for (int j = 0; j < n; ++j) a.Probs[lo + j] = (float)row[j * step];
  }
  samp_barrier<CL>();   // also: no block leaves while others reach into its shared memory or read *Rng
  if (rank == 0 && tid == 0) {
    if (a.temp > 0.0f) { *a.Rng = rng_next; chosen = s->chosen; }
    a.OutT[0] = chosen;
    if (a.Ctrl) {
      a.Ctrl[CTRL_SELECTED] = chosen;
      a.Ctrl[CTRL_TOKEN] = chosen;
      a.Ctrl[CTRL_POS] = a.Ctrl[CTRL_POS] + 1;
      a.Ctrl[CTRL_LEN] = a.Ctrl[CTRL_LEN] + 1;
    }
  }
}
__global__ void __launch_bounds__(kSampThreads) SampleToken(const SampleTokenArgs a) { sample_token<1>(a); }
__global__ void __cluster_dims__(kSampCluster, 1, 1) __launch_bounds__(kSampThreads) SampleTokenCluster(const SampleTokenArgs a) {
  sample_token<kSampCluster>(a);
}
template <int CL>
static uint32_t sample_smem(const void *args) {
  const int V = ((const SampleTokenArgs *)args)->V, per = kSampThreads * CL;
  const size_t row = (size_t)((V + per - 1) / per) * kSampThreads * 8;
  return (uint32_t)(sizeof(SampShared) + (row <= kSampRowBytes ? row : 0));
}

#define F(f) AINFER_ARG(SampleTokenArgs, f)
#define SAMPLE_FIELDS                                                                                                                            \
  F(Logits), F(Seen), F(Work), F(Mark), F(Rng), F(OutT), F(Probs), F(Ctrl), F(V), F(nseen), F(temp), F(top_k), F(top_p), F(rep_penalty)
AINFER_REGISTER(SampleToken, SampleTokenArgs, kSampThreads, 0, 0, sample_smem<1>, SAMPLE_FIELDS);
AINFER_REGISTER(SampleTokenCluster, SampleTokenArgs, kSampThreads, kSampCluster, 0, sample_smem<kSampCluster>, SAMPLE_FIELDS);
#undef SAMPLE_FIELDS
#undef F

}  // namespace ainfer
