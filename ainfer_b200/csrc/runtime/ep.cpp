// Expert-parallel mixture-of-experts block for a decode batch (the one place the decode path
// shards across GPUs). Experts are split evenly over the ranks (contiguous ids, E / R per rank);
// the router and the shared expert are replicated; rank r owns batch rows [r * B / R, (r + 1) * B / R).
// Per layer, on the device's stream:
//   A  owner:   post-attention RMSNorm + quantiser, router logits, top-k, dispatch plan, permute
//      exchange of the dispatch buffer (one fixed-size slot per peer; NCCL send/recv in one group)
//   B  experts: group received items by expert, gather, grouped tensor-core GEMM gate/up,
//               SiLU-multiply + quantiser, grouped GEMM down, un-permute into the return buffer;
//               the shared expert of the owned rows is one more problem of the same launches
//      exchange of the return buffer
//   C  owner:   slot-ordered combine with the residual
// Every piece keeps the single-token kernels' arithmetic, so each token's row is bit-identical
// to the one-GPU decode kernels' whatever the batch and the number of ranks. The reference
// decodes one token on one device (tools/decode/decode_l0.cpp:666-674 is its dense MLP) and has
// no counterpart for the exchange.
//
// NCCL is bound at run time (dlopen of libnccl.so.2, the library the process already uses if any);
// a world of one rank needs none and groups its own rows in place, without dispatch and return buffers.
#include "ep.h"

#include <dlfcn.h>

#include <cstring>

namespace ainfer {

namespace {

// ---- the few NCCL entry points used, declared here so that the runtime builds without CUDA headers ----
struct NcclUniqueId { char internal[128]; };
typedef struct ncclComm *NcclComm;
struct Nccl {
  void *lib = nullptr;
  int (*GetUniqueId)(NcclUniqueId *) = nullptr;
  int (*CommInitRank)(NcclComm *, int, NcclUniqueId, int) = nullptr;
  int (*CommDestroy)(NcclComm) = nullptr;
  int (*Send)(const void *, size_t, int, int, NcclComm, void *) = nullptr;
  int (*Recv)(void *, size_t, int, int, NcclComm, void *) = nullptr;
  int (*GroupStart)() = nullptr;
  int (*GroupEnd)() = nullptr;
  const char *(*GetErrorString)(int) = nullptr;
  std::string err;
  bool load() {
    if (lib) return true;
    lib = dlopen("libnccl.so.2", RTLD_NOW | RTLD_GLOBAL);
    if (!lib) { err = std::string("cannot load libnccl.so.2: ") + dlerror(); return false; }
    auto sym = [&](const char *n) { void *p = dlsym(lib, n); if (!p) err = std::string("libnccl.so.2 lacks ") + n; return p; };
    GetUniqueId = (decltype(GetUniqueId))sym("ncclGetUniqueId");
    CommInitRank = (decltype(CommInitRank))sym("ncclCommInitRank");
    CommDestroy = (decltype(CommDestroy))sym("ncclCommDestroy");
    Send = (decltype(Send))sym("ncclSend");
    Recv = (decltype(Recv))sym("ncclRecv");
    GroupStart = (decltype(GroupStart))sym("ncclGroupStart");
    GroupEnd = (decltype(GroupEnd))sym("ncclGroupEnd");
    GetErrorString = (decltype(GetErrorString))sym("ncclGetErrorString");
    if (!err.empty()) { lib = nullptr; return false; }
    return true;
  }
};
Nccl g_nccl;
constexpr int kNcclUint8 = 1;

int item_bytes(int H) { return H + ((H / 128 * 4 + 15) & ~15); }

}  // namespace

struct EpMoe::Impl {
  NcclComm comm = nullptr;
  std::map<std::string, ainfer_kernel_t> kernels;
  std::vector<void *> owned;
  std::vector<ainfer_list_t> lists;   // per layer: A, B, C (world > 1) or one list (world == 1)
  std::vector<ainfer_event_t> events;
};

#define EP_CHECK(call)                                        \
  do {                                                        \
    if ((call) != AINFER_OK) {                                \
      err = ainfer_last_error(dev);                           \
      return 1;                                               \
    }                                                         \
  } while (0)

int ep_unique_id(void *out128, std::string &err) {
  if (!g_nccl.load()) { err = g_nccl.err; return 1; }
  NcclUniqueId id;
  int r = g_nccl.GetUniqueId(&id);
  if (r) { err = std::string("ncclGetUniqueId: ") + g_nccl.GetErrorString(r); return 1; }
  std::memcpy(out128, &id, sizeof id);
  return 0;
}

template <typename T>
int EpMoe::alloc(T **p, size_t bytes) {
  void *q = nullptr;
  if (ainfer_mem_alloc(dev, bytes ? bytes : 16, 256, &q) != AINFER_OK) { err = ainfer_last_error(dev); return 1; }
  if (ainfer_mem_fill(dev, q, 0, bytes ? bytes : 16) != AINFER_OK) { err = ainfer_last_error(dev); return 1; }
  impl->owned.push_back(q);
  *p = (T *)q;
  return 0;
}

namespace {
struct Rec {   // appends launches to a list (none: launches at once); arguments by index in member order
  EpMoe *e;
  ainfer_list_t list;
  int status = 0;
  ainfer_kernel_t kernel(const char *name) {
    auto it = e->impl->kernels.find(name);
    if (it != e->impl->kernels.end()) return it->second;
    ainfer_kernel_t k = nullptr;
    if (ainfer_kernel_get(e->dev, name, &k) != AINFER_OK) {
      e->err = std::string("entry ") + name + " not found";
      status = 1;
      return nullptr;
    }
    e->impl->kernels[name] = k;
    return k;
  }
  template <typename T>
  void set(ainfer_kernel_t k, uint32_t &idx, const T &v) {
    if (status) return;
    if (ainfer_kernel_set_arg(k, idx, sizeof(T), &v) != AINFER_OK) { e->err = ainfer_last_error(e->dev); status = 1; }
    ++idx;
  }
  template <typename... A>
  void launch(const char *name, uint32_t groups, const A &...args) {
    if (status) return;
    ainfer_kernel_t k = kernel(name);
    if (!k) return;
    uint32_t idx = 0;
    (set(k, idx, args), ...);
    if (status) return;
    // several ranks: exchanges enter the queue between launches
    if ((list ? ainfer_list_append_launch(list, k, groups)
              : e->world == 1 ? ainfer_kernel_launch_next(e->dev, k, groups) : ainfer_kernel_launch(e->dev, k, groups)) != AINFER_OK) {
      e->err = ainfer_last_error(e->dev);
      status = 1;
    }
  }
  void copy(void *dst, const void *src, size_t bytes) {
    if (status) return;
    if (ainfer_list_append_memcpy(list, dst, src, bytes) != AINFER_OK) { e->err = ainfer_last_error(e->dev); status = 1; }
  }
};
// Rows of a problem of the experts' products when `items` (row, expert) pairs go to E experts: a unit of 16, 32 or 64
// rows has five, four or three stages of weights in flight, and most experts should be one unit. us of a layer's grouping, products and
// quantiser in problems of 16 / 32 / 64 rows. 512 experts of 512 x 2048, ten a row, by mean rows of an expert: 2 178 / 204 / 232, 8
// 230 / 251 / 283, 12 265 / 275 / 302, 13.7 293 / 287 / 315, 16 338 / 301 / 326. 128 experts, eight a row: 12 81 / 87 / 98, 16 96 / 91 /
// 100, 20 118 / 96 / 106, 24 133 / 103 / 113, 30 153 / 128 / 121, 60 273 / 221 / 195; with rows that favour experts by rank^-0.7 12
// 86 / 86 / 101, 16 99 / 104 / 102, 24 126 / 117 / 114, 30 152 / 136 / 131. Where a problem of every expert is one round of units on the
// SMs, a second problem of some is a second round: 64 experts of 256 x 1024, four a row: 8 19.0 / 20.8 / 24.3, 10 22.6 / 21.3 / 24.6,
// 12 23.6 / 21.6 / 25.1, 16 27.4 / 22.8 / 26.0, 20 30.2 / 28.8 / 27.1, 24 34.1 / 30.3 / 28.5.
int problem_rows(int items, int E, int I, int sm_count) {
  const bool one_round = 2L * E * (I / 128) <= 2L * sm_count;
  return items <= (one_round ? 8 : 12) * E ? 16 : items <= (one_round ? 20 : 24) * E ? 32 : 64;
}
}  // namespace

int EpMoe::create(DeviceModel *model, const void *id128, int rank_, int world_, int batch_, int flags_) {
  m = model;
  dev = m->dev;
  rank = rank_; world = world_; batch = batch_; flags = flags_;
  impl = new Impl;
  const ModelConfig &c = m->cfg;
  H = c.hidden; E = c.experts; k = c.top_k; I = c.expert_inter; shared = c.shared_experts != 0;
  if (world < 1 || world > 64 || rank < 0 || rank >= world) { err = "usage: 0 <= rank < world <= 64"; return 2; }
  if (batch < world || batch % world) { err = "usage: the batch must divide over the ranks"; return 2; }
  if (E % world) { err = "usage: the experts must divide evenly over the ranks"; return 2; }
  if (E > 1024 || H % 256 || I % 128) { err = "usage: unsupported shape (experts <= 1024, hidden % 256 == 0, intermediate % 128 == 0)"; return 2; }
  n = batch / world;
  epr = E / world;
  cap = n * k;
  const int most = world == 1 && (flags & EP_LARGE) ? 8192 : 2048;
  if (cap > most || batch * k > most) { err = "usage: batch x top-k above the planner's limit (" + std::to_string(most) + " items)"; return 2; }
  // a limit of the forms this block was first built from; problems of at most 64 rows would take these shapes too
  if (batch > 64 && !(256 % (H / 128) == 0 && 256 % (I / 128) == 0)) { err = "usage: more than 64 rows need hidden and intermediate sizes whose group counts divide 256"; return 2; }
  slot_d = (uint32_t)((16 + (size_t)cap * 16 + (size_t)cap * item_bytes(H) + 15) & ~(size_t)15);
  slot_r = (uint32_t)((size_t)cap * H * 4);
  ainfer_device_info info;
  EP_CHECK(ainfer_device_get_info(dev, &info));
  sm_count = info.sm_count;
  const int G = H / 128, rows = world * cap;   // rows: most items a rank can receive
  int r = 0;
  const int shn = shared ? n : 0;   // the owned rows follow the received items in the grouped layout
  r |= alloc(&Res, (size_t)n * H * 4); r |= alloc(&X, (size_t)n * H * 4); r |= alloc(&Hn, (size_t)n * H * 4);
  if (flags & EP_RES_ADD) { r |= alloc(&Add, (size_t)n * H * 4); r |= alloc(&ResSum, (size_t)n * H * 4); }
  r |= alloc(&Logits, (size_t)n * (E + 1) * 4); r |= alloc(&Bias, (size_t)E * 4);
  r |= alloc(&SelIdx, (size_t)n * (k + 1) * 4); r |= alloc(&SelW, (size_t)n * (k + 1) * 4); r |= alloc(&NearGap, (size_t)n * 4);
  r |= alloc(&ItemDest, (size_t)cap * 4);
  if (world > 1) {
    r |= alloc(&Send, (size_t)world * slot_d); r |= alloc(&Recv, (size_t)world * slot_d);
    r |= alloc(&Ret, (size_t)world * slot_r); r |= alloc(&Back, (size_t)world * slot_r);
  }
  r |= alloc(&Sorted, (size_t)rows * 4); r |= alloc(&Counts, 32); r |= alloc(&Lists, 16);
  const int least = world == 1 ? 16 : 64;   // an expert with more rows than problem_rows() is cut into problems of that many
  const size_t most_problems = (size_t)epr + 1 + (size_t)rows / least + (size_t)n / least + 2;
  r |= alloc(&GroupsGU, 2 * most_problems * 32); r |= alloc(&GroupsD, most_problems * 32);
  r |= alloc(&XQs, (size_t)(rows + n) * H); r |= alloc(&SQs, (size_t)(rows + n) * G * 4);
  r |= alloc(&GU, (size_t)(rows + shn) * 2 * I * 4); r |= alloc(&AQ, (size_t)(rows + shn) * I);
  r |= alloc(&ASQ, (size_t)(rows + shn) * (I / 128) * 4);
  r |= alloc(&Y2, (size_t)(rows + shn) * H * 4);
  if (r) return 1;
  // the owner's quantised rows live at the tail of the grouped layout: the shared expert reads them in place
  Q8 = XQs + (size_t)rows * H;
  SQ = SQs + (size_t)rows * G;
  Ysh = shared ? Y2 + (size_t)rows * H : nullptr;
  if (world > 1) {
    if (!id128) { err = "usage: a world of several ranks needs the shared NCCL id"; return 2; }
    if (!g_nccl.load()) { err = g_nccl.err; return 1; }
    NcclUniqueId id;
    std::memcpy(&id, id128, sizeof id);
    int nr = g_nccl.CommInitRank(&impl->comm, world, id, rank);
    if (nr) { err = std::string("ncclCommInitRank: ") + g_nccl.GetErrorString(nr); return 1; }
  }
  EP_CHECK(ainfer_device_stream(dev, &stream));
  return 0;
}

namespace {
// Norm and quantiser of `rows` owned rows, router logits, selection: the part both forms of the block begin with.
int emit_route(EpMoe *e, Rec &r, int L, int rows) {
  const ModelConfig &c = e->m->cfg;
  const std::string p = layer_prefix(L);
  DeviceTensor router = e->m->tensor(p + "mlp.gate.weight");
  DeviceTensor sgate = e->m->tensor(p + "mlp.shared_expert_gate.weight");
  if (!router.entry || (e->shared && !sgate.entry)) { e->err = "missing " + p + "mlp.gate.weight / shared_expert_gate.weight"; return 1; }
  const bool add = (e->flags & EP_RES_ADD) != 0;
  r.launch("RmsNormQuant", (uint32_t)rows, (const float *)e->Res, (const float *)(add ? e->Add : nullptr), (float *)(add ? e->ResSum : nullptr),
           (const float *)(e->m->post_norm + (size_t)L * e->H), e->Hn, e->Q8, e->SQ, (int32_t)e->H, (float)c.rms_eps);
  const int tpb = rows > 128 ? 16 : 8;   // tokens per block: fewer reads of the weights, or enough blocks
  r.launch("RouterLogitsRows", (uint32_t)(((e->E + 1 + 31) / 32) * ((rows + tpb - 1) / tpb)), (const uint16_t *)router.data,
           (const uint16_t *)(e->shared ? sgate.data : nullptr), (const float *)e->Hn,
           (const float *)((e->flags & EP_ROUTER_BIAS) ? e->Bias : nullptr), e->Logits, (int32_t)e->E, (int32_t)e->H, (int32_t)rows, (int32_t)tpb);
  r.launch("RouterSelectRows", (uint32_t)rows, (const float *)e->Logits, e->SelIdx, e->SelW, e->NearGap, (int32_t)e->E, (int32_t)e->k,
           (int32_t)(e->shared ? 1 : 0));
  return 0;
}
// The experts' products over the grouped rows: problems of GroupsGU / GroupsD.
void emit_experts(EpMoe *e, Rec &r, int front, int shared_rows, int max_rows, const int32_t *lists) {   // front: rows the received items may take
  const uint32_t blocks = (uint32_t)(2 * e->sm_count);
  r.launch("Int4GemmA8TcGrouped", blocks, (const void *)e->GroupsGU, lists, (const int8_t *)e->XQs, (const float *)e->SQs,
           e->GU, (int32_t)e->I, (int32_t)e->H, (int32_t)max_rows, (int32_t)(2 * e->I));
  r.launch("SiluQuantRows", (uint32_t)(front + shared_rows), (const float *)e->GU, (const int32_t *)e->Counts, e->AQ, e->ASQ, (int32_t)e->I,
           (int32_t)(e->world * e->cap), (int32_t)front);
  r.launch("Int4GemmA8TcGrouped", blocks, (const void *)e->GroupsD, lists + 1, (const int8_t *)e->AQ, (const float *)e->ASQ,
           e->Y2, (int32_t)e->H, (int32_t)e->I, (int32_t)max_rows, (int32_t)e->H);
}
// One rank: `rows` of its rows, no dispatch. (A dispatch buffer, its copy, the un-permute and its copy moved
// every item's 2 KB four times and its 8 KB output three times; the planner walked all earlier items of each.)
int emit_local(EpMoe *e, Rec &r, int L, int rows) {
  if (emit_route(e, r, L, rows)) return 1;
  const ExpertW *tab = (const ExpertW *)e->m->expert_tables + (size_t)L * (e->E + 1);
  const int items = rows * e->k, shared_rows = e->shared ? rows : 0, cut = std::min(rows, problem_rows(items, e->E, e->I, e->sm_count));
  r.launch("EpGroupLocalCut", 1u, (const int32_t *)e->SelIdx, tab, e->Sorted, e->ItemDest, e->GroupsGU, e->GroupsD, e->Counts, (int32_t)rows,
           (int32_t)e->k, (int32_t)e->E, (int32_t)e->I, (int32_t)e->cap, (int32_t)shared_rows, (int32_t)cut, e->Lists);
  r.launch("EpGatherLocal", (uint32_t)items, (const int8_t *)e->Q8, (const float *)e->SQ, (const int32_t *)e->Sorted, e->XQs, e->SQs, (int32_t)e->H,
           (int32_t)e->k);
  emit_experts(e, r, items, shared_rows, cut, e->Lists);
  const float *res_in = (e->flags & EP_RES_ADD) ? e->ResSum : e->Res;   // what the combine adds the experts' outputs to
  r.launch("EpCombine", (uint32_t)(rows * ((e->H + 255) / 256)), res_in, (const unsigned char *)e->Y2, (const int32_t *)e->ItemDest,
           (const float *)e->SelW, (const float *)(e->shared ? e->Ysh : nullptr), e->X, e->Res, (int32_t)e->k, (int32_t)e->H, (uint32_t)0);
  return r.status;
}
}  // namespace

// Records the lists of one layer: [A, B, C] for several ranks, [all] for one.
int EpMoe::record_layer(int L) {
  const int rows = world * cap;
  const ExpertW *tab = (const ExpertW *)m->expert_tables + (size_t)L * (E + 1);
  auto new_list = [&](ainfer_list_t *l) {
    if (ainfer_list_create(dev, l) != AINFER_OK) { err = ainfer_last_error(dev); return 1; }
    impl->lists.push_back(*l);
    return 0;
  };
  auto close = [&](Rec &r) {
    if (r.status) return 1;
    if (ainfer_list_close(r.list) != AINFER_OK) { err = ainfer_last_error(dev); return 1; }
    return 0;
  };
  ainfer_list_t la = nullptr;
  if (new_list(&la)) return 1;
  Rec r{this, la};
  if (world == 1) return emit_local(this, r, L, n) ? 1 : close(r);
  // ---- A: route the owned rows and pack their items ----
  const float *res_in = (flags & EP_RES_ADD) ? ResSum : Res;   // what the combine adds the experts' outputs to
  if (emit_route(this, r, L, n)) return 1;
  r.launch("EpPlan", 1u, (const int32_t *)SelIdx, Send, ItemDest, (int32_t)n, (int32_t)k, (int32_t)epr, (int32_t)world, (int32_t)cap, slot_d);
  r.launch("EpPack", (uint32_t)cap, (const int8_t *)Q8, (const float *)SQ, (const int32_t *)ItemDest, Send, (int32_t)k, (int32_t)H, (int32_t)cap,
           slot_d);
  if (close(r) || new_list(&la)) return 1;
  r.list = la;
  // ---- B: the experts of this rank on everything received ----
  r.launch("EpGroup", 1u, (const unsigned char *)Recv, tab, Sorted, GroupsGU, GroupsD, Counts, (int32_t)world, (int32_t)rank, (int32_t)epr,
           (int32_t)cap, (int32_t)I, slot_d, (int32_t)rows, (int32_t)(shared ? n : 0), (int32_t)E,
           (int32_t)64);
  r.launch("EpGather", (uint32_t)rows, (const unsigned char *)Recv, (const int32_t *)Sorted, (const int32_t *)Counts, XQs, SQs, (int32_t)H,
           (int32_t)cap, slot_d);
  emit_experts(this, r, rows, shared ? n : 0, std::min(batch, 64), Counts + 5);
  r.launch("EpScatter", (uint32_t)rows, (const float *)Y2, (const int32_t *)Sorted, (const int32_t *)Counts, Ret, (int32_t)H, slot_r);
  if (close(r) || new_list(&la)) return 1;
  r.list = la;
  // ---- C: combine ----
  r.launch("EpCombine", (uint32_t)(n * ((H + 255) / 256)), res_in, (const unsigned char *)Back, (const int32_t *)ItemDest,
           (const float *)SelW, (const float *)(shared ? Ysh : nullptr), X, Res, (int32_t)k, (int32_t)H, slot_r);
  return close(r);
}

int EpMoe::ensure_layer(int L) {
  const int nl = m->cfg.layers + m->cfg.mtp_layers;
  if (L < 0 || L >= nl) { err = "usage: no such layer"; return 2; }
  if (layer_lists.empty()) layer_lists.assign((size_t)nl, -1);
  if (layer_lists[L] >= 0) return 0;
  const int first = (int)impl->lists.size();
  int r = record_layer(L);
  if (r) return r;
  layer_lists[L] = first;
  return 0;
}

int EpMoe::exchange(void *send, void *recv, uint32_t slot) {
  int r = g_nccl.GroupStart();
  for (int p = 0; p < world && !r; ++p) {
    r = g_nccl.Send((const char *)send + (size_t)p * slot, slot, kNcclUint8, p, impl->comm, stream);
    if (!r) r = g_nccl.Recv((char *)recv + (size_t)p * slot, slot, kNcclUint8, p, impl->comm, stream);
  }
  const int e = g_nccl.GroupEnd();
  if (!r) r = e;
  if (r) { err = std::string("NCCL exchange: ") + g_nccl.GetErrorString(r); return 1; }
  return 0;
}

int EpMoe::run_layer(int L, float *seg_ms) {
  int r = ensure_layer(L);
  if (r) return r;
  const int i = layer_lists[L];
  auto stamp = [&](int j) {
    if (!seg_ms) return 0;
    while ((int)impl->events.size() <= j) {
      ainfer_event_t ev = nullptr;
      if (ainfer_event_create(dev, &ev) != AINFER_OK) { err = ainfer_last_error(dev); return 1; }
      impl->events.push_back(ev);
    }
    if (ainfer_event_record(impl->events[j]) != AINFER_OK) { err = ainfer_last_error(dev); return 1; }
    return 0;
  };
  if (stamp(0)) return 1;
  if (world == 1) {
    EP_CHECK(ainfer_list_execute(impl->lists[i]));
    if (stamp(1) || stamp(2) || stamp(3) || stamp(4)) return 1;
  } else {
    EP_CHECK(ainfer_list_execute(impl->lists[i]));
    if (stamp(1)) return 1;
    if (exchange(Send, Recv, slot_d)) return 1;
    if (stamp(2)) return 1;
    EP_CHECK(ainfer_list_execute(impl->lists[i + 1]));
    if (stamp(3)) return 1;
    if (exchange(Ret, Back, slot_r)) return 1;
    if (stamp(4)) return 1;
    EP_CHECK(ainfer_list_execute(impl->lists[i + 2]));
  }
  if (stamp(5)) return 1;
  if (seg_ms) {
    EP_CHECK(ainfer_sync(dev, ~0ull));
    for (int j = 0; j < 5; ++j) {
      float ms = 0;
      EP_CHECK(ainfer_event_elapsed_ms(impl->events[j], impl->events[j + 1], &ms));
      seg_ms[j] += ms;
    }
  }
  return 0;
}

int EpMoe::run_rows(int L, int rows) {
  if (world > 1) return run_layer(L, nullptr);
  if (L < 0 || L >= m->cfg.layers + m->cfg.mtp_layers || rows < 0 || rows > n) { err = "usage: no such layer, or more rows than the block holds"; return 2; }
  Rec r{this, nullptr};
  return rows ? emit_local(this, r, L, rows) : 0;
}

int EpMoe::run_stack(int first, int count, float *seg_ms) {
  for (int L = first; L < first + count; ++L) {
    int r = run_layer(L, seg_ms);
    if (r) return r;
  }
  return 0;
}

void EpMoe::destroy() {
  if (!impl) return;
  ainfer_sync(dev, ~0ull);
  for (ainfer_list_t l : impl->lists) ainfer_list_destroy(l);
  for (auto &kv : impl->kernels) ainfer_kernel_release(kv.second);
  for (ainfer_event_t e : impl->events) ainfer_event_destroy(e);
  for (void *p : impl->owned) ainfer_mem_free(dev, p);
  if (impl->comm) g_nccl.CommDestroy(impl->comm);
  delete impl;
  impl = nullptr;
}

}  // namespace ainfer
