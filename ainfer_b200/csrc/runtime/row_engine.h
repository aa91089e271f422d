// What the row engines share: tensor lists, prepared matrices, device buffers, and the products of rows
// and of a decode step's single row.
#pragma once
#include <algorithm>
#include <string>
#include <vector>

#include "arch.h"

namespace ainfer {

inline int round_up(int v, int m) { return (v + m - 1) / m * m; }
inline std::string layer_name(int L) { return "l" + std::to_string(L) + "."; }
std::string json_num(double v);   // every digit

// ----------------------------------------------------------------- tensors ---
// One bf16 tensor of an architecture and how a synthetic model fills it (N(0, std^2), or a constant).
struct RowTensor { std::string name; std::vector<uint64_t> shape; float std_, constant; };
void plan_row_tensors(const std::vector<RowTensor> &t, const std::string &arch_json, int vocab, Container &dir, std::vector<SynthSpec> &specs);
int check_row_tensors(const Container &dir, const std::vector<RowTensor> &t, std::string &err);

struct RowMatrix {           // bf16 rows of ldw values (ldw a multiple of 8, zero padding)
  const uint16_t *w = nullptr;
  const float *bias = nullptr;
  int N = 0, K = 0, ldw = 0;
};

// Preparation of a model's weights; what it allocates belongs to the model.
struct RowLoader : KernelCalls {
  DeviceModel *m;
  std::map<std::string, ainfer_kernel_t> handles;
  RowLoader(DeviceModel *model, std::string *err);
  void *alloc(size_t bytes);
  const float *widen(const std::string &name);                 // fp32 copy on the device
  std::vector<uint16_t> host(const std::string &name);         // bf16 values on the host
  const float *upload(const std::vector<float> &v);
  const float *gain(const std::string &name);                  // 1 + the stored weight
  // the rows of matrices with the same row length as one; copied only when rows need padding or do not adjoin
  RowMatrix stack(const std::vector<std::string> &names);
  void finish();                                               // waits, releases the handles
};

// ------------------------------------------------------------------ engine ---
enum { ACT_NONE = 0, ACT_RELU2 = 1, ACT_SOFTCAP = 2 };
struct alignas(64) TensorMap { unsigned char b[128]; };

struct RowEngineBase : RowEngine {
  DeviceModel *m = nullptr;
  ainfer_device_t dev = nullptr;
  int nseq = 0, max_ctx = 0, sm_count = 1;
  bool f32 = false;
  std::vector<void *> owned;
  std::string alloc_err;

  ~RowEngineBase() override;
  int begin(DeviceModel *model, int n, int ctx, int cap_rows, bool in_f32, std::string &err);
  size_t esz() const { return f32 ? 4 : 2; }
  int alloc_bytes(size_t bytes, void **out);
  template <typename T>
  int alloc(size_t count, T **out) {
    void *p = nullptr;
    if (alloc_bytes(count * sizeof(T), &p)) return 1;
    *out = (T *)p;
    return 0;
  }
  // Y[rows][N] = act(X W^T + bias); X in the activation type, out16: Y bf16 (else fp32)
  void linear(KernelCalls &k, const RowMatrix &mt, const char *Xp, int ldx, int rows, void *Yp, int ldy, int act, bool out16, float cap = 0.0f);
  // one fp32 row; the same for kernels that prepare the row themselves: rows per block and blocks
  int gemv_rows(int N) const { return (N + 2 * sm_count - 1) / (2 * sm_count); }
  uint32_t gemv_blocks(int N) const { return (uint32_t)((N + gemv_rows(N) - 1) / gemv_rows(N)); }
  void gemv(KernelCalls &k, const RowMatrix &mt, const float *x, float *y, int act, float cap = 0.0f);
  // name of the instance of a kernel family whose padded head size holds `dim`
  static std::string sized(const char *base, int dim) {
    for (int d : {32, 64, 96, 128, 192})
      if (dim <= d) return base + std::to_string(d);
    return base + std::string("256");
  }
  // Whether products of many rows go by pairs of blocks (LinearTcPair, LinearTcGroupedPair). A pair starts about a
  // microsecond later and reads a third less from L2, which shows in wide tiles over a long launch only. us alone / in
  // pairs, outputs x K: 2048 rows (tiles of 240) 8192 x 2048 59.0 / 55.2, 2048 x 8192 52.3 / 48.9, 4096 x 4096
  // 53.1 / 50.0, 8192 x 1536 46.3 / 43.6, but 6144 x 1536 (three rounds) 32.5 / 33.3, 4096 x 2048 (two) 29.0 / 30.0, 8192 x
  // 1024 (four) 34.1 / 36.2; 1800 rows (tiles of 208) 8192 x 2048 54.4 / 53.2, 2048 x 8192 49.0 / 47.6; tiles of 176 always
  // lose (1500 rows, 8192 x 2048 48.1 / 49.4; 2048 x 8192 44.3 / 46.2). 32 experts of 375 rows 1024 x 2048 61.4 / 56.9,
  // 2048 x 1024 60.5 / 61.5; of 100 rows 33.8 / 34.9.
  static bool pairs_pay(int nt, long rounds, int K) { return nt >= 208 && K >= 1536 && rounds * K >= 6144; }
  // Blocks of a step's attention per (sequence, key head): few tiles each when there are many sequences. The cut decides
  // the order of the sums, so it depends on the sequences and heads alone and not on the context that was asked for:
  // the same tokens give the same logits in a session or batch of any length. (Fewer blocks for batches, three an SM, all of them
  // resident, took 254 us against 277 for a step of 16 sequences of Sinepel at 600 and 422 against 433 for 64 of Robopel at 700; but a
  // batch's logits moved by 0.5 % and 1.6 %, about their distance from 64 bits, and came no nearer to it.)
  int step_splits(int max_kv_heads) const {
    if (nseq == 1) return std::max(1, std::min(16, 2 * sm_count / max_kv_heads));
    return std::max(1, std::min(16, 8 * sm_count / (std::min(nseq, 8 * sm_count) * max_kv_heads)));
  }
};

}  // namespace ainfer
