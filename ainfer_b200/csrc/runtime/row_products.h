// W4A8 products of the INT4 hybrid's rows: Y[rows][N] = X[rows][K] . W^T for up to four matrices over the same quantised
// rows. What the prompt passes and the batch engine share.
#pragma once
#include <algorithm>
#include <initializer_list>

#include "launcher.h"
#include "model.h"

namespace ainfer {

struct RowProduct {
  DeviceTensor t;
  float *Y;
};
inline void row_products(KernelCalls &l, const char *who, int sm_count, std::initializer_list<RowProduct> of, const int8_t *XQ, const float *SQ, int K,
                         int rows) {
  if (l.status) return;
  const int G = K / 128;
  struct { const uint8_t *P; const uint16_t *S; float *Y; int32_t N; } m[4] = {};
  int n = 0;
  long tiles = 0;
  for (const RowProduct &p : of) {
    if (!p.t.entry || (int)p.t.entry->shape[1] != K || p.t.entry->storage != DT_INT4_SYM_G128) {
      l.fail(2, std::string(who) + ": missing tensor or unexpected shape/storage" + (p.t.entry ? " of " + p.t.entry->name : std::string()));
      return;
    }
    const int N = (int)p.t.entry->shape[0];
    if (rows <= 8 && G <= 256 && 256 % G == 0) {
      // few rows: the dp4a kernel streams the weights once and has a fraction of the tensor-core kernel's latency
      const uint32_t t = (uint32_t)((N + 256 / G - 1) / (256 / G));
      l.launch("Int4GemvA8Multi", std::min<uint32_t>(t, 2u * (uint32_t)sm_count), (const uint8_t *)p.t.data, (const uint16_t *)p.t.scales, XQ, SQ, p.Y,
               (int32_t)N, (int32_t)K, (int32_t)rows, (int32_t)N);
      continue;
    }
    m[n].P = (const uint8_t *)p.t.data; m[n].S = (const uint16_t *)p.t.scales; m[n].Y = p.Y; m[n].N = N;
    tiles += (N + 127) / 128;
    ++n;
  }
  if (!n) return;
  const uint32_t blocks = (uint32_t)std::min<long>(tiles * ((rows + 15) / 16), 2L * sm_count);
  if (n == 1)
    l.launch("Int4GemmA8Tc", blocks, m[0].P, m[0].S, XQ, SQ, m[0].Y, m[0].N, (int32_t)K, (int32_t)rows, m[0].N);
  else
    // one launch: a matrix of 32 rows alone is a launch of 8..11 us that a few blocks run
    l.launch("Int4GemmA8TcMany", blocks, XQ, SQ, (int32_t)K, (int32_t)rows, (int32_t)n, m[0].P, m[0].S, m[0].Y, m[0].N, m[1].P, m[1].S, m[1].Y,
             m[1].N, m[2].P, m[2].S, m[2].Y, m[2].N, m[3].P, m[3].S, m[3].Y, m[3].N);
}

}  // namespace ainfer
