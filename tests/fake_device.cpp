// The device boundary of the runtime library on host memory, for tests without a GPU: nothing computes. Copies that may be
// asynchronous and launches wait in one queue until something blocks, so a host buffer is read as late as the interface allows. Every
// launch is logged when its turn comes, the token embedding with the control blocks it would read.
// FAKE_FAIL=<kernel>:<n>: the n-th launch of that kernel is refused.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "ainfer_cuda.h"

struct ainfer_device_s { int unused; };
struct ainfer_kernel_s { std::string name; std::map<uint32_t, std::vector<char>> args; };
struct ainfer_list_s { std::vector<std::function<void()>> ops; };
struct ainfer_event_s { int unused; };

static ainfer_device_s the_device;
static std::vector<std::function<void()>> queue;
static std::string log_text;
static std::map<std::string, int> launches;

static int drain() {
  for (auto &op : queue) op();
  queue.clear();
  return AINFER_OK;
}
static std::function<void()> launch_op(ainfer_kernel_t k, uint32_t groups) {
  const ainfer_kernel_s at = *k;
  return [at, groups]() {
    log_text += at.name + " " + std::to_string(groups);
    const uint32_t arg = at.name == "EmbedRow" ? 2 : at.name == "EmbedPosRows" ? 3 : 0;
    if (arg) {
      const int32_t *ctrl = *reinterpret_cast<int32_t *const *>(at.args.at(arg).data());
      for (uint32_t i = 0; i < groups; ++i) log_text += " " + std::to_string(ctrl[4 * i]) + "@" + std::to_string(ctrl[4 * i + 1]);
    }
    log_text += "\n";
  };
}

extern "C" {
const char *fake_log() { return log_text.c_str(); }
void fake_clear() { log_text.clear(); }
int fake_queued() { return (int)queue.size(); }

int ainfer_device_open(int, ainfer_device_t *out) { *out = &the_device; return AINFER_OK; }
int ainfer_device_close(ainfer_device_t) { return drain(); }
int ainfer_device_get_info(ainfer_device_t, ainfer_device_info *i) {
  std::memset(i, 0, sizeof *i);
  std::snprintf(i->name, sizeof i->name, "host");
  i->sm_count = 148; i->cc_major = 10; i->l2_bytes_mb = 126;
  i->total_mem = i->free_mem = 180ull << 30;
  return AINFER_OK;
}
const char *ainfer_last_error(ainfer_device_t) { return "refused by the test"; }
int ainfer_mem_alloc(ainfer_device_t, size_t bytes, size_t, void **out) { *out = std::calloc(1, bytes); return *out ? AINFER_OK : AINFER_ERR_OOM; }
int ainfer_mem_free(ainfer_device_t, void *p) { drain(); std::free(p); return AINFER_OK; }
int ainfer_host_alloc(ainfer_device_t d, size_t bytes, void **out) { return ainfer_mem_alloc(d, bytes, 1, out); }
int ainfer_host_free(ainfer_device_t d, void *p) { return ainfer_mem_free(d, p); }
int ainfer_memcpy_h2d(ainfer_device_t, void *d, const void *s, size_t n) { drain(); std::memcpy(d, s, n); return AINFER_OK; }
int ainfer_memcpy_d2h(ainfer_device_t dev, void *d, const void *s, size_t n) { return ainfer_memcpy_h2d(dev, d, s, n); }
int ainfer_memcpy_d2d(ainfer_device_t dev, void *d, const void *s, size_t n) { return ainfer_memcpy_h2d(dev, d, s, n); }
int ainfer_mem_fill(ainfer_device_t, void *d, int v, size_t n) { drain(); std::memset(d, v, n); return AINFER_OK; }
int ainfer_memcpy_h2d_async(ainfer_device_t, void *d, const void *s, size_t n) {
  queue.push_back([=] { std::memcpy(d, s, n); });
  return AINFER_OK;
}
int ainfer_memcpy_d2h_async(ainfer_device_t dev, void *d, const void *s, size_t n) { return ainfer_memcpy_h2d_async(dev, d, s, n); }
int ainfer_control_write_async(ainfer_device_t dev, void *d, const ainfer_control *c) { return ainfer_memcpy_h2d_async(dev, d, c, sizeof *c); }
int ainfer_control_write(ainfer_device_t dev, void *d, const ainfer_control *c) { return ainfer_memcpy_h2d(dev, d, c, sizeof *c); }
int ainfer_tensor_map_bf16(ainfer_device_t, void *map, const void *, uint64_t, uint64_t, uint64_t, uint32_t) { std::memset(map, 0, 128); return AINFER_OK; }
int ainfer_kernel_get(ainfer_device_t, const char *name, ainfer_kernel_t *out) { *out = new ainfer_kernel_s{name, {}}; return AINFER_OK; }
int ainfer_kernel_release(ainfer_kernel_t k) { delete k; return AINFER_OK; }
int ainfer_kernel_max_groups(ainfer_kernel_t, uint32_t *groups) { *groups = 148; return AINFER_OK; }
int ainfer_kernel_set_arg(ainfer_kernel_t k, uint32_t i, size_t n, const void *v) {
  k->args[i].assign((const char *)v, (const char *)v + n);
  return AINFER_OK;
}
int ainfer_kernel_launch(ainfer_device_t, ainfer_kernel_t k, uint32_t groups) {
  const char *f = std::getenv("FAKE_FAIL");
  if (f && k->name + ":" + std::to_string(++launches[k->name]) == f) return AINFER_ERR_DEVICE;
  queue.push_back(launch_op(k, groups));
  return AINFER_OK;
}
int ainfer_kernel_launch_next(ainfer_device_t d, ainfer_kernel_t k, uint32_t groups) { return ainfer_kernel_launch(d, k, groups); }
int ainfer_list_create(ainfer_device_t, ainfer_list_t *out) { *out = new ainfer_list_s; return AINFER_OK; }
int ainfer_list_one_step(ainfer_list_t) { return AINFER_OK; }
int ainfer_list_append_launch(ainfer_list_t l, ainfer_kernel_t k, uint32_t groups) { l->ops.push_back(launch_op(k, groups)); return AINFER_OK; }
int ainfer_list_append_memcpy(ainfer_list_t l, void *d, const void *s, size_t n) { l->ops.push_back([=] { std::memcpy(d, s, n); }); return AINFER_OK; }
int ainfer_list_append_fill(ainfer_list_t l, void *d, int v, size_t n) { l->ops.push_back([=] { std::memset(d, v, n); }); return AINFER_OK; }
int ainfer_list_close(ainfer_list_t) { return AINFER_OK; }
int ainfer_list_destroy(ainfer_list_t l) { drain(); delete l; return AINFER_OK; }
int ainfer_list_execute(ainfer_list_t l) { queue.insert(queue.end(), l->ops.begin(), l->ops.end()); return AINFER_OK; }
int ainfer_sync(ainfer_device_t, uint64_t) { return drain(); }
int ainfer_event_create(ainfer_device_t, ainfer_event_t *out) { *out = new ainfer_event_s; return AINFER_OK; }
int ainfer_event_record(ainfer_event_t) { return AINFER_OK; }
int ainfer_event_elapsed_ms(ainfer_event_t, ainfer_event_t, float *ms) { *ms = 1; return AINFER_OK; }
int ainfer_event_destroy(ainfer_event_t e) { delete e; return AINFER_OK; }
int ainfer_device_stream(ainfer_device_t, void **s) { *s = nullptr; return AINFER_OK; }
}
