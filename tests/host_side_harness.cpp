// Host-only harness for tests/test_host_side.py: exports the parts of the library's host side
// that need no CUDA call.  Built by the test with g++; not part of the library.
#include "qb_host.cuh"

#include <cstring>

namespace {
size_t g_room, g_used;
struct FakeAlloc {  // allocates from g_room bytes
  static constexpr size_t kMin = 256;
  static int alloc(void** p, size_t bytes) {
    if (bytes > g_room) return 2;
    g_used = bytes;
    *p = &g_used;
    return 0;
  }
  static void release(void*) { g_used = 0; }
};
}  // namespace

extern "C" {

// Grows one buffer to each size in turn with `room` bytes to be had: the bytes then in use, or 0
// where the buffer refuses.
void h_grow(uint64_t room, const uint64_t* sizes, int count, uint64_t* used) {
  qb::GrowBuf<FakeAlloc> b;
  g_room = room;
  g_used = 0;
  for (int i = 0; i < count; ++i) used[i] = b.ensure(sizes[i]) ? 0 : g_used;
}

// The graph key of a BatchShape given as its uint64 fields; returns the key's length.
int h_batch_graph_key(const uint64_t* fields, int nfields, uint64_t* out, int room) {
  qb::BatchShape s{};
  if (nfields * 8 != (int)sizeof(s)) return -1;
  memcpy(&s, fields, sizeof(s));
  const std::vector<uint64_t> k = qb::batch_graph_key(s);
  for (int i = 0; i < (int)k.size() && i < room; ++i) out[i] = k[i];
  return (int)k.size();
}

int h_exact_form_fits(uint64_t records) { return qb::exact_form_fits(records) ? 1 : 0; }

// W and sum |Q| of a host matrix; sum and the integer flag in out[0], out[1]
int h_load(const void* q, int n, int64_t ldq, int dtype, double* W, double* out) {
  const qb_problem p{n, dtype, q, ldq, 0, 0};
  bool is_int = false;
  const int rc = qb::load_host_problem_into(&p, W, &out[0], &is_int);
  out[1] = is_int;
  return rc;
}

}  // extern "C"
