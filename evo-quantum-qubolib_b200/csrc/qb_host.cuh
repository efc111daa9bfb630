// qb_host.cuh -- host-only parts of the library that need no CUDA call.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/qubo_b200.h"
#include "qb_common.cuh"

namespace qb {

// A buffer that grows on demand and keeps its room.  It takes an eighth more than asked, so that
// the next, slightly larger call does not allocate again, but at most 16 MB more, and where that
// much cannot be had just what is asked.  A: alloc(&p, bytes) (0 on success), release(p), kMin.
template <class A>
struct GrowBuf {
  static constexpr size_t kMaxSlack = (size_t)16 << 20;
  void* p = nullptr;
  size_t cap = 0;
  int ensure(size_t bytes) {
    if (bytes <= cap) return 0;
    release();
    const size_t least = std::max(bytes, A::kMin), want = std::max(bytes + std::min(bytes / 8, kMaxSlack), A::kMin);
    size_t got = want;
    int e = A::alloc(&p, want);
    if (e && want > least) e = A::alloc(&p, got = least);
    if (e)
      p = nullptr;
    else
      cap = got;
    return e;
  }
  void release() {
    if (p) A::release(p);
    p = nullptr;
    cap = 0;
  }
};

// The exact form's largest whole-problem search: 2^32 records of 2^16 states (n = 48).  Its
// sharded form holds 24 bytes per record, 103 GB here, and refuses more for want of memory; the
// whole-problem form holds next to nothing and would keep the GPU busy in one launch, for
// minutes at n = 49 and for weeks at n = 62.
constexpr uint64_t kExactMaxRecords = 1ull << 32;
inline bool exact_form_fits(uint64_t records) { return records <= kExactMaxRecords; }

// Everything a captured batch graph holds by value: copy sizes, grids, shared-memory sizes, the
// kernels' scalar parameters and the buffers' addresses.  A batch may replay the graph of an
// earlier one only where all of it is equal; the arrays the copies carry may differ.
struct BatchShape {
  uint64_t problems, w_doubles, arena_bytes, cap;  // copies, candidate room
  uint64_t gtab_items, units, selections, tc_runs;  // grids (tc_runs: CTAs + 1)
  uint64_t sm_gtab, sm_gray, sm_exact, sm_tc;       // dynamic shared memory
  uint64_t any_gray, tc_pair;                       // which kernels
  uint64_t tc_n_max;  // largest n of the tensor-core problems: fixes the kernel's shared-memory
                      // layout, which sm_tc does not tell (at least 120 KB for every n)
  uint64_t offsets[9];    // of the arena's parts
  uint64_t addresses[9];  // host and device buffers, stream
};

inline std::vector<uint64_t> batch_graph_key(const BatchShape& s) {
  std::vector<uint64_t> k = {s.problems, s.w_doubles, s.arena_bytes, s.cap,     s.gtab_items, s.units,    s.selections,
                             s.tc_runs,  s.sm_gtab,   s.sm_gray,     s.sm_exact, s.sm_tc,      s.any_gray, s.tc_pair,
                             s.tc_n_max};
  k.insert(k.end(), s.offsets, s.offsets + 9);
  k.insert(k.end(), s.addresses, s.addresses + 9);
  return k;
}

inline int dtype_size(int dt) {
  switch (dt) {
    case QB_F32: return 4;
    case QB_F64: return 8;
    case QB_I8: return 1;
    case QB_I16: return 2;
    case QB_I32: return 4;
    case QB_I64: return 8;
    default: return 0;
  }
}

template <class T>
int host_problem_typed(const qb_problem* p, double* Wout, double* abs_sum) {
  const int n = p->n;
  const T* src = static_cast<const T*>(p->q);
  const size_t ld = (size_t)p->ldq;
  double s = 0.0;
  bool bad = false;
  for (int i = 0; i < n; ++i) {
    const T* row = src + i * ld;
    const double d = (double)row[i];
    bad |= !std::isfinite(d);
    s += std::fabs(d);
    Wout[(size_t)i * n + i] = d;
    for (int j = i + 1; j < n; ++j) {
      const double a = (double)row[j], b = (double)src[j * ld + i];
      bad |= !std::isfinite(a) || !std::isfinite(b);
      s += std::fabs(a) + std::fabs(b);
      Wout[(size_t)i * n + j] = Wout[(size_t)j * n + i] = a + b;
    }
  }
  if (bad) return QB_EINVAL;
  *abs_sum = s;
  return QB_OK;
}

// Q in host memory (any dtype, 1 <= n <= 62) -> W (n x n doubles, written to Wout) and sum |Q_ij|,
// without intermediate copies (the batched search packs thousands of these) unless the address is
// not a multiple of the element size, as a view into a byte buffer can have it.
inline int load_host_problem_into(const qb_problem* p, double* Wout, double* abs_sum, bool* is_int) {
  *is_int = p->dtype >= QB_I8;
  const size_t es = (size_t)dtype_size(p->dtype);
  if (es && (uintptr_t)p->q % es) {
    alignas(8) unsigned char tmp[kMaxN * kMaxN * 8];
    const size_t row = (size_t)p->n * es;
    for (int i = 0; i < p->n; ++i)
      memcpy(tmp + i * row, static_cast<const unsigned char*>(p->q) + (size_t)i * (size_t)p->ldq * es, row);
    qb_problem at = *p;
    at.q = tmp;
    at.ldq = p->n;
    return load_host_problem_into(&at, Wout, abs_sum, is_int);
  }
  switch (p->dtype) {
    case QB_F32: return host_problem_typed<float>(p, Wout, abs_sum);
    case QB_F64: return host_problem_typed<double>(p, Wout, abs_sum);
    case QB_I8: return host_problem_typed<int8_t>(p, Wout, abs_sum);
    case QB_I16: return host_problem_typed<int16_t>(p, Wout, abs_sum);
    case QB_I32: return host_problem_typed<int32_t>(p, Wout, abs_sum);
    case QB_I64: return host_problem_typed<int64_t>(p, Wout, abs_sum);
    default: return QB_EINVAL;
  }
}

}  // namespace qb
