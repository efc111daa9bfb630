// qb_host.cuh -- host-only parts of the library that need no CUDA call.
#pragma once
#include <cstdint>
#include <vector>

namespace qb {

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

}  // namespace qb
