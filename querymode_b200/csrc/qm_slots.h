// qm_slots.h — sizes of hash tables (host arithmetic).
#pragma once

#include <algorithm>
#include <cstdint>

constexpr int QM_MAX_LOG2_SLOTS = 31;

// Slots wanted for a number of groups: 2.1 each, any number.  At 1.6 the
// longest of a warp's 32 probes grows (20M rows into 500,000 groups: scan 0.76
// -> 0.94 ms); rounded up to a power of two (2.1-4.3 each) the table is larger
// to clear, rank and emit.
inline int64_t qm_slots_wanted(int64_t groups) { return std::max<int64_t>(1024, groups * 2 + groups / 8); }

inline int qm_log2_ceil(int64_t x) {
  int l = 0;
  while (((int64_t)1 << l) < x) l++;
  return l;
}

// Slots of a one-shot table (a table too small for its groups overflows and
// is made again).  Deduplicating kernels read the key alone while they probe,
// so for them it is rounded up to a power of two (20M rows into 2,000 groups,
// five columns: scan 2.39 -> 1.90 ms).
inline int64_t qm_hash_slots(int64_t groups, bool dedupe = false) {
  const int64_t want = std::min<int64_t>((int64_t)1 << QM_MAX_LOG2_SLOTS, qm_slots_wanted(groups));
  return dedupe ? (int64_t)1 << qm_log2_ceil(want) : want;
}

// log2 of the slots a stream's table of n_slots grows to for `groups` groups:
// 0 none needed, above QM_MAX_LOG2_SLOTS more than a table may have.  (A power
// of two: growing push by push re-hashes rarely.)
inline int qm_grown_log2(int64_t groups, int64_t n_slots) {
  return qm_slots_wanted(groups) <= n_slots ? 0 : qm_log2_ceil(qm_slots_wanted(groups));
}
