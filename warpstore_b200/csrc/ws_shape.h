// Shared memory of the hash scan's CTAs, chosen on the host from the plan and the capacity alone (no CUDA here: the
// tests compile it by itself).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace ws {

// Per-CTA table of the hash scan (aggHash, ws_kern.cuh): `slots` entries, `copies` copies of the accumulators of the first
// keys, `bytes` for both, and a buffer of `spill` bytes for the rows bound for the global table.
struct HashTable {
  size_t slots = 0, bytes = 0, spill = 0;
  int copies = 1;
};
constexpr size_t kMaxHashSlots = 4096, kMinHashSlots = 64;

// cap: rows of the global table (a power of two; callers choose about twice the expected groups);
// slotBytes: a slot's key word, key number, key values and accumulators; accBytes: its accumulators;
// copyKeys, maxCopies: keys with copies, copies of each at most (powers of two);
// resident: CTAs an SM holds by the kernel's registers; tableKB: a given size of the table (0: choose);
// compiled: a compiled plan (the interpreter keeps accumulator rows).
//
// Compiled plans.  A table of the whole capacity never fills, so nearly no row leaves the chip, and a small spill buffer
// does; it is taken where it costs at most one resident CTA (COUNT and two SUMs into 500 groups: 399 us with half the
// slots, 229 us so).  Half the capacity holds the expected groups at a high load: next best under the same
// condition (COUNT and eight SUMs: 571 us against 761 us).  Else the table catches hot keys only and the scan waits
// for the global table, where resident warps count more than slots: 24 KB, and as much for the spill
// buffer (100M Zipf rows, four CTAs: 31 KB of table 4.47 ms, 24 KB 4.21 ms; two CTAs 5.4 ms).
//
// The interpreter's slot loops dominate its scan and run once more for rows that miss the table, and its stacks live in
// the L1 that shared memory leaves: a small table for few groups (aggHash goes past it where many rows miss).
//
// Wide plans keep a table: at least kMinHashSlots slots while they fit kMinTableBytes, and copies only of what
// is left (COUNT and 16 SUMs into 16 groups without a table: 8.06 ms, with one 0.32 ms).
inline HashTable hashTable(int64_t cap, size_t slotBytes, size_t accBytes, size_t copyKeys, int maxCopies, int resident,
                           size_t tableKB, bool compiled) {
  constexpr size_t K = 1024, kSm = 226 * K, kCtaReserve = K, kMinTableBytes = 48 * K;
  HashTable t;
  const size_t whole = (size_t)std::max<int64_t>(cap, (int64_t)kMinHashSlots), half = std::max(whole / 2, kMinHashSlots);
  size_t share = 0;  // shared memory of a CTA
  auto fits = [&](size_t slots, size_t spill) {
    if (slots > kMaxHashSlots) return false;
    for (int r = std::max(resident, 1); r >= std::max(resident - 1, 1); --r) {
      share = kSm / (size_t)r - kCtaReserve;
      if (slots * slotBytes + spill <= share) return true;
    }
    return false;
  };
  size_t budget;
  if (tableKB) {
    t.slots = kMaxHashSlots, t.spill = 24 * K, budget = tableKB * K;
  } else if (!compiled) {
    t.slots = std::min<size_t>(whole, 256), t.spill = 24 * K, budget = 56 * K;
  } else if (fits(whole, 8 * K)) {
    t.slots = whole, t.spill = 8 * K, budget = share - t.spill;
  } else if (fits(half, 12 * K)) {
    t.slots = half, t.spill = std::min(24 * K, share - half * slotBytes), budget = share - t.spill;
  } else {
    t.slots = kMaxHashSlots, t.spill = 24 * K, budget = 24 * K;
  }
  while (t.slots > kMinHashSlots && t.slots * slotBytes > budget) t.slots >>= 1;
  if (t.slots * slotBytes > std::max(budget, kMinTableBytes)) t.slots = 0;
  t.bytes = t.slots * slotBytes;
  if (t.slots)
    for (t.copies = maxCopies; t.copies > 1 && t.bytes + copyKeys * t.copies * accBytes > budget;) t.copies >>= 1;
  if (t.copies > 1) t.bytes += copyKeys * t.copies * accBytes;
  return t;
}

}  // namespace ws
