// Room of the LE-list entry buffers.  A list entry lies in three parallel arrays: its
// key (target, priority), its distance and, during resident batches, the table slot of
// its pair.  k_le_batches indexes all three by the entry's number and knows one bound,
// so the bound is what the shortest of the three really holds: it is computed here from
// the buffers' bytes and not from the counts that they were asked for with.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

namespace psc {

constexpr size_t kLeKeyBytes = 8, kLeDistBytes = 4, kLeSlotBytes = 4;

// Entries to have room for before a launch: a batch adds at most `cap` (one per table
// slot), and a launch is worth at least two of the largest.
inline uint64_t le_entries_wanted(uint64_t len, uint64_t cap) { return len + 2 * cap; }

// Entries that buffers of these sizes hold.
inline uint64_t le_room(size_t key_bytes, size_t dist_bytes, size_t slot_bytes) {
  return std::min({(uint64_t)(key_bytes / kLeKeyBytes), (uint64_t)(dist_bytes / kLeDistBytes),
                   (uint64_t)(slot_bytes / kLeSlotBytes)});
}

}  // namespace psc
