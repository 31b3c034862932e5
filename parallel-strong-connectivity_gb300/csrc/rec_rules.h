// Sizes of adjacency records (VRec) and of the searches that work on them.
#pragma once
#include <stdint.h>

namespace psc {

constexpr int kRecEdges = 6;  // targets in a record
// Largest degree of a graph that uses records: nearly all of its vertices have
// few edges beyond the record.
constexpr uint64_t kRecMaxDeg = 64;

// Resident rounds of the decomposition (ldd_low_round): entries of a wave, and waves after which
// a search is cut on a graph of this largest degree.  What is left goes to the next round, where
// its expansion begins with its first edge again, so a round has to finish the entries that its
// first wave took: every vertex is then expanded whole in some round, and the rounds come to
// an end.
constexpr int kLrWave = 12;
constexpr uint32_t kLddWaves = 10;
inline constexpr uint32_t ldd_waves(uint64_t max_deg) {
  const uint32_t need = (uint32_t)((max_deg + kRecEdges - 1) / kRecEdges);
  return need > kLddWaves ? need : kLddWaves;
}
constexpr uint32_t kLrMaxRounds = 1u << 16;  // of one launch

}  // namespace psc
