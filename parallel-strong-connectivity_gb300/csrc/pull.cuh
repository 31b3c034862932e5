// In-list scans shared by the pull rounds of the reach and BFS engines.
#pragma once
#include "common.cuh"

namespace psc {

constexpr int kPullP = 4;
constexpr uint32_t kPullSolo = 64;
// CG: the bitmap was written earlier in the same launch, so it is read past L1.
template <bool CG = false>
__device__ __forceinline__ bool fb_test(const uint32_t* fb, uint32_t x) {
  return ((CG ? __ldcg(&fb[x >> 5]) : __ldg(&fb[x >> 5])) >> (x & 31)) & 1u;
}

// Solo scan of one unvisited vertex's in-list [j, lim): kPullP in-edges at a
// time until a frontier in-neighbour is found.
template <bool CG = false>
__device__ __forceinline__ bool pull_scan(const uint32_t* __restrict__ B_E,
                                          const uint32_t* fb_in, uint64_t& j,
                                          uint64_t lim) {
  bool found = false;
  while (j < lim && !found) {
    uint32_t x[kPullP];
#pragma unroll
    for (int k = 0; k < kPullP; k++) x[k] = j + k < lim ? __ldg(&B_E[j + k]) : 0xFFFFFFFFu;
    bool hit[kPullP];
#pragma unroll
    for (int k = 0; k < kPullP; k++) hit[k] = x[k] != 0xFFFFFFFFu && fb_test<CG>(fb_in, x[k]);
    uint64_t step = lim - j < (uint64_t)kPullP ? lim - j : (uint64_t)kPullP;
#pragma unroll
    for (int k = kPullP - 1; k >= 0; k--)
      if (hit[k]) {
        found = true;
        step = k + 1;
      }
    j += step;
  }
  return found;
}

// The whole warp scans the in-lists left over from the solo phase, one
// vertex at a time, 32 * kPullP in-edges per step, until a hit.
template <bool CG = false>
__device__ __forceinline__ void pull_long(const uint32_t* __restrict__ B_E,
                                          const uint32_t* fb_in, uint32_t longm,
                                          uint64_t j, uint64_t e, bool& found,
                                          unsigned long long& scanned) {
  const unsigned lane = lane_id();
  while (longm) {
    const int l = __ffs(longm) - 1;
    longm &= longm - 1;
    const uint64_t lb = __shfl_sync(kFull, j, l), le = __shfl_sync(kFull, e, l);
    bool f = false;
    uint64_t jj = lb;
    for (; jj < le && !f; jj += 32 * kPullP) {
      bool hit = false;
#pragma unroll
      for (int k = 0; k < kPullP; k++) {
        const uint64_t q = jj + k * 32 + lane;
        if (q < le) hit |= fb_test<CG>(fb_in, __ldg(&B_E[q]));
      }
      f = __any_sync(kFull, hit);
    }
    if (lane == 0) scanned += (jj < le ? jj : le) - lb;
    if (lane == (unsigned)l) found = f;
  }
}

}  // namespace psc
