// Hand-over of vertices between the warps of a search without rounds (reach.cu): how many
// vertices a warp takes and gives away at a time.
//
// The slots have room for every vertex once, and for kAsyncSlack more.  A vertex is put
// into them when a search gives it away, and it was claimed just once, so it comes there a
// second time only if it was taken from them and then put back unexpanded.  That must not
// happen while searches give vertices away (nothing would bound how often), only when a
// launch stops, once per warp.  So whatever a ring holds of taken vertices after a wave lies
// among the kAsyncKeep entries at its front, which are kept:
//   any degrees:  up to 32 taken, 16 or more of them expanded by the first wave;
//   low degrees:  up to kAsyncTakeLow taken, kLowWave of them expanded by the first wave, and
//                 in front of the rest up to kLowWave entries that came back with targets left.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define PSC_RULE __host__ __device__ __forceinline__
#else
#define PSC_RULE inline
#endif

namespace psc {

constexpr uint32_t kAsyncKeep = 16;
constexpr uint32_t kAsyncTake = 32;      // any degrees (k_reach_async)
constexpr uint32_t kAsyncFewWave = 16;   // its smallest wave
constexpr uint32_t kLowWave = 12;        // low degrees (k_reach_async_low)
constexpr uint32_t kAsyncTakeLow = 16;
static_assert(kAsyncTake - kAsyncFewWave <= kAsyncKeep, "taken vertices are kept");
static_assert(kAsyncTakeLow - kLowWave + kLowWave <= kAsyncKeep,
              "taken vertices and entries that came back are kept");
// Vertices put into the slots a second time when a launch stops: what a warp had taken.
constexpr uint64_t kAsyncSlack = 1u << 18;
constexpr uint64_t kAsyncMaxWarps = kAsyncSlack / kAsyncTake;

// Slots prepared for one launch, after `full` launches that ran out of them: searches of kNN
// 10^7 and a 4096^2 grid use 0.2 to 2 % of n (clearing n of them, 64 MB, took 20 of the 180 us
// of a search of a few vertices), and every frontier has room four times.
constexpr uint64_t kAsyncSlots = 1ull << 24;
PSC_RULE uint32_t async_slots(uint64_t n, uint64_t frontier, uint32_t full) {
  uint64_t want = n / 16 > (1u << 18) ? n / 16 : (1u << 18);
  if (full) want = full > 2 ? kAsyncSlots : want << (4 * full);
  if (want < 4 * frontier) want = 4 * frontier;
  if (want > kAsyncSlots) want = kAsyncSlots;
  return (uint32_t)(want < n ? want : n);
}

// Vertices that an idle warp asks for: one, or its share of the backlog.
PSC_RULE uint32_t async_take(int32_t backlog, uint32_t warps, uint32_t most) {
  if (backlog <= (int32_t)warps) return 1;
  const uint32_t share = (uint32_t)backlog / warps;
  return share < most ? share : most;
}

// Vertices of the `held` queued ones that go to `hungry` idle warps.
PSC_RULE uint32_t async_give(int32_t hungry, uint32_t held) {
  if (hungry <= 0 || held <= kAsyncKeep) return 0;
  return held - kAsyncKeep < (uint32_t)hungry ? held - kAsyncKeep : (uint32_t)hungry;
}

}  // namespace psc
