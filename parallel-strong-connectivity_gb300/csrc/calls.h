// Calls at work on a device, over all handles and threads of the process.
//
// A resident launch holds its SMs for a whole phase of a solve, and mostly waits.  Alone it takes
// all of them; launches of several calls that all did would run one after the other.  So
// a launch takes the device's SMs divided by the calls at work, but never fewer than
// kResidentFloor, behind which launches queue.  Nothing else depends on the count: the
// results are the same on any number of SMs.
// Solves per second, a thread and a handle each, 1 / 4 / 8 / 16 threads: R-MAT 2^16 in rounds from
// the host 1,390 / 4,170 / 6,060 / 7,700, every launch on all SMs 3,130 / 4,530 / 4,720 / -, shares
// 3,150 / 11,600 / 15,400 / 16,300; kNN 10^6 255 / 772 / 935 / 1,010, 530 / 658 / 664 / -, 530 /
// 1,610 / 1,840 / 2,010.  Floors, 16 threads: R-MAT 2^19 with 4 SMs 2,950, 32 6,100, 48 5,870 (from
// the host 4,510); kNN 10^6 1,630, 2,010, 1,600.  (Shares by the graphs' edges instead of equal
// ones: no difference in a stream of requests of 10^3 to 10^7 vertices.)
#pragma once
#include <algorithm>
#include <atomic>

namespace psc {

constexpr int kResidentFloor = 32;
constexpr int kCallDevices = 64;
inline std::atomic<int> g_calls[kCallDevices];

// One call, from its first work to its return on whatever path.
class CallScope {
 public:
  explicit CallScope(int device)
      : n_(device >= 0 && device < kCallDevices ? &g_calls[device] : nullptr) {
    if (n_) n_->fetch_add(1, std::memory_order_relaxed);
  }
  ~CallScope() {
    if (n_) n_->fetch_sub(1, std::memory_order_relaxed);
  }
  CallScope(const CallScope&) = delete;
  CallScope& operator=(const CallScope&) = delete;

 private:
  std::atomic<int>* n_;
};

inline int calls_at_work(int device) {
  if (device < 0 || device >= kCallDevices) return 1;
  return std::max(1, g_calls[device].load(std::memory_order_relaxed));
}

// SMs of a resident launch on a device of num_sms.
inline int resident_share(int num_sms, int calls) {
  return std::min(num_sms, std::max(num_sms / std::max(1, calls), kResidentFloor));
}

}  // namespace psc
