// cluster_capacity.h -- remembered answers to "how many clusters of n CTAs of a
// kernel run at once" (a GPC's SM count need not be a multiple of n), asked of
// the runtime once per device and size.  Host code only.
#pragma once

#include <atomic>

namespace b200d2 {

class ClusterCapacity {
 public:
  static constexpr int kDevices = 64, kSizes = 8;  // sizes 1 .. kSizes
  // query(): the runtime's answer, <= 0 when it has none.  Without an answer a
  // cluster counts as one (the caller's estimate then avoids it) and the next
  // call asks again.
  template <class Query>
  int get(int device, int n, Query query) {
    if (device < 0 || device >= kDevices || n < 1 || n > kSizes) {
      const int m = query();
      return m > 0 ? m : 1;
    }
    std::atomic<int>& known = known_[device][n - 1];
    int m = known.load();
    if (m > 0) return m;
    m = query();
    if (m <= 0) return 1;
    known.store(m);
    return m;
  }

 private:
  std::atomic<int> known_[kDevices][kSizes] = {};
};

}  // namespace b200d2
