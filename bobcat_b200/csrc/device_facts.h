// Whole numbers that depend on the device alone (its SMs, the clusters of a kernel that fit), looked up when first
// asked for and kept per device. Launches of several threads ask at once: each look-up gives the same number, so whoever comes
// first may store it.
#pragma once

#include <atomic>

namespace bc {
namespace k {

template <int N>
class DeviceFacts {
  public:
    // Fact `i` of `device`; `look_up(&value)` gives it (positive), or false, which is returned and not kept.
    template <typename F>
    bool get(int device, int i, F&& look_up, int* out) {
        if (device < 0 || device >= kDevices) return look_up(out);
        std::atomic<int>& kept = values_[device][i];
        *out = kept.load(std::memory_order_relaxed);
        if (*out > 0) return true;
        if (!look_up(out)) return false;
        kept.store(*out, std::memory_order_relaxed);
        return true;
    }

  private:
    static constexpr int kDevices = 64;
    std::atomic<int> values_[kDevices][N] = {};
};

}  // namespace k
}  // namespace bc
