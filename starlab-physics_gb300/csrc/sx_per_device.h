// A host-side value of its own for each CUDA device, found on the first call made
// with that device current: kernel attributes (shared-memory limit, cluster sizes)
// and what occupancy queries tell belong to a device, not to the process.
#pragma once
#include <mutex>

namespace sx {

class PerDevice {
  public:
    // find() runs once per device, under the lock; for a device out of range on
    // every call
    template <typename Find>
    int get(int device, Find find) {
        if (device < 0 || device >= kDevices) return find();
        std::lock_guard<std::mutex> lock(mutex_);
        if (!known_[device]) {
            value_[device] = find();
            known_[device] = true;
        }
        return value_[device];
    }

  private:
    static constexpr int kDevices = 64;
    std::mutex mutex_;
    bool known_[kDevices] = {};
    int value_[kDevices] = {};
};

}  // namespace sx
