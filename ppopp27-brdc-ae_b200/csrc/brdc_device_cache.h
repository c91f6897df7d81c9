// brdc_device_cache.h -- what the host asks a device once and keeps: the
// occupancy of a kernel does not change while the process runs.
//
// Handles of several threads may ask first at the same time, so the query
// runs under a once flag: one thread runs it, the others wait for its answer.
#pragma once

#include <mutex>

namespace brdc {

constexpr int kMaxDevices = 64;

template <class T>
class DeviceCache {
  public:
    // query(device) -> T, run once per device; a device past the table gets
    // T{} (no occupancy).
    template <class Query>
    T get(int device, Query query) {
        if (device < 0 || device >= kMaxDevices) {
            return T{};
        }
        std::call_once(once_[device], [&]() { value_[device] = query(device); });
        return value_[device];
    }

  private:
    std::once_flag once_[kMaxDevices];
    T value_[kMaxDevices] = {};
};

} // namespace brdc
