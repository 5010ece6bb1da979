// A number that a device has, found out once per device (a process may use
// several, and one thread another than the next).
#pragma once

#include <atomic>
#include <cstdint>

namespace umapb {

class PerDevice {
public:
    template <class Find>
    int64_t get(int device, Find find) {
        if (device < 0 || device >= DEVICES) return find();
        int64_t x = known_[device].load(std::memory_order_relaxed);
        if (x == 0) {   // threads that come at once find the same
            x = find();
            known_[device].store(x, std::memory_order_relaxed);
        }
        return x;
    }

private:
    static constexpr int DEVICES = 64;
    std::atomic<int64_t> known_[DEVICES] = {};
};

}  // namespace umapb
