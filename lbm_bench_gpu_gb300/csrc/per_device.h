// per_device.h -- host values kept per device ordinal (no CUDA).
#pragma once

#include <atomic>

namespace lbm {

constexpr int kMaxDevices = 64;

// A value that belongs to a device: a kernel's attributes, its resident blocks
// and the SM count differ between the devices of a process, so an answer found
// on one must not be taken for another.  Safe with several threads: those that
// ask for a device's value for the first time at once each find it.
template <typename T>
class PerDevice {
public:
    // The value of `device`; find() gives it (true) or fails (false: nothing is
    // kept, and the next call tries again).
    template <typename Find>
    bool get(int device, T &out, Find &&find)
    {
        const bool kept = device >= 0 && device < kMaxDevices;
        if (kept && slots_[device].known.load(std::memory_order_acquire)) {
            out = slots_[device].value.load(std::memory_order_relaxed);
            return true;
        }
        if (!find(out)) return false;
        if (kept) {
            slots_[device].value.store(out, std::memory_order_relaxed);
            slots_[device].known.store(true, std::memory_order_release);
        }
        return true;
    }

private:
    struct Slot {
        std::atomic<bool> known{false};
        std::atomic<T> value{T()};
    };
    Slot slots_[kMaxDevices];
};

}  // namespace lbm
