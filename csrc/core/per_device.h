// per_device.h - a value that belongs to a GPU (a limit set on it, a number asked of it), found at its first use there.
#pragma once
#include <atomic>
#include <mutex>

namespace hc {

template <typename T> class PerDevice {
  public:
    // make(&value) returns whether the value is good.  One that is not is handed back but not kept: the next call asks again.
    template <typename Make> T Get(int device, Make make)
    {
        T v{};
        if (device < 0 || device >= kDevices) {
            make(&v);
            return v;
        }
        Slot &s = slots_[device];
        if (s.ready.load(std::memory_order_acquire)) return s.value;
        std::lock_guard<std::mutex> lk(mu_);
        if (s.ready.load(std::memory_order_relaxed)) return s.value;
        if (make(&v)) {
            s.value = v;
            s.ready.store(true, std::memory_order_release);
        }
        return v;
    }

  private:
    static constexpr int kDevices = 64;
    struct Slot {
        std::atomic<bool> ready{false};
        T value{};
    };
    std::mutex mu_;
    Slot slots_[kDevices];
};

}  // namespace hc
