// device_once.h -- state that belongs to one device of the process (a kernel's
// shared-memory attribute, the address of a __device__ variable), made at the
// first use on each device.  Host code without CUDA: the caller passes the device.
#pragma once
#include <atomic>

namespace agb {

constexpr int MAX_DEVICES = 64;

// run(dev, make): make() unless it has returned true on this device before.  A
// failure is not remembered.  Two threads may both call make(), which must allow it.
class DeviceOnce {
public:
    template <class Make> bool run(int dev, const Make& make)
    {
        if (dev < 0 || dev >= MAX_DEVICES) return make();
        if (done_[dev].load(std::memory_order_acquire)) return true;
        if (!make()) return false;
        done_[dev].store(true, std::memory_order_release);
        return true;
    }

private:
    std::atomic<bool> done_[MAX_DEVICES] = {};
};

// get(dev, make): the pointer make() returned on this device; null is not remembered.
template <typename T> class DevicePointer {
public:
    template <class Make> T* get(int dev, const Make& make)
    {
        if (dev < 0 || dev >= MAX_DEVICES) return make();
        T* p = at_[dev].load(std::memory_order_acquire);
        if (p) return p;
        p = make();
        if (p) at_[dev].store(p, std::memory_order_release);
        return p;
    }

private:
    std::atomic<T*> at_[MAX_DEVICES] = {};
};

}  // namespace agb
