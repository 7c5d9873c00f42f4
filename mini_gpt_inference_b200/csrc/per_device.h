// A kernel's limit on dynamic shared memory is a setting of the kernel on one device: what this process has raised it to, per
// kernel and device.  Plain C++ (the setter is the caller's), so that it can be tested without a GPU.
#pragma once

#include <map>
#include <mutex>
#include <utility>

class PerDeviceLimits {
  public:
    // Calls set() unless the limit of `kernel` on `device` has been raised to `bytes` or more already; a set() that fails (returns
    // other than 0) is tried again by the next call, and its answer is returned.
    template <typename Set>
    int raise(const void* kernel, int device, int bytes, Set set) {
        std::lock_guard<std::mutex> lock(mu_);
        int& held = held_[{kernel, device}];
        if (held >= bytes) return 0;
        const int e = set();
        if (e == 0) held = bytes;
        return e;
    }

  private:
    std::mutex mu_;
    std::map<std::pair<const void*, int>, int> held_;
};
