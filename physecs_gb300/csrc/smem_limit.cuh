// smem_limit.cuh — the dynamic shared memory a kernel may use, raised as launches ask for it.
//
// The limit is an attribute of the kernel on each device, shared by all worlds of the
// process, and worlds on different threads launch at the same time with different sizes.
// So it is only ever raised, and a launch that goes on finds it at its own size or above:
// looking and setting are one step under a lock.  Plain C++, tested on the host
// (tests/test_smem_limit.py).
#pragma once
#include <mutex>

namespace psx {

class SmemLimit {
public:
    // set(bytes) changes the attribute on device `dev`, the calling thread's current one
    template <class Set>
    void raise(int dev, int bytes, Set&& set) {
        if (dev < 0 || dev >= kDevices) { set(bytes); return; }
        std::lock_guard<std::mutex> hold(lock_);
        if (bytes <= at_[dev]) return;
        set(bytes);
        at_[dev] = bytes;
    }

private:
    static constexpr int kDevices = 64;
    std::mutex lock_;
    int at_[kDevices] = {};
};

}  // namespace psx
