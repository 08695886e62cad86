// The dynamic shared-memory limit that has been asked for one kernel, per device.  No CUDA in here: the caller passes
// the driver call that sets it.
#pragma once
#include <atomic>
#include <mutex>
#include <stddef.h>

namespace pl {

constexpr int MAX_DEVICES = 64;

// Setting the limit is a driver call, its effect lasts as long as the context, and it lowers a limit as readily as it
// raises one.  So it is set only when a call needs more than any call before it, by one thread at a time, and looked at
// again once it is that thread's turn: a thread that saw no limit yet must not put a small one over another's large one
// that a launch relies on.
class SmemLimit {
public:
    // set(bytes): 0 on success, else the error that raise() returns
    template <typename Set>
    int raise(int device, size_t bytes, Set set) {
        const bool cached = device >= 0 && device < MAX_DEVICES;
        if (cached && granted_[device].load(std::memory_order_acquire) >= bytes + 1) return 0;
        std::lock_guard<std::mutex> lock(mutex_);
        if (cached && granted_[device].load(std::memory_order_relaxed) >= bytes + 1) return 0;
        const int rc = set(bytes);
        if (rc == 0 && cached) granted_[device].store(bytes + 1, std::memory_order_release);
        return rc;
    }

private:
    std::atomic<size_t> granted_[MAX_DEVICES] = {};   // bytes + 1; 0: nothing asked for yet
    std::mutex mutex_;
};

}  // namespace pl
