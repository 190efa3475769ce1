// device_once.cuh -- set-up that is needed once per device, such as kernel attributes, which
// cudaFuncSetAttribute sets for the current device alone.
#pragma once
#include <atomic>

namespace flg {

// Which devices have been set up.  Threads may race to the first set-up (it is idempotent); a set-up that
// failed is tried again, and devices beyond the 64 remembered are set up on each call.
class DeviceOnce {
    std::atomic<unsigned long long> done_{0};

public:
    bool todo(int dev) const { return dev < 0 || dev >= 64 || !(done_.load(std::memory_order_acquire) >> dev & 1); }
    void set(int dev) {
        if (dev >= 0 && dev < 64) done_.fetch_or(1ull << dev, std::memory_order_release);
    }
};

}  // namespace flg

// runs the statements (which return from the caller on an error) once per device
#define FLG_ONCE_PER_DEVICE(...)          \
    do {                                  \
        static ::flg::DeviceOnce once_;   \
        int dev_ = 0;                     \
        FLG_CUDA(cudaGetDevice(&dev_));   \
        if (once_.todo(dev_)) {           \
            __VA_ARGS__;                  \
            once_.set(dev_);              \
        }                                 \
    } while (0)
