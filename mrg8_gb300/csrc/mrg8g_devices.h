// mrg8g_devices.h -- one record per CUDA device.
#pragma once
#include <deque>

namespace mrg8g {

// Records by device index, made on first use.  A record never moves: callers
// keep its address across kernel launches and stream waits while other threads
// first use other devices (access itself is the owner's to lock).
template <class T>
class PerDevice {
public:
    T& at(int dev) {
        while ((int)records_.size() <= dev) records_.emplace_back();
        return records_[dev];
    }

private:
    std::deque<T> records_;
};

}  // namespace mrg8g
