// Launch set-up that belongs to one device's context: function attributes, and what the device answers
// about a kernel's placement.  No device code.
#pragma once

#include <map>
#include <mutex>

namespace bsg {

// f() once per device, by one thread; every caller gets its result.  A call that throws leaves nothing
// behind, so the next one tries again.
class PerDevice {
public:
    template <class F>
    int get(int device, F f) {
        std::lock_guard<std::mutex> lock(mutex_);
        const auto it = values_.find(device);
        if (it != values_.end()) return it->second;
        const int value = f();
        values_.emplace(device, value);
        return value;
    }

private:
    std::mutex mutex_;
    std::map<int, int> values_;
};

}  // namespace bsg
