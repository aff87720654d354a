// Values that belong to a kernel on a device, kept for the process: function attributes
// (shared memory, cluster sizes) and what follows from them count for the device that
// was current when they were set, and engines of one process may use several.
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace d3 {

template <class T>
class PerDevice {
public:
    // The value of (device, kernel).  make(value) computes it at the first call and
    // returns whether it holds; it is asked again after a failure.
    template <class F>
    T get(int device, const void* kernel, F&& make)
    {
        std::lock_guard<std::mutex> guard(lock_);
        const auto key = std::make_pair(device, kernel);
        const auto it = values_.find(key);
        if (it != values_.end()) return it->second;
        T value{};
        if (make(value)) values_.emplace(key, value);
        return value;
    }

private:
    std::mutex lock_;
    std::map<std::pair<int, const void*>, T> values_;
};

}  // namespace d3
