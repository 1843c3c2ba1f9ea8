// A value per device, made on first use: kernel attributes belong to the device
// that is current when they are set, and so do the counts of what runs at once.
#pragma once

#include <map>
#include <mutex>

namespace nricp_b200 {

template <typename T>
class PerDevice {
public:
    // The device's value; `make` runs once per device and what it throws is not
    // kept.  References stay valid.
    template <typename Make>
    const T& of(int device, Make make) {
        std::lock_guard<std::mutex> lock(mu_);
        auto it = values_.find(device);
        if (it == values_.end()) it = values_.emplace(device, make()).first;
        return it->second;
    }

private:
    std::mutex mu_;
    std::map<int, T> values_;
};

}  // namespace nricp_b200
