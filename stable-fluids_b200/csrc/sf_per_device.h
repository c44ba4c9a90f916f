// sf_per_device.h -- a value found once for each device. Kernel attributes,
// and what occupancy queries say under them, belong to a device: a program may
// create contexts on several.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <mutex>

namespace sfb {

template <typename T>
class PerDevice {
public:
    // The value of the current device, made by make() at the first call. The
    // reference stays valid: nothing is ever taken out.
    template <typename Make>
    const T& get(Make make) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess) cudaGetLastError();
        std::lock_guard<std::mutex> lock(mu_);
        auto it = values_.find(device);
        if (it == values_.end()) it = values_.emplace(device, make()).first;
        return it->second;
    }

private:
    std::mutex mu_;
    std::map<int, T> values_;
};

}  // namespace sfb
