// smem_limits.h -- the dynamic shared-memory limits raised so far.
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace fair {

// The runtime keeps a kernel's limit per device, so a limit raised on one
// device says nothing about another. Never lowers a limit: launches of one
// kernel with different sizes may be under way on several threads.
class SmemLimits {
    std::mutex mu;
    std::map<std::pair<int, const void *>, std::size_t> top;

  public:
    // raise(): sets the limit of `kernel` on the current device `device`, 0 if done.
    template <class Raise> int allow(int device, const void *kernel, std::size_t bytes, Raise raise) {
        std::lock_guard<std::mutex> lock(mu);
        const auto key = std::make_pair(device, kernel);
        const auto it = top.find(key);
        if (it != top.end() && bytes <= it->second) return 0;
        const int e = raise();
        if (e == 0) top[key] = bytes;
        return e;
    }
};

}  // namespace fair
