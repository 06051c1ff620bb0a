// Limits that hold per device and kernel and are raised on demand: the dynamic
// shared memory a kernel may be launched with (set_smem).
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace arecgb {

// raise(device, kernel, bytes, set) calls set(bytes) when the limit is below `bytes` and
// keeps it if that returns 0.  A limit is never lowered: it is process-wide, so a
// caller on another host thread with a smaller size cannot drop it between this
// caller's raise and its launch.
class RaisedLimits {
  public:
    template <typename F>
    int raise(int device, const void *kernel, size_t bytes, F &&set) {
        std::lock_guard<std::mutex> lk(mu);
        size_t &cur = limit[{device, kernel}];
        if (bytes <= cur) return 0;
        if (const int rc = set(bytes)) return rc;
        cur = bytes;
        return 0;
    }

  private:
    std::mutex mu;
    std::map<std::pair<int, const void *>, size_t> limit;
};

}  // namespace arecgb
