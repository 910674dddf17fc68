// Dynamic shared memory of the walk blocks: its limit, the widest block that stays
// within it, and the kernels' opt-ins above the 48 KB every kernel may use.
// Host code without CUDA's types, so that it runs where there is no GPU.
#pragma once

#include <cstddef>
#include <mutex>
#include <set>
#include <utility>

namespace sph3 {

constexpr size_t kMaxBlockSmem = 200 * 1024;

// The widest block (or team) of at most `warps`: the deepest stacks leave room
// for fewer warps than the tables of team sizes would take.
inline int warps_that_fit(int warps, size_t warp_bytes) {
    while (warps > 1 && warps * warp_bytes > kMaxBlockSmem) warps /= 2;
    return warps;
}

// Calls set(kernel, bytes), which returns 0 on success, once per kernel and
// device: an opt-in holds on the device that was current when it was made.
class SmemOptIn {
  public:
    template <class Set>
    int once(int device, const void *kernel, Set set) {
        std::lock_guard<std::mutex> lk(mu_);
        if (done_.count({device, kernel})) return 0;
        const int rc = set(kernel, (int)kMaxBlockSmem);
        if (rc == 0) done_.insert({device, kernel});
        return rc;
    }

  private:
    std::mutex mu_;
    std::set<std::pair<int, const void *>> done_;
};

}  // namespace sph3
