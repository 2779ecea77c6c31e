// Resident CTAs per SM of a kernel, kept per device once the driver has answered
// (a query of its own took 0.5 us of every frame).  An answer that failed is not
// kept: the caller gets 1 for this launch and the next one asks again.
#pragma once

#include <atomic>

namespace cr {

struct OccupancyCache {
    static constexpr int kDevices = 64;
    std::atomic<int> per_sm[kDevices] = {};  // 0: not known
};

// query(): CTAs per SM on `device`, the current one, or 0 where it failed.
template <typename Query>
int cached_occupancy(OccupancyCache& cache, int device, Query query) {
    const bool keep = device >= 0 && device < OccupancyCache::kDevices;
    int n = keep ? cache.per_sm[device].load(std::memory_order_relaxed) : 0;
    if (n > 0) return n;
    n = query();
    if (n <= 0) return 1;
    if (keep) cache.per_sm[device].store(n, std::memory_order_relaxed);
    return n;
}

}  // namespace cr
