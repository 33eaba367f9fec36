// cpab_occupancy.h -- resident CTAs per SM, remembered per kernel, block size
// and shared memory.  (Host only.)
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>

namespace cpab {

// Asked again on every launch, with as many sizes of shared memory as a program
// has launch sizes (FP64 scratch follows the tile, which follows the points: up
// to 32 per space), so it grows with them; a bound far above that starts it
// anew.  Safe with several threads.
class OccupancyCache {
public:
    static constexpr size_t kMost = 4096;

    template <class Query>  // int query(): CTAs per SM, called when not yet known
    int get(const void *kern, int block, size_t smem, Query &&query)
    {
        std::lock_guard<std::mutex> lock(mu_);
        const auto key = std::make_tuple(kern, block, smem);
        const auto at = known_.find(key);
        if (at != known_.end()) return at->second;
        if (known_.size() >= kMost) known_.clear();
        return known_[key] = query();
    }

private:
    std::mutex mu_;
    std::map<std::tuple<const void *, int, size_t>, int> known_;
};

}  // namespace cpab
