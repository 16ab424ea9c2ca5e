// Where the per-pixel lists of a view lie in its part of the list buffer (host side of the inspection calls; plain C++).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <utility>
#include <vector>

namespace trips
{
// True when the lists [starts[i], starts[i] + counts[i]) fill [0, n_frags) exactly: no list leaves the range, no two overlap and
// no slot belongs to none of them.  Their order does not matter.
inline bool lists_cover(const uint32_t* starts, const uint32_t* counts, size_t n_lists, uint64_t n_frags)
{
    std::vector<std::pair<uint32_t, uint32_t>> lists;
    for (size_t i = 0; i < n_lists; ++i)
        if (counts[i]) lists.emplace_back(starts[i], counts[i]);
    std::sort(lists.begin(), lists.end());
    uint64_t next = 0;
    for (const auto& [start, count] : lists)
    {
        if (start != next) return false;
        next += count;
    }
    return next == n_frags;
}
}  // namespace trips
