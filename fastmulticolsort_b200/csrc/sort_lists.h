// sort_lists.h -- how many segments the lists of a sort round hold at most.
#pragma once

#include <algorithm>
#include <cstdint>

namespace fmcs {

// Finished segments (one row, or no key bits left) of more rows than this are
// copied by tiles across the grid, smaller ones by a warp each.
constexpr uint32_t kCopySplit = 4096;

// Entries of each list.  A list's segments are disjoint, so one of segments of
// at least m rows has at most n / m of them.
struct SortListCaps {
    uint64_t large;        // segments of a radix level: more than local_max rows
    uint64_t copy;         // finished segments of up to kCopySplit rows
    uint64_t copy_large;   // finished segments of more (on-chip sizes among them: local_max may be larger)
};

// (finished segments are children of large ones, at most 256 of each a level)
inline SortListCaps sort_list_caps(uint64_t n, uint32_t local_max, uint32_t key_bits)
{
    SortListCaps c;
    c.large = n / ((uint64_t)local_max + 1) + 2;
    const uint64_t levels = (key_bits + 7) / 8;
    c.copy = std::min<uint64_t>(n, (levels + 1) * 256 * c.large) + 2;
    c.copy_large = n / (kCopySplit + 1) + 2;
    return c;
}

}  // namespace fmcs
