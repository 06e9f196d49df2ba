// Search of a sorted near list that is read in tiles.
#pragma once

#include "pair_rules.cuh"

namespace hsb {

// First place in trial[0 .. count) whose panel is not below s.
HS_HD uint32_t nearTilePlace(const uint32_t *trial, uint32_t count, uint32_t s) {
    uint32_t lo = 0, hi = count;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) / 2;
        if (trial[mid] < s)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Whether a panel that is not in this tile is in no tile of the list. Exactly one
// tile says so of a missing panel: the one it would lie inside, or the one it
// would lie before (after the previous tile's last panel `previous`), or the last.
HS_HD bool nearTileMisses(uint32_t place, uint32_t count, bool first, bool last, uint32_t previous, uint32_t s) {
    if (place == 0)
        return first || s > previous;
    return place < count || last;
}

}  // namespace hsb
