// entries.h -- a warp's walk over the entries [beg, end) of a tile of rows,
// 32 U at a time: lane l takes entries 32 i + l of a step, i = 0 .. U - 1.
// Counted in 64 bits: a pattern has up to 2^32 - 16 entries, and the last
// step reaches up to 32 U - 1 entries past a tile's end.
#pragma once

#include <cstdint>

#include "hd.h"

namespace pbrcm {

template <int U>
struct EntrySteps {
    uint64_t k0;   // first entry of this step
    uint32_t end;  // of the tile
    PBRCM_HD EntrySteps(uint32_t beg, uint32_t end_) : k0(beg), end(end_) {}
    PBRCM_HD bool more() const { return k0 < end; }
    PBRCM_HD void next() { k0 += 32u * U; }
    // k: the lane's entry i of this step; false past the tile's end
    PBRCM_HD bool entry(int i, uint32_t lane, uint32_t& k) const
    {
        const uint64_t e = k0 + 32u * (uint32_t)i + lane;
        k = (uint32_t)e;
        return e < end;
    }
};

}  // namespace pbrcm
