// window_sizes.h -- what a warp's workspace of the batched window miner holds.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace sg {

struct WindowSizes {
    uint64_t list_cap;   // places of the task's list (vertical search) or entries of its stack
    uint64_t v_words;    // 32-bit words of a vertical row, whole 16-byte pieces (0: horizontal search)
};

// max_len: transactions of the longest window.  The vertical search lists the task's
// transactions (4 bytes each); the horizontal one stacks every level's database as masks.
// Lists end just below 2^30 places, and a longer window is mined on the handle instead,
// so the rows end there too: wvtask_kernel counts the words of its 128 rows in 32 bits.
inline WindowSizes window_sizes(uint64_t max_len, bool vertical) {
    WindowSizes s;
    s.list_cap = std::min<uint64_t>(std::max<uint64_t>(8192, (vertical ? 1 : 2) * max_len + 1024) & ~3ull,
                                    (1ull << 30) - (1ull << 14));
    s.v_words = vertical ? ((std::min(max_len, s.list_cap) + 31) / 32 + 1 + 3) & ~3ull : 0;
    return s;
}

}  // namespace sg
