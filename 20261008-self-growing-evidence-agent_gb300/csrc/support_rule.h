// support_rule.h -- when an AUTO support call streams its candidates' rows.
#pragma once

#include <stdint.h>

namespace sg {

// Streaming (cand_stream_kernel) reads every row of every candidate from L2 or HBM, 256
// words a step; staging (k1_lane_tm_kernel) reads the bitmaps once per SM, a chunk of 16
// words at a time, whatever the number of candidates, and pays per box of 256 rows.  Few
// candidates stream; more than 100,000 + 30,000 a box never do (at 1,048,576 transactions
// the two meet there).  Below that line the estimates decide, in us a call, fitted to calls
// of 5,000 to 280,000 candidates of 2..8 items (streamed / staged):
//   5,000 txns x 640 rows:      100,000 60 / 46; 190,000 102 / 58
//   20,000 x 1,400:             100,000 99 / 144; 280,000 249 / 221
//   1,048,576 x 640:            50,000 1,407 / 3,525; 190,000 5,102 / 6,488 (sensor rows 6,036 / 6,066)
//   4,194,304 x 640 (336 MB):   50,000 8,917 / 14,011; 190,000 33,036 / 25,855 (sensor rows 43,971 / 24,178)
//   16,777,216 x 640 (1.3 GB):  20,000 17,372 / 49,879; 100,000 87,017 / 72,183 (112,056 / 69,529)
// A history of fewer than 256 words costs streaming a whole step, and bitmaps beyond L2 cost it
// up to 2.25 times as much a step; the staged form reads them in step by construction.
inline bool support_streams(uint64_t n_cand, uint32_t d, uint64_t n_words) {
    const uint64_t boxes = (d + 255) / 256;
    if (n_cand >= 100000 + 30000 * boxes) return false;
    constexpr double kL2 = 126e6;   // bytes
    const double bytes = (double)d * (double)n_words * 8, n = 1e-3 * (double)n_cand;   // thousands
    const double far = bytes > kL2 ? 1 + 1.25 * (1 - kL2 / bytes) : 1;
    const double streamed = 5 + n * (0.08 + 0.44 * far * (double)((n_words + 255) / 256));
    const double staged = 25 + (double)((n_words + 15) / 16) * (0.95 + 0.47 * (double)boxes + 0.0207 * n);
    return streamed <= staged;
}

}  // namespace sg
