// support_rule.h -- the kernel of an AUTO support call.
#pragma once

#include <stdint.h>

#ifndef SG_HOST_DEVICE
#ifdef __CUDACC__
#define SG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SG_HOST_DEVICE inline
#endif
#endif

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

// Whether a call that does not stream looks if its data are sparse enough for pair groups
// (kernels_pair.cu), which costs it 40 us when they are not: calls of 2e9 candidate-words
// (2.4 ms) or more, of enough candidates.  Groups are counted 32 at a time, two units of
// work each, by 32 warps an SM: few candidates fill few groups, and few rows make few
// pairs, whose groups are of eight, so the line rises below 256 rows.  1,048,576 sparse
// transactions, in us (k1_lane_tm_kernel / pair groups):
//   64 rows:    130,000 candidates 4,116 / 8,144; 400,000 9,545 / 10,581; 600,000 13,410 / 11,926
//   128 rows:   130,000 4,108 / 6,155; 400,000 9,545 / 10,191; 600,000 13,415 / 12,229
//   180 rows:   200,000 5,696 / 6,414; 300,000 7,649 / 7,978; 400,000 9,547 / 8,682
//   256 rows:   130,000 4,116 / 4,379; 200,000 5,695 / 5,077; 1,000,000 20,991 / 12,910
//   1,024 rows: 130,000 5,524 / 5,914; 200,000 7,110 / 6,767; 1,000,000 22,349 / 12,855
inline bool support_pairs(uint64_t n_cand, uint32_t d, uint64_t n_words) {
    const uint64_t least = 160000 + (d < 256 ? 2000 * (uint64_t)(256 - d) : 0);
    return n_cand >= least && n_cand * n_words >= 2000000000ull;
}

// The gate of such a call, on the device: whether sampled candidates are too dense for pair
// groups.  live: how many of the sampled 32-bit words of their first two rows' ANDs hold a
// bit; items: the candidates' items, once per 32 words sampled.
//
// Up to a sixth of live words pays for candidates of four items and more.  Shorter ones have
// few further rows to skip, and every word where the first four rows are left is counted on a
// slow path: all live words for two items.  A pair group costs more the fewer candidates share
// it, so the line falls below 400 candidates a row.  1,048,576 transactions, every row with the
// same share of bits, in us (k1_lane_tm_kernel / pair groups):
//   600,000 of 2 items:    300 rows, 1% 7,445 / 5,968, 4% 7,447 / 10,859; 1,024 rows, 2% 8,352 / 10,351
//   600,000 of 3 items:    300 rows, 4% 9,370 / 7,196; 1,024 rows, 4% 10,264 / 9,966, 6% 10,266 / 12,121
//   250,000 of 3 items:    300 rows, 4% 5,117 / 4,757; 1,024 rows, 2% 6,016 / 5,657, 4% 6,016 / 6,674
//   600,000 of 4 items:    1,024 rows, 6% 12,133 / 10,010, 8% 12,133 / 12,140
//   600,000 of 3..8 items: 1,024 rows, 7% (14% of the words live) 14,801 / 11,995, 10% 14,800 / 16,392
SG_HOST_DEVICE bool pair_dense(uint32_t live, uint32_t sampled, uint32_t items, uint64_t n_cand, uint32_t d) {
    if (sampled == 0) return false;
    const float k = 32.f * (float)items / (float)sampled;
    float line = 1.f / 6;
    if (k <= 2) line = 0.0035f;
    else if (k < 3) line = 0.0035f + 0.0565f * (k - 2) * (k - 2);
    else if (k < 4) line = 0.06f + 0.1067f * (k - 3);
    const float shared = (float)n_cand / (400.f * (float)d);
    if (shared < 1) line *= shared;
    return (float)live > line * (float)sampled;
}

}  // namespace sg
