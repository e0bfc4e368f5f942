// cooc_plan.h -- how the fp4 co-occurrence kernel's work is cut and dealt to the CTAs.
//
// A tile of the output is summed over the transactions in double steps (512 of them), in
// runs: a CTA's part of one tile in one run is a unit, and every unit ends with the tile's
// counts added to the output, which takes as long as about 7.5 double steps.  All tiles of
// a run come before the next run; the last run is the rest.
#pragma once

#include <stdint.h>

#include <algorithm>

#ifndef SG_HOST_DEVICE
#ifdef __CUDACC__
#define SG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SG_HOST_DEVICE inline
#endif
#endif

namespace sg {

constexpr uint64_t kF4MaxSteps = (1u << 20) / 512;   // double steps summed in one accumulator
struct F4Work {
    uint32_t d, col_tiles;      // rows; 256-row column tiles
    uint64_t tiles;
    uint64_t run, last;         // double steps of a run of transactions, and of the last run
    uint64_t full;              // double steps of all tiles in the runs before the last
    uint64_t total;             // double steps of the whole product
    uint64_t share, body;       // double steps of a CTA that works below `body`
    uint64_t tail_cta;          // the CTAs from here on take the last run,
    uint64_t tail_share;        // so many double steps (whole units) each
    uint64_t ctas;
};

// A CTA's part of the work: [g0, g1).
SG_HOST_DEVICE void f4_part(const F4Work &w, uint64_t cta, uint64_t &g0, uint64_t &g1) {
    const bool tail = cta >= w.tail_cta;
    const uint64_t end = tail ? w.total : w.body, share = tail ? w.tail_share : w.share;
    g0 = tail ? w.full + (cta - w.tail_cta) * share : cta * share;
    g1 = g0 + share < end ? g0 + share : end;
}

// The tile and double step at position g of the work, and how many follow in its
// run (itself included).  Row tile bi (128 rows) meets the column tiles from
// bi / 2 on.
SG_HOST_DEVICE uint64_t f4_unit(const F4Work &w, uint64_t g, uint32_t &bi, uint32_t &bj, uint64_t &step0) {
    const uint64_t len = g < w.full ? w.run : w.last;
    const uint64_t u = g < w.full ? g / w.run : (g - w.full) / w.last;
    const uint64_t s = g < w.full ? g - u * w.run : g - w.full - u * w.last;
    const uint64_t r = g < w.full ? u / w.tiles : w.full / (w.tiles * w.run);
    uint64_t t = g < w.full ? u - r * w.tiles : u;
    step0 = r * w.run + s;
    bi = 0;
    while (t >= w.col_tiles - (bi >> 1)) {
        t -= w.col_tiles - (bi >> 1);
        ++bi;
    }
    bj = (bi >> 1) + (uint32_t)t;
    return len - s;
}

// Most units that `share` double steps in a row touch, of units `len` long; aligned: when
// shares and units start together.
inline uint64_t f4_touched(uint64_t share, uint64_t len, bool aligned) {
    if (aligned && share % len == 0) return share / len;
    if (aligned && len % share == 0) return 1;
    return share < 2 ? 1 : (share - 2) / len + 2;
}

// The plan for d rows and n_words words of transactions (both > 0).
//
// A CTA's share is an even part of the product, and a run where runs allow it: most CTAs
// then have one unit.  The rest that the last run is can be any length, though: dealt
// evenly too, a rest of one double step gave a CTA a share's worth of units, each with its
// counts to add (1,024 rows x 512 words: nine, 94 us a call; the e4m3 form took 84).  So the
// last run may be dealt in whole units to the CTAs left over, and a run may be longer
// than the even share, fewer of them; the plan whose busiest CTA has the least to do is taken,
// counting a unit as 7.5 double steps.
// Calls in us, e4m3 with 256 x 256 blocks (cooc_tc256_kernel) / everything dealt evenly / this
// plan: 1,024 rows x 512 words 84 / 94 / 31; 1,400 x 128 70 / 61 / 26; 1,024 x 2,048 123 / 70 /
// 56; 1,400 x 16,384 1,064 / 577 / 577.  An even share may be a single double step: at two,
// the least before, 126 rows x 512 words took 17.6, now 15.7, and 64 x 80 14.5 against 13.6
// of the e4m3 form, now 13.5.
inline F4Work f4_plan(uint32_t d, uint64_t n_words, uint64_t n_sm) {
    F4Work w{};
    w.d = d;
    w.col_tiles = (d + 255) / 256;
    const uint32_t row_tiles = (d + 127) / 128;
    for (uint32_t bi = 0; bi < row_tiles; ++bi) w.tiles += w.col_tiles - (bi >> 1);
    const uint64_t steps = (n_words + 7) / 8;
    w.total = w.tiles * steps;
    constexpr uint64_t kUnit = 15, kStep = 2;   // costs
    auto cut = [&](uint64_t run) {
        const uint64_t runs = (steps + run - 1) / run;
        w.run = run;
        w.last = steps - (runs - 1) * run;
        w.full = w.tiles * run * (runs - 1);
    };
    // everything dealt evenly
    const uint64_t even = (w.total + n_sm - 1) / n_sm;
    cut(std::min<uint64_t>(std::min<uint64_t>(steps, kF4MaxSteps), even));
    w.share = w.tail_share = even;
    w.body = w.total;
    w.ctas = w.tail_cta = (w.total + even - 1) / even;
    uint64_t units = f4_touched(even, w.last, w.full % even == 0);
    if (w.full) units = std::max(units, f4_touched(even, w.run, true));
    uint64_t best = kStep * even + kUnit * units;
    if (units == 1 || even > kF4MaxSteps) return w;
    // the last run in whole units, behind runs of `run`, a CTA for each of their units
    auto consider = [&](uint64_t run) {
        const uint64_t runs = (steps + run - 1) / run, last = steps - (runs - 1) * run;
        const uint64_t before = w.tiles * (runs - 1);
        if (run > kF4MaxSteps || before >= n_sm) return;
        const uint64_t each = (w.tiles + n_sm - before - 1) / (n_sm - before);
        uint64_t cost = each * (kStep * last + kUnit);
        if (before) cost = std::max(cost, kStep * run + kUnit);
        if (cost >= best) return;
        best = cost;
        cut(run);
        w.share = run;
        w.body = w.full;
        w.tail_cta = before;
        w.tail_share = each * last;
        w.ctas = before + (w.tiles + each - 1) / each;
    };
    const uint64_t runs = (steps + w.run - 1) / w.run;
    consider(w.run);
    for (uint64_t r = runs - 1; r > 0 && r + 4 >= runs; --r) consider((steps + r - 1) / r);
    return w;
}

}  // namespace sg
