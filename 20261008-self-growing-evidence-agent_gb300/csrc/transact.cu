// transact.cu -- sensor stream -> transactions on the GPU.
//
// Reference: code/pipeline/skab_spike.py
//   fit_bins            :38-52  per-sensor quantiles at linspace(0, 1, n_bins+1)
//                               (numpy "linear" method), unique edges, a
//                               constant column gets [e0 - 0.5, e0 + 0.5]
//   bin_index           :55-58  searchsorted(edges, v, side="right") - 1, clamped
//   window_transactions :62-80  windows s = 0, stride, ..., s + window <= n; the
//                               median of each sensor over the window picks one
//                               item per sensor; the label is the window's max
// Items are dense ids sensor * n_bins + bin.
//
// Device work: the row-major [n, S] matrix is transposed to columns; every
// order statistic numpy's quantile needs is found exactly by a 6-pass MSD
// radix select over order-preserving 64-bit keys of the doubles; the quantile interpolation runs in explicitly rounded
// double intrinsics, so no multiply-add is fused and the edges are the same
// doubles numpy computes; one thread per (window, sensor) sorts its window
// and bins the median.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "engine.h"

namespace sg {

namespace {

constexpr uint32_t kMaxWindow = 256;

__device__ __forceinline__ uint64_t dkey(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    return (b >> 63) ? ~b : (b | (1ull << 63));
}
__device__ __forceinline__ double dkey_inv(uint64_t k) {
    const uint64_t b = (k >> 63) ? (k & ~(1ull << 63)) : ~k;
    return __longlong_as_double((long long)b);
}

// Row-major [n, S] -> columns, through a 64 x 32 tile: both sides move whole
// 256-byte runs.
constexpr uint32_t kTileRows = 64, kTileCols = 32;
__global__ void __launch_bounds__(256) to_columns_kernel(const double *__restrict__ rows, uint64_t n, uint32_t S,
                                                         double *__restrict__ cols, uint32_t *__restrict__ nan_count) {
    __shared__ double tile[kTileCols][kTileRows + 1];
    const uint32_t c0 = blockIdx.y * kTileCols;
    const uint32_t cx = threadIdx.x & 31, ry = threadIdx.x >> 5;     // load: 32 columns x 8 rows a step
    const uint32_t rx = threadIdx.x & 63, cy = threadIdx.x >> 6;     // store: 64 rows x 4 columns a step
    uint32_t bad = 0;
    for (uint64_t r0 = (uint64_t)blockIdx.x * kTileRows; r0 < n; r0 += (uint64_t)gridDim.x * kTileRows) {
#pragma unroll
        for (uint32_t r = ry; r < kTileRows; r += 8)
            if (r0 + r < n && c0 + cx < S) {
                const double v = rows[(r0 + r) * S + c0 + cx];
                bad += v != v;
                tile[cx][r] = v;
            }
        __syncthreads();
#pragma unroll
        for (uint32_t c = cy; c < kTileCols; c += 4)
            if (r0 + rx < n && c0 + c < S) cols[(uint64_t)(c0 + c) * n + r0 + rx] = tile[c][rx];
        __syncthreads();
    }
    if (bad) atomicAdd(nan_count, bad);
}

// Order statistics of every sensor by an MSD radix select whose passes run on
// the whole chip: a pass histograms the next kDigit key bits of the values
// under each still open prefix (CTAs own runs of a column and add their
// shared-memory histograms to global ones), and a select step moves every rank
// to its digit.  Ranks with the same prefix share a histogram.
//
// After the third pass few values are left under the open prefixes (22 bits), so
// that pass also lists them, and the others read the list; a column whose values
// crowd under them (ties) has no list and is read whole.
//
// Bound: HBM/L2, one read of the columns per pass and group of prefixes, and
// shared-memory atomics.  1,000,000 rows x 21 sensors, 13 ranks: 0.36 ms for the
// six passes (0.65 without lists) against 7.3 ms for one CTA per (sensor, rank)
// and eight passes; the transpose 68 us (143 us when every lane stored to its own
// column).
constexpr int kDigitBits = 11;
constexpr uint32_t kDigits = 1u << kDigitBits;
constexpr int kPasses = 6;            // 5 x 11 + 9 bits
constexpr uint32_t kHistGroup = 6;    // prefixes counted at a time: 48 KB of histograms
constexpr int kHistThreads = 512;
constexpr int kListPass = 2;          // the pass that lists the values under the open prefixes
constexpr uint32_t kListBlock = 4096; // values a CTA lists at most: more, and the column has no list
__host__ __device__ constexpr int digit_shift(int pass) {
    return 64 - kDigitBits * (pass + 1) > 0 ? 64 - kDigitBits * (pass + 1) : 0;
}

// Per sensor: R ranks, ascending.  prefix[r], left[r] (rank inside the prefix),
// group[r] (index of its prefix among the distinct ones), distinct prefixes
// open[0 .. n_open).
struct SelectState {
    uint64_t *prefix, *left, *open;
    uint32_t *group, *n_open;
    // values under the open prefixes after kListPass, as keys: list_n[s] of them at list + s * cap,
    // or, above cap, none (cap 0: no lists)
    uint64_t *list;
    uint32_t *list_n;
    uint32_t cap;
};

__global__ void select_init_kernel(SelectState st, uint32_t S, uint32_t R, const uint64_t *__restrict__ ranks) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S * R; i += gridDim.x * blockDim.x) {
        st.prefix[i] = 0;
        st.left[i] = ranks[i % R];
        st.group[i] = 0;
        st.open[i] = 0;
        if (i < S) {
            st.n_open[i] = 1;
            if (st.cap) st.list_n[i] = 0;
        }
    }
}

// blockIdx.x: run of rows; blockIdx.y: sensor.  hist[s][group][digit].
// kMode: the columns are read; read and the values found listed; or the lists read
// where there are lists.
enum SelectMode : int { SELECT_READ, SELECT_LIST, SELECT_FROM_LIST };
template <int kMode>
__global__ void __launch_bounds__(kHistThreads) select_hist_kernel(const double *__restrict__ cols, uint64_t n,
                                                                   SelectState st, uint32_t R, int pass,
                                                                   uint32_t *__restrict__ hist) {
    __shared__ uint32_t h[kHistGroup * kDigits];
    __shared__ uint32_t listed, list_at;
    extern __shared__ uint64_t found[];   // kListBlock keys in kListPass
    const uint32_t s = blockIdx.y;
    constexpr bool listing = kMode == SELECT_LIST;
    bool from_list = false;
    const uint64_t *list = nullptr;
    const uint32_t n_open = st.n_open[s];
    const int shift = digit_shift(pass), up = pass ? digit_shift(pass - 1) : 64;
    const uint32_t digits = 1u << (up - shift);
    const double *col = cols + (uint64_t)s * n;
    if (kMode == SELECT_FROM_LIST) {
        const uint32_t have = st.list_n[s];
        from_list = have <= st.cap;
        list = st.list + (uint64_t)s * st.cap;
        if (from_list) n = have;
    }
    if (listing && threadIdx.x == 0) listed = 0;
    const uint64_t per = (n + gridDim.x - 1) / gridDim.x;
    const uint64_t i0 = min(n, blockIdx.x * per), i1 = min(n, i0 + per);
    for (uint32_t g0 = 0; g0 < n_open; g0 += kHistGroup) {
        const uint32_t ng = min(kHistGroup, n_open - g0);
        uint64_t want[kHistGroup];
#pragma unroll
        for (uint32_t g = 0; g < kHistGroup; ++g) want[g] = st.open[(uint64_t)s * R + g0 + min(g, ng - 1)];
        for (uint32_t i = threadIdx.x; i < ng * kDigits; i += kHistThreads) h[i] = 0;
        __syncthreads();
        for (uint64_t i = i0 + threadIdx.x; i < i1; i += kHistThreads) {
            const uint64_t key = kMode == SELECT_FROM_LIST && from_list ? list[i] : dkey(col[i]);
            const uint64_t pre = pass ? key >> up : 0;
            uint32_t at = kHistGroup;
#pragma unroll
            for (int g = kHistGroup - 1; g >= 0; --g) at = pre == want[g] ? (uint32_t)g : at;
            if (at < ng) {
                atomicAdd(&h[at * kDigits + ((uint32_t)(key >> shift) & (digits - 1))], 1u);
                if (listing && listed < kListBlock) {
                    const uint32_t to = atomicAdd(&listed, 1u);
                    if (to < kListBlock) found[to] = key;
                }
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < ng * kDigits; i += kHistThreads)
            if (h[i]) atomicAdd(&hist[((uint64_t)s * R + g0) * kDigits + i], h[i]);
        __syncthreads();
    }
    if (!listing) return;
    const uint32_t m = listed;
    // a full CTA may have left values out: the top bit then says that there is no list
    if (threadIdx.x == 0)
        list_at = m < kListBlock ? atomicAdd(&st.list_n[s], m) : atomicOr(&st.list_n[s], 0x80000000u);
    __syncthreads();
    const uint64_t to = list_at;
    if (m < kListBlock)
        for (uint32_t i = threadIdx.x; i < m; i += kHistThreads)
            if (to + i < st.cap) st.list[(uint64_t)s * st.cap + to + i] = found[i];
}

// One CTA per sensor, a warp per rank: the digit that holds the rank; then the
// distinct prefixes of the next pass, and the histograms cleared for it.  The
// last pass writes the statistics.  A lane's 64 counts are loaded at once and kept
// (11 us a pass; 22 us with 8 warps and counts read one by one).
constexpr int kStepThreads = 512;
__global__ void __launch_bounds__(kStepThreads) select_step_kernel(SelectState st, uint32_t R, int pass,
                                                          uint32_t *__restrict__ hist, double *__restrict__ out,
                                                          uint32_t out_stride) {
    const uint32_t s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int shift = digit_shift(pass), up = pass ? digit_shift(pass - 1) : 64;
    uint64_t *prefix = st.prefix + (uint64_t)s * R, *left = st.left + (uint64_t)s * R, *open = st.open + (uint64_t)s * R;
    uint32_t *group = st.group + (uint64_t)s * R;
    uint32_t *hs = hist + (uint64_t)s * R * kDigits;
    const uint32_t n_open = st.n_open[s];
    constexpr uint32_t kMine = kDigits / 32;   // counts per lane
    for (uint32_t r = warp; r < R; r += kStepThreads / 32) {
        const uint4 *h = reinterpret_cast<const uint4 *>(hs + (uint64_t)group[r] * kDigits + lane * kMine);
        uint32_t c[kMine], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < kMine / 4; ++i) {
            const uint4 v = h[i];
            c[4 * i] = v.x, c[4 * i + 1] = v.y, c[4 * i + 2] = v.z, c[4 * i + 3] = v.w;
        }
#pragma unroll
        for (uint32_t i = 0; i < kMine; ++i) sum += c[i];
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        uint64_t k = left[r];
        const uint64_t below = incl - sum;
        __syncwarp();
        if (k >= below && k < incl) {   // exactly one lane
            k -= below;
            uint32_t d = 0;
            bool open_at = true;        // the counts before the rank's digit are taken off
#pragma unroll
            for (uint32_t i = 0; i < kMine; ++i) {
                open_at = open_at && k >= c[i];
                if (open_at) {
                    k -= c[i];
                    ++d;
                }
            }
            prefix[r] = (prefix[r] << (up - shift)) | (lane * kMine + d);
            left[r] = k;
            if (pass == kPasses - 1) out[(uint64_t)s * out_stride + r] = dkey_inv(prefix[r]);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n_open * kDigits; i += blockDim.x) hs[i] = 0;
    if (threadIdx.x == 0) {
        uint32_t m = 0;
        for (uint32_t r = 0; r < R; ++r) {   // ranks ascend, so their prefixes do
            if (r == 0 || prefix[r] != prefix[r - 1]) open[m++] = prefix[r];
            group[r] = m - 1;
        }
        st.n_open[s] = m;
    }
}

// numpy linear quantile for quantile q of sensor s: lo/hi are the order
// statistics at floor(h) and floor(h)+1 (both the last one when h >= n-1),
// gamma = h - floor(h) (h - (-1) above the bounds, where lo == hi), and
// lerp(a, b, g) = g >= 0.5 ? b - (b - a) * (1 - g) : a + (b - a) * g.
__global__ void quantile_kernel(const double *__restrict__ stats, uint32_t R, const uint32_t *__restrict__ lo_idx,
                                const uint32_t *__restrict__ hi_idx, const double *__restrict__ gamma, uint32_t nq,
                                uint32_t S, double *__restrict__ edges) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq * S) return;
    const uint32_t s = i / nq, q = i - s * nq;
    const double a = stats[(uint64_t)s * R + lo_idx[q]];
    const double b = stats[(uint64_t)s * R + hi_idx[q]];
    const double g = gamma[q];
    const double diff = __dsub_rn(b, a);
    double v = __dadd_rn(a, __dmul_rn(diff, g));
    if (g >= 0.5) v = __dsub_rn(b, __dmul_rn(diff, __dsub_rn(1.0, g)));
    edges[i] = v;
}

// numpy's median of `window` values `step` elements apart (the mean of the two
// middle values for an even count).  W > 0: the values, as ordered integer keys
// padded to W, pass through Batcher's odd-even merge sort in registers (an
// array indexed by a loop lives in local memory, and double compares run on the
// narrow FP64 pipe); W = 0, for longer windows: insertion sort.
// 66,665 windows of 30 rows x 21 sensors: 0.20 ms (insertion sort 1.26 ms).
template <int W>
__device__ __forceinline__ double window_median(const double *__restrict__ col, uint32_t window, uint64_t step) {
    if constexpr (W > 0) {
        uint64_t k[W];
#pragma unroll
        for (int j = 0; j < W; ++j) k[j] = (uint32_t)j < window ? dkey(col[(uint64_t)j * step]) : ~0ull;
#pragma unroll
        for (int p = 1; p < W; p *= 2)
#pragma unroll
            for (int q = p; q >= 1; q /= 2)
#pragma unroll
                for (int x = 0; x + q < W; ++x)
                    if (x >= q % p && (x - q % p) % (2 * q) < q && x / (2 * p) == (x + q) / (2 * p)) {
                        const bool sw = k[x] > k[x + q];
                        const uint64_t lo = sw ? k[x + q] : k[x], hi = sw ? k[x] : k[x + q];
                        k[x] = lo;
                        k[x + q] = hi;
                    }
        uint64_t a = 0, b = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            if ((uint32_t)j == (window - 1) / 2) a = k[j];
            if ((uint32_t)j == window / 2) b = k[j];
        }
        return (window & 1) ? dkey_inv(b) : __ddiv_rn(__dadd_rn(dkey_inv(a), dkey_inv(b)), 2.0);
    } else {
        double buf[kMaxWindow];
        for (uint32_t j = 0; j < window; ++j) {
            const double v = col[j * step];
            uint32_t k = j;
            while (k > 0 && buf[k - 1] > v) {
                buf[k] = buf[k - 1];
                --k;
            }
            buf[k] = v;
        }
        return (window & 1) ? buf[window / 2] : __ddiv_rn(__dadd_rn(buf[window / 2 - 1], buf[window / 2]), 2.0);
    }
}

// One thread per (window, sensor): median of the window's values, binned.  The
// row-major stream is read: neighbouring lanes are neighbouring sensors.
template <int W>
__global__ void __launch_bounds__(128) window_bin_kernel(const double *__restrict__ rows, uint32_t S, uint32_t window,
                                  uint32_t stride, uint64_t n_win, const double *__restrict__ edges,
                                  const uint32_t *__restrict__ n_edges, uint32_t edge_stride, uint32_t n_bins,
                                  const int32_t *__restrict__ anomaly, uint32_t *__restrict__ items,
                                  int32_t *__restrict__ labels) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n_win * S) return;
    const uint64_t w = i / S;
    const uint32_t s = (uint32_t)(i - w * S);
    const uint64_t start = w * stride;
    const double med = window_median<W>(rows + start * S + s, window, S);
    const double *e = edges + (uint64_t)s * edge_stride;
    const uint32_t m = n_edges[s];
    uint32_t cnt = 0;   // edges <= med (searchsorted side="right")
    for (uint32_t j = 0; j < m; ++j) cnt += e[j] <= med;
    int32_t b = (int32_t)cnt - 1;
    if (b < 0) b = 0;
    if (b > (int32_t)m - 2) b = (int32_t)m - 2;
    items[w * S + s] = s * n_bins + (uint32_t)b;
    if (s == 0) {
        int32_t mx = 0;
        if (anomaly) {
            mx = anomaly[start];
            for (uint32_t j = 1; j < window; ++j) mx = max(mx, anomaly[start + j]);
        }
        labels[w] = mx;
    }
}

// ---------------------------------------------------------------- online (P²) edges
//
// code/pipeline/online_discretize.py: every sensor keeps n_bins-1 five-marker
// estimators (P2Quantile :22-71) at quantiles i/n_bins; run_file (:111-128)
// feeds every row of every window, in window order, to every estimator (rows
// shared by overlapping windows are fed again) and after each window bins the
// window median with the edges of that moment (OnlineBinner.edges :87-103).
// An estimator is a sequential recurrence, so the parallel axis is the chain
// (sensor, estimator).  A warp carries `lanes` chains (1..32): few chains run
// one to a warp, so that every chain has a scheduler's double pipe to itself;
// many chains share a warp.  All arithmetic is explicitly rounded (no fused
// multiply-add), in the reference's order, so the estimates are the
// reference's bit for bit.
//
// When the estimate stops changing.  The reference's value() is the middle
// marker qv[2], and its marker rule can never move markers 2 and 3 for most
// quantiles.  With gap_i = n[i+1] - n[i], the setup gives gaps (1+2q, 2q,
// 2-2q, 1-2q); a sample in cell k adds 1 to every position and 1 more to
// positions 1..k, so gap_0 grows by [k >= 1] and gap_i (i = 1..3) shrinks by
// [k == i] -- gaps 1..3 never grow.  Marker i is tested only when d = gap_{i-1}
// >= 1 and span = gap_{i-1} + gap_i > 1, and a move needs qv[i] + qp < qv[i+1]
// with qp = (d+1) (qv[i+1] - qv[i-1]) / span >= (d+1)/span (qv[i+1] - qv[i]),
// so it needs (d+1)/span < 1, i.e. gap_i > 1.  Marker 3 needs gap_3 = 1-2q > 1:
// never.  Marker 2 needs gap_1 = 2q >= 1 and gap_2 = 2-2q > 1: never for
// q != 1/2.  With q = j/n_bins and n_bins <= 64 both inequalities miss by at
// least 1/64, far beyond the rounding of the positions and of qp.  So for q !=
// 1/2 the estimate is fixed at the setup (the third smallest of the first five
// samples).  For q = 1/2 the positions are integers and marker 2 can be tested
// only while no sample fell in cell 1 or 2 (gap_1 = gap_2 = 1), or never when
// qv[1] = qv[2] = qv[3] (qp = 0).  The kernel runs the recurrence until its
// chain reaches such a state and then writes the fixed estimate for every
// remaining window; `full` turns the shortcut off (the tests compare both).

constexpr uint32_t kMaxOnlineBins = 64;

// stable insertion sort of five registers (Python's sorted on equal keys)
__device__ __forceinline__ void sort5(double (&a)[5]) {
#pragma unroll
    for (int i = 1; i < 5; ++i)
#pragma unroll
        for (int j = i; j > 0; --j)
            if (a[j - 1] > a[j]) {
                const double t = a[j - 1];
                a[j - 1] = a[j];
                a[j] = t;
            }
}

__global__ void nan_count_kernel(const double *__restrict__ v, uint64_t n, uint32_t *__restrict__ nan_count) {
    uint32_t c = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c += v[i] != v[i];
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(nan_count, c);
}

// est[(w * S + s) * m + j] = estimate j of sensor s after window w; chain c =
// s * m + j reads rows[t * S + s] (row-major values: neighbouring lanes read
// neighbouring sensors).
__global__ void __launch_bounds__(128) p2_kernel(const double *__restrict__ rows, uint32_t S, uint32_t m,
                                                 const double *__restrict__ quant, uint32_t window, uint32_t stride,
                                                 uint64_t n_win, uint32_t lanes, uint32_t full,
                                                 double *__restrict__ est) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t c = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * lanes + lane;
    if (lane >= lanes || c >= (uint64_t)S * m) return;
    const uint32_t s = (uint32_t)(c / m), j = (uint32_t)(c - (uint64_t)s * m);
    const double q = quant[j];
    const bool half = q == 0.5;
    const uint64_t chains = (uint64_t)S * m;
    double qv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    double np_[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    uint32_t n_init = 0;   // the same for every chain: all see the same rows
    bool fixed = false;
    uint64_t w = 0;
    for (; w < n_win && !fixed; ++w) {
        const double *x_ptr = rows + w * stride * S + s;
        for (uint32_t t = 0; t < window; ++t) {
            const double x = x_ptr[(uint64_t)t * S];
            if (n_init < 5) {
#pragma unroll
                for (int i = 0; i < 5; ++i)
                    if ((uint32_t)i == n_init) qv[i] = x;
                if (++n_init == 5) {
                    sort5(qv);
                    np_[0] = 0.0;
                    np_[1] = __dadd_rn(1.0, __dmul_rn(2.0, q));
                    np_[2] = __dadd_rn(1.0, __dmul_rn(4.0, q));
                    np_[3] = __dadd_rn(3.0, __dmul_rn(2.0, q));
                    np_[4] = 4.0;
                    if (!full && (!half || (qv[1] == qv[2] && qv[2] == qv[3]))) {
                        fixed = true;
                        break;
                    }
                }
                continue;
            }
            int k;
            if (x < qv[0]) {
                qv[0] = x;
                k = 0;
            } else if (x < qv[1]) {
                k = 0;
            } else if (x < qv[2]) {
                k = 1;
            } else if (x < qv[3]) {
                k = 2;
            } else if (x <= qv[4]) {
                k = 3;
            } else {
                qv[4] = x;
                k = 3;
            }
#pragma unroll
            for (int i = 0; i < 5; ++i) np_[i] = __dadd_rn(np_[i], 1.0);
#pragma unroll
            for (int i = 1; i < 4; ++i)
                if (i <= k) np_[i] = __dadd_rn(np_[i], 1.0);
#pragma unroll
            for (int i = 1; i < 4; ++i) {
                const double d = __dsub_rn(np_[i], np_[i - 1]);
                const double span = __dsub_rn(np_[i + 1], np_[i - 1]);
                if (d >= 1.0 && span > 1.0) {
                    const double qp = __ddiv_rn(__dmul_rn(__dadd_rn(d, 1.0), __dsub_rn(qv[i + 1], qv[i - 1])), span);
                    const double moved = __dadd_rn(qv[i], qp);
                    if (qv[i - 1] < moved && moved < qv[i + 1]) qv[i] = moved;
                }
            }
            // q = 1/2: once a sample fell in cell 1 or 2, marker 2 is never tested again
            if (!full && (k == 1 || k == 2)) {
                fixed = true;
                break;
            }
        }
        double v;
        if (n_init >= 5) {
            v = qv[2];
        } else {
            // fewer than five samples: numpy's median of them (unused slots sort last)
            double a[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) a[i] = (uint32_t)i < n_init ? qv[i] : __longlong_as_double(0x7ff0000000000000ll);
            sort5(a);
            v = a[0];
#pragma unroll
            for (int i = 1; i < 5; ++i)
                if ((uint32_t)i == n_init / 2) v = (n_init & 1) ? a[i] : __ddiv_rn(__dadd_rn(a[i - 1], a[i]), 2.0);
        }
        est[w * chains + c] = v;
    }
    // the estimate no longer changes: every remaining window gets it
    for (; w < n_win; ++w) est[w * chains + c] = qv[2];
}

// One thread per (window, sensor): edges from the sensor's estimates after the
// window, then the window median binned with them.
template <int W>
__global__ void __launch_bounds__(128) online_bin_kernel(const double *__restrict__ rows, uint32_t S, uint32_t window, uint32_t stride,
                                  uint64_t n_win, const double *__restrict__ est, uint32_t n_bins,
                                  const int32_t *__restrict__ anomaly, double *__restrict__ edges,
                                  uint32_t *__restrict__ items, int32_t *__restrict__ labels) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n_win * S) return;
    const uint64_t w = i / S;
    const uint32_t s = (uint32_t)(i - w * S);
    const uint32_t m = n_bins - 1;
    double q[kMaxOnlineBins - 1];
    const double *src = est + i * m;
    for (uint32_t j = 0; j < m; ++j) {
        const double v = src[j];
        uint32_t k = j;
        while (k > 0 && q[k - 1] > v) {
            q[k] = q[k - 1];
            --k;
        }
        q[k] = v;
    }
    double span = __dsub_rn(q[m - 1], q[0]);
    if (1e-9 > span) span = 1e-9;   // max(q[-1] - q[0], 1e-9)
    const double min_gap = __dmul_rn(0.05, span);
    if (n_bins == 3) {
        if (__dsub_rn(q[1], q[0]) < min_gap) {
            const double mid = __ddiv_rn(__dadd_rn(q[0], q[1]), 2.0);
            const double half = __ddiv_rn(min_gap, 2.0);
            q[0] = __dsub_rn(mid, half);
            q[1] = __dadd_rn(mid, half);
        }
    } else {
        for (uint32_t j = 1; j < m; ++j) {
            const double lo = __dadd_rn(q[j - 1], min_gap);
            if (q[j] < lo) q[j] = lo;
        }
    }
    double *e = edges + i * (n_bins + 1);
    e[0] = __dsub_rn(q[0], span);
    for (uint32_t j = 0; j < m; ++j) e[1 + j] = q[j];
    e[n_bins] = __dadd_rn(q[m - 1], span);
    const uint64_t start = w * stride;
    const double med = window_median<W>(rows + start * S + s, window, S);
    uint32_t cnt = 0;   // edges <= med (searchsorted side="right")
    for (uint32_t j = 0; j <= n_bins; ++j) cnt += e[j] <= med;
    int32_t b = (int32_t)cnt - 1;
    if (b < 0) b = 0;
    if (b > (int32_t)n_bins - 1) b = (int32_t)n_bins - 1;
    items[i] = s * n_bins + (uint32_t)b;
    if (s == 0) {
        int32_t mx = 0;
        if (anomaly) {
            mx = anomaly[start];
            for (uint32_t j = 1; j < window; ++j) mx = max(mx, anomaly[start + j]);
        }
        labels[w] = mx;
    }
}

// Calls f with the median's network size for the window as a compile-time constant.
template <class F> void with_median_width(uint32_t window, F &&f) {
    if (window <= 16) f(std::integral_constant<int, 16>());
    else if (window <= 32) f(std::integral_constant<int, 32>());
    else if (window <= 64) f(std::integral_constant<int, 64>());
    else f(std::integral_constant<int, 0>());
}

// The calls' device buffers stay with the handle while they are small; a large
// stream's are given back when the call ends.
struct TxBuffers {
    TxWorkspace &w;
    size_t keep;
    explicit TxBuffers(sgfim_handle *h) : w(h->tx), keep(kept_between_calls(h->hbm_budget, 1ull << 30)) {}
    ~TxBuffers() {
        if (w.bytes() > keep) w.release();
    }
};

}  // namespace

}  // namespace sg

using namespace sg;

extern "C" int sgfim_transactionize_online(sgfim_handle *h, const double *values, uint64_t n_rows,
                                           uint32_t n_sensors, const int32_t *anomaly, uint32_t window,
                                           uint32_t stride, uint32_t n_bins, uint32_t flags, double *edges_out,
                                           uint32_t *items_out, int32_t *labels_out, uint64_t *n_windows_out) {
    if (!h) return SGFIM_EINVAL;
    if (!values && n_rows) return fail(h, SGFIM_EINVAL, "null values");
    if (n_sensors == 0 || window < 1 || stride < 1)
        return fail(h, SGFIM_EINVAL, "n_sensors, window and stride must be >= 1");
    if (n_bins < 2 || n_bins > kMaxOnlineBins) return fail(h, SGFIM_EINVAL, "n_bins must be in 2..64");
    if (window > kMaxWindow) return fail(h, SGFIM_EINVAL, "window longer than 256 rows");
    if ((uint64_t)n_sensors * n_bins > 0xffffffffull) return fail(h, SGFIM_EINVAL, "too many items");
    const uint64_t n_win = n_rows >= window ? (n_rows - window) / stride + 1 : 0;
    if (n_windows_out) *n_windows_out = n_win;
    if (n_win && (!items_out || !labels_out)) return fail(h, SGFIM_EINVAL, "null output");
    if ((n_win * n_sensors + 127) / 128 > 0x7fffffffull) return fail(h, SGFIM_EINVAL, "too many windows");
    API_GUARD_BEGIN
    SG_CUDA_TRY(cudaSetDevice(h->device));
    cudaStream_t st = h->stream;
    const uint32_t S = n_sensors, m = n_bins - 1;
    TxBuffers guard(h);
    DevBuf &d_rows = h->tx.rows, &d_est = h->tx.cols, &d_out = h->tx.small, &d_anom = h->tx.anom;
    if (n_win) {
        const size_t mat = (size_t)n_rows * S * 8;
        d_rows.reserve(mat, st);
        // out: nan count | quantiles | labels | items | edges
        size_t off = 0;
        auto carve = [&](size_t bytes) {
            const size_t o = off;
            off += (bytes + 255) & ~(size_t)255;
            return o;
        };
        const size_t o_nan = carve(4), o_q = carve((size_t)m * 8), o_lab = carve(n_win * 4),
                     o_items = carve(n_win * S * 4), o_edges = carve(n_win * S * (n_bins + 1) * 8);
        d_out.reserve(off, st);
        d_est.reserve(n_win * S * m * 8, st);
        char *base = d_out.as<char>();
        std::vector<double> quant(m);
        for (uint32_t j = 0; j < m; ++j) quant[j] = (double)(j + 1) / (double)n_bins;   // i / n_bins
        SG_CUDA_TRY(cudaMemcpyAsync(d_rows.ptr, values, mat, cudaMemcpyHostToDevice, st));
        SG_CUDA_TRY(cudaMemsetAsync(base + o_nan, 0, 4, st));
        SG_CUDA_TRY(cudaMemcpyAsync(base + o_q, quant.data(), (size_t)m * 8, cudaMemcpyHostToDevice, st));
        const uint64_t total = n_rows * S;
        nan_count_kernel<<<(unsigned)std::min<uint64_t>((total + 255) / 256, (uint64_t)h->n_sm * 8), 256, 0, st>>>(
            d_rows.as<double>(), total, reinterpret_cast<uint32_t *>(base + o_nan));
        SG_CUDA_TRY(cudaGetLastError());
        uint32_t nan_count = 0;
        SG_CUDA_TRY(cudaMemcpyAsync(&nan_count, base + o_nan, 4, cudaMemcpyDeviceToHost, st));
        SG_CUDA_TRY(cudaStreamSynchronize(st));
        if (nan_count) return fail(h, SGFIM_EINVAL, "the stream holds NaN values");
        // chains per warp: one while there are fewer chains than schedulers, then
        // as many as it takes to keep the warp count at about one per scheduler
        const uint64_t chains = (uint64_t)S * m;
        const uint64_t sched = (uint64_t)h->n_sm * 4;
        uint32_t lanes = (flags >> 8) & 63u;
        if (lanes == 0) lanes = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, (chains + sched - 1) / sched));
        if (lanes > 32) return fail(h, SGFIM_EINVAL, "more than 32 chains per warp");
        const uint64_t warps = (chains + lanes - 1) / lanes;
        p2_kernel<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(d_rows.as<double>(), S, m,
                                                              reinterpret_cast<const double *>(base + o_q), window,
                                                              stride, n_win, lanes, (flags & SGFIM_TX_P2_FULL) ? 1u : 0u,
                                                              d_est.as<double>());
        SG_CUDA_TRY(cudaGetLastError());
        if (anomaly) {
            d_anom.reserve(n_rows * 4, st);
            SG_CUDA_TRY(cudaMemcpyAsync(d_anom.ptr, anomaly, n_rows * 4, cudaMemcpyHostToDevice, st));
        }
        const uint64_t nt = n_win * S;
        with_median_width(window, [&](auto W) {
            online_bin_kernel<W()><<<(unsigned)((nt + 127) / 128), 128, 0, st>>>(
                d_rows.as<double>(), S, window, stride, n_win, d_est.as<double>(), n_bins,
                anomaly ? d_anom.as<int32_t>() : nullptr, reinterpret_cast<double *>(base + o_edges),
                reinterpret_cast<uint32_t *>(base + o_items), reinterpret_cast<int32_t *>(base + o_lab));
        });
        SG_CUDA_TRY(cudaGetLastError());
        h->launches += 3;
        SG_CUDA_TRY(cudaMemcpyAsync(items_out, base + o_items, nt * 4, cudaMemcpyDeviceToHost, st));
        SG_CUDA_TRY(cudaMemcpyAsync(labels_out, base + o_lab, n_win * 4, cudaMemcpyDeviceToHost, st));
        if (edges_out)
            SG_CUDA_TRY(cudaMemcpyAsync(edges_out, base + o_edges, nt * (n_bins + 1) * 8, cudaMemcpyDeviceToHost, st));
        SG_CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (flags & SGFIM_TX_LOAD) {
        std::vector<uint64_t> rp(n_win + 1);
        for (uint64_t w = 0; w <= n_win; ++w) rp[w] = w * S;
        return sgfim_load_csr(h, rp.data(), items_out, n_win);
    }
    return SGFIM_OK;
    API_GUARD_END(h)
}

extern "C" int sgfim_transactionize(sgfim_handle *h, const double *values, uint64_t n_rows, uint32_t n_sensors,
                                    const int32_t *anomaly, uint32_t window, uint32_t stride, uint32_t n_bins,
                                    uint32_t flags, double *edges_out, uint32_t *n_edges_out, uint32_t *items_out,
                                    int32_t *labels_out, uint64_t *n_windows_out) {
    if (!h) return SGFIM_EINVAL;
    if (!values && n_rows) return fail(h, SGFIM_EINVAL, "null values");
    if (n_sensors == 0 || n_bins < 1 || window < 1 || stride < 1)
        return fail(h, SGFIM_EINVAL, "n_sensors, n_bins, window and stride must be >= 1");
    if (window > kMaxWindow) return fail(h, SGFIM_EINVAL, "window longer than 256 rows");
    if (n_rows == 0) return fail(h, SGFIM_EINVAL, "empty stream");
    if ((uint64_t)n_sensors * n_bins > 0xffffffffull) return fail(h, SGFIM_EINVAL, "too many items");
    const uint64_t n_win = n_rows >= window ? (n_rows - window) / stride + 1 : 0;
    if (n_windows_out) *n_windows_out = n_win;
    if (!edges_out || !n_edges_out || (n_win && (!items_out || !labels_out)))
        return fail(h, SGFIM_EINVAL, "null output");
    API_GUARD_BEGIN
    SG_CUDA_TRY(cudaSetDevice(h->device));
    cudaStream_t st = h->stream;
    const uint32_t S = n_sensors, nq = n_bins + 1;
    // quantile positions exactly as numpy computes them
    std::vector<double> q(nq), gamma(nq);
    const double step = 1.0 / (double)n_bins;
    for (uint32_t i = 0; i < nq; ++i) q[i] = (double)i * step + 0.0;
    q[nq - 1] = 1.0;
    std::vector<uint64_t> need;   // order statistics
    std::vector<uint32_t> lo_pos(nq), hi_pos(nq);
    std::vector<uint64_t> lo_rank(nq), hi_rank(nq);
    const double nm1 = (double)(n_rows - 1);
    for (uint32_t i = 0; i < nq; ++i) {
        volatile double h_ = nm1 * q[i];   // one rounding, as numpy's (n - 1) * quantiles
        const double hv = h_;
        double prev = std::floor(hv);
        uint64_t lo, hi;
        if (hv >= nm1) {
            lo = hi = n_rows - 1;
            prev = -1.0;
        } else {
            lo = (uint64_t)prev;
            hi = lo + 1;
        }
        volatile double g_ = hv - prev;
        gamma[i] = g_;
        lo_rank[i] = lo;
        hi_rank[i] = hi;
        need.push_back(lo);
        need.push_back(hi);
    }
    std::sort(need.begin(), need.end());
    need.erase(std::unique(need.begin(), need.end()), need.end());
    for (uint32_t i = 0; i < nq; ++i) {
        lo_pos[i] = (uint32_t)(std::lower_bound(need.begin(), need.end(), lo_rank[i]) - need.begin());
        hi_pos[i] = (uint32_t)(std::lower_bound(need.begin(), need.end(), hi_rank[i]) - need.begin());
    }
    const uint32_t R = (uint32_t)need.size();
    // ranks selected at a time: their histograms stay within 64 MB
    const uint32_t batch =
        (uint32_t)std::min<uint64_t>(R, std::max<uint64_t>(1, (64ull << 20) / ((uint64_t)S * kDigits * 4)));

    TxBuffers guard(h);
    DevBuf &d_rows = h->tx.rows, &d_cols = h->tx.cols, &d_small = h->tx.small, &d_anom = h->tx.anom,
           &d_items = h->tx.items;
    const size_t mat = (size_t)n_rows * S * 8;
    d_rows.reserve(mat, st);
    d_cols.reserve(mat, st);
    // small buffers: nan count | ranks | stats | lo | hi | gamma | edges | n_edges | labels | select state | histograms
    size_t off = 0;
    auto carve = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    const size_t o_nan = carve(4), o_rank = carve((size_t)R * 8), o_stat = carve((size_t)S * R * 8),
                 o_lo = carve(nq * 4), o_hi = carve(nq * 4), o_g = carve(nq * 8), o_edge = carve((size_t)S * nq * 8),
                 o_ne = carve((size_t)S * 4), o_lab = carve(std::max<uint64_t>(n_win, 1) * 4),
                 o_sel = carve((size_t)S * batch * 32 + (size_t)S * 4), o_hist = carve((size_t)S * batch * kDigits * 4);
    d_small.reserve(off, st);
    char *base = d_small.as<char>();
    SG_CUDA_TRY(cudaMemcpyAsync(d_rows.ptr, values, mat, cudaMemcpyHostToDevice, st));
    SG_CUDA_TRY(cudaMemsetAsync(base + o_nan, 0, 4, st));
    SG_CUDA_TRY(cudaMemcpyAsync(base + o_rank, need.data(), (size_t)R * 8, cudaMemcpyHostToDevice, st));
    SG_CUDA_TRY(cudaMemcpyAsync(base + o_lo, lo_pos.data(), nq * 4, cudaMemcpyHostToDevice, st));
    SG_CUDA_TRY(cudaMemcpyAsync(base + o_hi, hi_pos.data(), nq * 4, cudaMemcpyHostToDevice, st));
    SG_CUDA_TRY(cudaMemcpyAsync(base + o_g, gamma.data(), nq * 8, cudaMemcpyHostToDevice, st));
    SG_CUDA_TRY(cudaMemsetAsync(base + o_hist, 0, (size_t)S * batch * kDigits * 4, st));
    const unsigned tiles = (unsigned)std::min<uint64_t>((n_rows + kTileRows - 1) / kTileRows, 1u << 20);
    to_columns_kernel<<<dim3(tiles, (S + kTileCols - 1) / kTileCols), 256, 0, st>>>(
        d_rows.as<double>(), n_rows, S, d_cols.as<double>(), reinterpret_cast<uint32_t *>(base + o_nan));
    SG_CUDA_TRY(cudaGetLastError());
    ++h->launches;
    SelectState sel;
    sel.prefix = reinterpret_cast<uint64_t *>(base + o_sel);
    sel.left = sel.prefix + (size_t)S * batch;
    sel.open = sel.left + (size_t)S * batch;
    sel.group = reinterpret_cast<uint32_t *>(sel.open + (size_t)S * batch);
    sel.n_open = sel.group + (size_t)S * batch;
    uint32_t *hist = reinterpret_cast<uint32_t *>(base + o_hist);
    // lists for a sixteenth of each column; short columns are read whole
    sel.cap = n_rows >= (1u << 16) ? (uint32_t)std::min<uint64_t>(n_rows / 16, 1u << 28) : 0u;
    h->tx.list.reserve((size_t)S * sel.cap * 8 + (size_t)S * 4, st);
    sel.list = h->tx.list.as<uint64_t>();
    sel.list_n = reinterpret_cast<uint32_t *>(sel.list + (size_t)S * sel.cap);
    // runs of at least 8,192 rows (a CTA clears and adds its histograms once), up to four CTAs per SM
    const unsigned runs = (unsigned)std::min<uint64_t>((n_rows + 8191) / 8192, (uint64_t)h->n_sm * 4 / S + 1);
    SG_CUDA_TRY(cudaFuncSetAttribute(select_hist_kernel<SELECT_LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize, kListBlock * 8));
    for (uint32_t rank0 = 0; rank0 < R; rank0 += batch) {
        const uint32_t rb = std::min(batch, R - rank0);
        select_init_kernel<<<(S * rb + 255) / 256, 256, 0, st>>>(
            sel, S, rb, reinterpret_cast<const uint64_t *>(base + o_rank) + rank0);
        SG_CUDA_TRY(cudaGetLastError());
        for (int pass = 0; pass < kPasses; ++pass) {
            const auto kernel = !sel.cap || pass < kListPass ? select_hist_kernel<SELECT_READ>
                                : pass == kListPass          ? select_hist_kernel<SELECT_LIST>
                                                             : select_hist_kernel<SELECT_FROM_LIST>;
            const size_t found_b = sel.cap && pass == kListPass ? kListBlock * 8 : 0;
            kernel<<<dim3(runs, S), kHistThreads, found_b, st>>>(d_cols.as<double>(), n_rows, sel, rb, pass, hist);
            SG_CUDA_TRY(cudaGetLastError());
            select_step_kernel<<<S, kStepThreads, 0, st>>>(sel, rb, pass, hist, reinterpret_cast<double *>(base + o_stat) + rank0,
                                                  R);
            SG_CUDA_TRY(cudaGetLastError());
        }
        h->launches += 1 + 2 * kPasses;
    }
    quantile_kernel<<<(S * nq + 127) / 128, 128, 0, st>>>(
        reinterpret_cast<const double *>(base + o_stat), R, reinterpret_cast<const uint32_t *>(base + o_lo),
        reinterpret_cast<const uint32_t *>(base + o_hi), reinterpret_cast<const double *>(base + o_g), nq, S,
        reinterpret_cast<double *>(base + o_edge));
    SG_CUDA_TRY(cudaGetLastError());
    ++h->launches;
    uint32_t nan_count = 0;
    std::vector<double> raw((size_t)S * nq);
    SG_CUDA_TRY(cudaMemcpyAsync(&nan_count, base + o_nan, 4, cudaMemcpyDeviceToHost, st));
    SG_CUDA_TRY(cudaMemcpyAsync(raw.data(), base + o_edge, raw.size() * 8, cudaMemcpyDeviceToHost, st));
    SG_CUDA_TRY(cudaStreamSynchronize(st));
    if (nan_count) return fail(h, SGFIM_EINVAL, "the stream holds NaN values");
    // np.unique of each sensor's quantiles (already ascending), constant column rule
    std::vector<double> edges((size_t)S * nq, 0.0);
    std::vector<uint32_t> n_edges(S);
    for (uint32_t s = 0; s < S; ++s) {
        std::vector<double> e(raw.begin() + (size_t)s * nq, raw.begin() + (size_t)(s + 1) * nq);
        std::stable_sort(e.begin(), e.end());
        std::vector<double> u;
        for (double x : e)
            if (u.empty() || !(x == u.back())) u.push_back(x);
        if (u.size() < 2) u = {u[0] - 0.5, u[0] + 0.5};
        n_edges[s] = (uint32_t)u.size();
        std::copy(u.begin(), u.end(), edges.begin() + (size_t)s * nq);
    }
    memcpy(edges_out, edges.data(), edges.size() * 8);
    memcpy(n_edges_out, n_edges.data(), (size_t)S * 4);
    if (n_win) {
        SG_CUDA_TRY(cudaMemcpyAsync(base + o_edge, edges.data(), edges.size() * 8, cudaMemcpyHostToDevice, st));
        SG_CUDA_TRY(cudaMemcpyAsync(base + o_ne, n_edges.data(), (size_t)S * 4, cudaMemcpyHostToDevice, st));
        if (anomaly) {
            d_anom.reserve(n_rows * 4, st);
            SG_CUDA_TRY(cudaMemcpyAsync(d_anom.ptr, anomaly, n_rows * 4, cudaMemcpyHostToDevice, st));
        }
        d_items.reserve(n_win * S * 4, st);
        const uint64_t nt = n_win * S;
        with_median_width(window, [&](auto W) {
            window_bin_kernel<W()><<<(unsigned)((nt + 127) / 128), 128, 0, st>>>(
                d_rows.as<double>(), S, window, stride, n_win, reinterpret_cast<const double *>(base + o_edge),
                reinterpret_cast<const uint32_t *>(base + o_ne), nq, n_bins, anomaly ? d_anom.as<int32_t>() : nullptr,
                d_items.as<uint32_t>(), reinterpret_cast<int32_t *>(base + o_lab));
        });
        SG_CUDA_TRY(cudaGetLastError());
        h->launches += 1;
        SG_CUDA_TRY(cudaMemcpyAsync(items_out, d_items.ptr, nt * 4, cudaMemcpyDeviceToHost, st));
        SG_CUDA_TRY(cudaMemcpyAsync(labels_out, base + o_lab, n_win * 4, cudaMemcpyDeviceToHost, st));
        SG_CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (flags & SGFIM_TX_LOAD) {
        std::vector<uint64_t> rp(n_win + 1);
        for (uint64_t w = 0; w <= n_win; ++w) rp[w] = w * S;
        return sgfim_load_csr(h, rp.data(), items_out, n_win);
    }
    return SGFIM_OK;
    API_GUARD_END(h)
}
