// kernels_bitmap.cu -- bitmap build and AND-popcount support counting.
//
// Reference counterparts (paths relative to the reference project root):
//   transpose_kernel   buildBitmap, code/engine_tensorfim/code/engine/src/kernel_bitmap.cu:342-380
//                      (host scatter there; one CTA per transaction tile here)
//   query_kernel       getResFrequencyCudaKernel, kernel_bitmap.cu:412-442 (one launch per
//                      DFS node there; thousands of queries per launch here)
//   k1_staged_kernel   the wave engine's maskBuild + BMMA counting, kernel_bmma.cu:603-768,
//                      restated for arbitrary k-item candidates with the bitmap chunk staged
//                      once per CTA in shared memory by TMA
#include <algorithm>
#include <cstdio>

#include "common.cuh"
#include "kernels.h"
#include "support_rule.h"

namespace sg {

// ---------------------------------------------------------------- transpose
// CSR transactions -> vertical bitmaps.  A CTA owns a tile of TW*64
// transactions and builds the d x TW-word tile in shared memory with 32-bit
// shared atomics, then writes each row's TW words (one 8*TW-byte run) and
// adds the tile's popcounts to the singleton counts.
__global__ void transpose_kernel(const uint64_t *__restrict__ row_ptr, const uint32_t *__restrict__ items,
                                 uint64_t n_txn, const int32_t *__restrict__ remap, uint32_t n_ids, uint32_t d,
                                 uint64_t *__restrict__ bm, uint64_t stride, uint32_t *__restrict__ counts,
                                 uint32_t tw) {
    extern __shared__ uint32_t tile[];  // d * 2*tw
    const uint32_t tw32 = 2 * tw;
    const uint64_t t0 = (uint64_t)blockIdx.x * tw * 64;
    const uint64_t t1 = min(n_txn, t0 + (uint64_t)tw * 64);
    for (uint32_t i = threadIdx.x; i < d * tw32; i += blockDim.x) tile[i] = 0;
    __syncthreads();
    for (uint64_t t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
        const uint32_t local = (uint32_t)(t - t0);
        for (uint64_t j = row_ptr[t]; j < row_ptr[t + 1]; ++j) {
            const uint32_t id = items[j];
            int32_t e = -1;
            if (remap) {
                if (id < n_ids) e = remap[id];
            } else if (id < d) {
                e = (int32_t)id;
            }
            if (e >= 0) atomicOr(&tile[(uint32_t)e * tw32 + (local >> 5)], 1u << (local & 31));
        }
    }
    __syncthreads();
    const uint64_t w0 = t0 / 64;
    for (uint32_t i = threadIdx.x; i < d * tw; i += blockDim.x) {
        const uint32_t e = i / tw, wl = i - e * tw;
        const uint64_t gw = w0 + wl;
        if (gw < stride) {
            const uint64_t v = (uint64_t)tile[e * tw32 + 2 * wl] | ((uint64_t)tile[e * tw32 + 2 * wl + 1] << 32);
            bm[(uint64_t)e * stride + gw] = v;
        }
    }
    if (counts) {
        for (uint32_t e = threadIdx.x; e < d; e += blockDim.x) {
            uint32_t s = 0;
            for (uint32_t k = 0; k < tw32; ++k) s += __popc(tile[e * tw32 + k]);
            if (s) atomicAdd(&counts[e], s);
        }
    }
}

// Fallback for very wide item spaces: global 64-bit atomics, one thread per transaction.
__global__ void transpose_global_kernel(const uint64_t *__restrict__ row_ptr, const uint32_t *__restrict__ items,
                                        uint64_t n_txn, const int32_t *__restrict__ remap, uint32_t n_ids,
                                        uint32_t d, unsigned long long *__restrict__ bm, uint64_t stride) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n_txn;
         t += (uint64_t)gridDim.x * blockDim.x) {
        for (uint64_t j = row_ptr[t]; j < row_ptr[t + 1]; ++j) {
            const uint32_t id = items[j];
            int32_t e = -1;
            if (remap) {
                if (id < n_ids) e = remap[id];
            } else if (id < d) {
                e = (int32_t)id;
            }
            if (e >= 0) atomicOr(&bm[(uint64_t)e * stride + (t >> 6)], 1ull << (t & 63));
        }
    }
}

__global__ void row_popc_kernel(const uint64_t *__restrict__ rows, uint64_t stride, uint64_t n_words, uint32_t d,
                                uint32_t *__restrict__ counts) {
    const uint32_t e = blockIdx.x;
    if (e >= d) return;
    uint32_t s = 0;
    for (uint64_t w = threadIdx.x; w < n_words; w += blockDim.x) s += popc64(rows[e * stride + w]);
    s = warp_sum(s);
    __shared__ uint32_t part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t v = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0;
        v = warp_sum(v);
        if (threadIdx.x == 0) counts[e] = v;
    }
}

void launch_transpose(const uint64_t *row_ptr, const uint32_t *items, uint64_t n_txn, const int32_t *remap,
                      uint32_t d, uint64_t *bitmaps, uint64_t stride, uint32_t *counts, cudaStream_t st,
                      int n_sm) {
    (void)n_sm;
    if (n_txn == 0 || d == 0) return;
    // n_ids of the remap table is passed through `counts` sizing by the caller; the
    // remap array covers every id that occurs (the caller builds it from the max id).
    const uint32_t n_ids = 0xffffffffu;
    const size_t budget = 160 * 1024;
    uint32_t tw = 32;
    while (tw > 1 && (size_t)d * tw * 8 > budget) tw >>= 1;
    SG_CUDA_TRY(cudaMemsetAsync(bitmaps, 0, (size_t)d * stride * 8, st));
    if ((size_t)d * tw * 8 > budget) {
        transpose_global_kernel<<<1024, 256, 0, st>>>(row_ptr, items, n_txn, remap, n_ids, d,
                                                      reinterpret_cast<unsigned long long *>(bitmaps), stride);
        SG_CUDA_TRY(cudaGetLastError());
        if (counts) launch_row_popc(bitmaps, stride, stride, d, counts, st);
        return;
    }
    const size_t smem = (size_t)d * tw * 8;
    SG_CUDA_TRY(cudaFuncSetAttribute(transpose_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (counts) SG_CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)d * 4, st));
    const uint64_t tiles = (n_txn + (uint64_t)tw * 64 - 1) / ((uint64_t)tw * 64);
    transpose_kernel<<<(unsigned)tiles, 512, smem, st>>>(row_ptr, items, n_txn, remap, n_ids, d, bitmaps, stride,
                                                          counts, tw);
    SG_CUDA_TRY(cudaGetLastError());
}

namespace {
// Candidate CSR from the host, checked and mapped on the device: bad[0] |= 1 when
// cand_ptr decreases anywhere; items become dense rows (ids that never occur map
// past the last row, where every support is 0).  remap null = identity on [0, n_ids).
__global__ void cand_prep_kernel(const uint64_t *__restrict__ cand_ptr, uint64_t n_cand, uint32_t *__restrict__ items,
                                 uint64_t n_items, const int32_t *__restrict__ remap, uint32_t n_ids,
                                 uint32_t *__restrict__ bad) {
    const uint64_t n = n_cand > n_items ? n_cand : n_items;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (i < n_cand && cand_ptr[i + 1] < cand_ptr[i]) atomicOr(bad, 1u);
        if (i < n_items) {
            const uint32_t id = items[i];
            uint32_t r = 0xfffffffeu;
            if (id < n_ids) {
                const int32_t m = remap ? remap[id] : (int32_t)id;
                if (m >= 0) r = (uint32_t)m;
            }
            items[i] = r;
        }
    }
}
}  // namespace

void launch_cand_prep(const uint64_t *cand_ptr, uint64_t n_cand, uint32_t *items, uint64_t n_items,
                      const int32_t *remap, uint32_t n_ids, uint32_t *bad, cudaStream_t st, int n_sm) {
    const uint64_t n = std::max<uint64_t>(std::max(n_cand, n_items), 1);
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)n_sm * 8);
    cand_prep_kernel<<<blocks, 256, 0, st>>>(cand_ptr, n_cand, items, n_items, remap, n_ids, bad);
    SG_CUDA_TRY(cudaGetLastError());
}

void launch_row_popc(const uint64_t *rows, uint64_t stride, uint64_t n_words, uint32_t d, uint32_t *counts,
                     cudaStream_t st) {
    if (d == 0) return;
    row_popc_kernel<<<d, 256, 0, st>>>(rows, stride, n_words, d, counts);
    SG_CUDA_TRY(cudaGetLastError());
}

// ---------------------------------------------------------------- streaming queries
// A warp owns one segment of one query's words: a step covers 256 words, two rows
// at a time (eight 16-byte loads in flight per lane), rows are read only where the
// AND of the mask and the rows before them still has a bit, and the row numbers
// travel in the lanes.  Few queries are cut into segments that fill the chip, whose
// counts add up in `out`.  A count below qb.thr may be reported as anything below
// it: a segment stops once its words miss more of the mask's mask_sup transactions
// than mask_sup - thr (the search tree's FHUT queries mostly do, and soon).  These
// queries wait for loads, not bandwidth: one 16-byte load per lane in flight, a
// warp per query took 113 ms of a 2,000,000-transaction search, now 24 ms.
constexpr uint32_t kQueryU = 4;
constexpr uint32_t kQueryStep = 64 * kQueryU;   // words a warp covers per step

constexpr uint32_t kQueryWarps = 96;            // per SM, four times what is resident: short tails

static uint32_t query_segments(uint64_t n_units, uint64_t n_words, int n_sm) {
    const uint64_t most = std::max<uint64_t>(1, (n_words + kQueryStep - 1) / kQueryStep);
    return (uint32_t)std::min<uint64_t>(most, std::max<uint64_t>(1, (uint64_t)n_sm * kQueryWarps / std::max<uint64_t>(n_units, 1)));
}

__global__ void __launch_bounds__(256, 3) query_kernel(QueryBatch qb, uint32_t n_seg, uint64_t seg_words) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t total = qb.n_q * n_seg;
    for (uint64_t unit = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; unit < total; unit += n_warps) {
        const uint64_t q = n_seg == 1 ? unit : unit / n_seg, seg = unit - q * n_seg;
        const uint64_t a = qb.q_ptr[q], k = qb.q_ptr[q + 1] - a;
        const uint64_t *mask = nullptr;
        bool lead = false;   // the first row belongs to the mask
        if (qb.mask_slot) {
            const uint32_t s = qb.mask_slot[q];
            if (s != kNoSlot) mask = qb.arena + (uint64_t)(s & ~kLeadRow) * qb.arena_stride;
            lead = s != kNoSlot && (s & kLeadRow);
        }
        uint32_t acc = 0;
        if (k == 0 && mask == nullptr) {
            acc = seg == 0 ? (uint32_t)qb.empty_value : 0u;
        } else {
            // the first 32 rows travel in the lanes
            const uint32_t mine = lane < k ? qb.q_items[a + lane] : 0u;
            bool bad = mine >= qb.d && lane < k;
            for (uint64_t i = 32 + lane; i < k; i += 32) bad |= qb.q_items[a + i] >= qb.d;
            if (!__any_sync(kAll, bad)) {
                const uint64_t w_first = qb.q_w0 ? (qb.q_w0[q] & ~1ull) : 0;
                const uint64_t w0 = max(w_first, seg * seg_words), w1 = min(qb.n_words, (seg + 1) * seg_words);
                const bool bounded = mask && qb.mask_sup;
                const uint32_t sup = bounded ? qb.mask_sup[q] : 0;
                const uint32_t slack = bounded && sup > qb.thr ? sup - qb.thr : 0;
                uint32_t part = 0, missed = 0;   // per lane
                for (uint64_t base = w0; base < w1; base += kQueryStep) {
                    const uint64_t at = base + 2 * lane;
                    uint4 v[kQueryU];
#pragma unroll
                    for (uint32_t u = 0; u < kQueryU; ++u) {
                        v[u] = make_uint4(0, 0, 0, 0);
                        if (at + 64 * u < w1) v[u] = mask ? ld_nc_v4(mask + at + 64 * u) : make_uint4(~0u, ~0u, ~0u, ~0u);
                    }
                    if (lead) {
                        const uint64_t *row = qb.rows + (uint64_t)__shfl_sync(kAll, mine, 0) * qb.row_stride + at;
#pragma unroll
                        for (uint32_t u = 0; u < kQueryU; ++u)
                            if (at + 64 * u < w1) v[u] = and4(v[u], ld_nc_v4(row + 64 * u));
                    }
                    if (bounded)
#pragma unroll
                        for (uint32_t u = 0; u < kQueryU; ++u) missed += popc4(v[u]);
                    bool left = true;   // some lane's AND still has a bit
                    for (uint64_t i = lead; i < k; i += 2) {
                        const uint64_t i2 = i + 1 < k ? i + 1 : i;   // an odd count ANDs its last row twice
                        const uint32_t x = i < 32 ? __shfl_sync(kAll, mine, (int)i) : qb.q_items[a + i];
                        const uint32_t y = i2 < 32 ? __shfl_sync(kAll, mine, (int)i2) : qb.q_items[a + i2];
                        const uint64_t *rx = qb.rows + (uint64_t)x * qb.row_stride + at;
                        const uint64_t *ry = qb.rows + (uint64_t)y * qb.row_stride + at;
                        uint4 r[kQueryU], o[kQueryU];
                        bool any = false;
#pragma unroll
                        for (uint32_t u = 0; u < kQueryU; ++u) {
                            const bool live = (v[u].x | v[u].y | v[u].z | v[u].w) != 0;
                            r[u] = o[u] = make_uint4(0, 0, 0, 0);
                            if (live) {
                                r[u] = ld_nc_v4(rx + 64 * u);
                                o[u] = ld_nc_v4(ry + 64 * u);
                            }
                            any |= live;
                        }
#pragma unroll
                        for (uint32_t u = 0; u < kQueryU; ++u) v[u] = and4(v[u], and4(r[u], o[u]));
                        left = __any_sync(kAll, any);
                        if (!left) break;
                    }
                    uint32_t got = 0;
                    if (left)
#pragma unroll
                        for (uint32_t u = 0; u < kQueryU; ++u) got += popc4(v[u]);
                    part += got;
                    if (bounded) {
                        missed -= got;
                        if (__reduce_add_sync(kAll, missed) > slack) break;
                    }
                    if (qb.mode == QUERY_ANY && __any_sync(kAll, part != 0)) break;
                    if (qb.mode == QUERY_ANY2 && __reduce_add_sync(kAll, part) >= 2) break;
                }
                acc = warp_sum(part);
            }
        }
        if (lane == 0) {
            if (n_seg == 1) qb.out[q] = acc;
            else if (acc) atomicAdd(&qb.out[q], acc);
        }
    }
}

// Tail counts of a wave's nodes: entry j of the concatenated tails belongs to
// node i (tail_ptr[i] <= j < tail_ptr[i+1]); out[j] = popc(mask(slot[i]) AND
// row(piv[i]) AND row(items[j])); piv[i] may be kNoSlot (the mask is the node's own;
// else it is its parent's).  A warp takes four entries at a time (the node found 32 places at
// a time), so a node's mask is read once for up to four of its items, ten 16-byte
// loads in flight per lane.  The population counts bound it (16 lanes a clock per
// SM): eight words pass through carry-save adders (R. W. Harley's method; H. S.
// Warren, Hacker's Delight, 2nd ed., section 5-1) into one count of eights.  Few
// entries are cut into segments like the queries.  (A warp per entry, a count per
// word: 28 ms of a 2,000,000-transaction search with
// a mask per child, whose making took 22 ms more; now 28 and 5.)
__device__ __forceinline__ void csa(uint32_t &high, uint32_t &low, uint32_t x, uint32_t y) {
    const uint32_t u = low ^ x;
    high = (low & x) | (u & y);
    low = u ^ y;
}
constexpr uint32_t kTailI = 4, kTailU = 2;   // entries, 16-byte pieces of each in flight

__global__ void __launch_bounds__(256, 3) tail_count_kernel(const uint64_t *__restrict__ rows, uint64_t row_stride,
                                                        uint64_t n_words, const uint64_t *__restrict__ arena,
                                                        uint64_t arena_stride, const uint32_t *__restrict__ slot,
                                                        const uint32_t *__restrict__ piv,
                                                        const uint64_t *__restrict__ tail_ptr, uint32_t n_nodes,
                                                        const uint32_t *__restrict__ items, uint32_t *__restrict__ out,
                                                        uint32_t n_seg, uint64_t seg_words, uint32_t search_step) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t n_entries = tail_ptr[n_nodes];
    const uint64_t total = (n_entries + kTailI - 1) / kTailI * n_seg;
    for (uint64_t unit = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; unit < total; unit += n_warps) {
        const uint64_t g = n_seg == 1 ? unit : unit / n_seg, seg = unit - g * n_seg;
        uint64_t j = g * kTailI;
        const uint64_t j_end = min(n_entries, j + kTailI);
        const uint64_t w0 = seg * seg_words, w1 = min(n_words, w0 + seg_words);
        // the node of entry j: 32 places at a time
        uint32_t lo = 0;
        for (uint32_t step = search_step;; step >>= 5) {
            const uint64_t at = (uint64_t)lo + (uint64_t)lane * step;
            const unsigned le = __ballot_sync(kAll, at < n_nodes && tail_ptr[at] <= j);
            lo += (31 - __clz(le)) * step;   // lane 0's place always holds
            if (step == 1) break;
        }
        while (j < j_end) {   // runs of one node's entries
            while (tail_ptr[lo + 1] <= j) ++lo;
            const uint32_t n = (uint32_t)(min(j_end, tail_ptr[lo + 1]) - j);
            const uint64_t *mask = arena + (uint64_t)slot[lo] * arena_stride;
            const uint64_t *lead = piv[lo] != kNoSlot ? rows + (uint64_t)piv[lo] * row_stride : mask;
            const uint64_t *r[kTailI];
#pragma unroll
            for (uint32_t i = 0; i < kTailI; ++i) r[i] = rows + (uint64_t)items[j + min(i, n - 1)] * row_stride;
            uint32_t ones[kTailI] = {0, 0, 0, 0}, twos[kTailI] = {0, 0, 0, 0}, fours[kTailI] = {0, 0, 0, 0};
            uint32_t eights[kTailI] = {0, 0, 0, 0};
            for (uint64_t base = w0; base < w1; base += 64 * kTailU) {
                uint4 m[kTailU], v[kTailI][kTailU];
#pragma unroll
                for (uint32_t u = 0; u < kTailU; ++u) {
                    const uint64_t w = base + 64 * u + 2 * lane;
                    const bool in = w < w1;
                    m[u] = in ? and4(ld_nc_v4(mask + w), ld_nc_v4(lead + w)) : make_uint4(0, 0, 0, 0);
#pragma unroll
                    for (uint32_t i = 0; i < kTailI; ++i)
                        v[i][u] = in && i < n ? ld_nc_v4(r[i] + w) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (uint32_t i = 0; i < kTailI; ++i) {
                    if (i >= n) break;
                    const uint4 x = and4(m[0], v[i][0]), y = and4(m[1], v[i][1]);
                    uint32_t t0, t1, f0, f1, e;
                    csa(t0, ones[i], x.x, x.y);
                    csa(t1, ones[i], x.z, x.w);
                    csa(f0, twos[i], t0, t1);
                    csa(t0, ones[i], y.x, y.y);
                    csa(t1, ones[i], y.z, y.w);
                    csa(f1, twos[i], t0, t1);
                    csa(e, fours[i], f0, f1);
                    eights[i] += __popc(e);
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < kTailI; ++i) {
                const uint32_t c = warp_sum(8 * eights[i] + 4 * __popc(fours[i]) + 2 * __popc(twos[i]) + __popc(ones[i]));
                if (lane == 0 && i < n) {
                    if (n_seg == 1) out[j + i] = c;
                    else if (c) atomicAdd(&out[j + i], c);
                }
            }
            j += n;
        }
    }
}

void launch_tail_counts(const uint64_t *rows, uint64_t row_stride, uint64_t n_words, const uint64_t *arena,
                        uint64_t arena_stride, const uint32_t *slot, const uint32_t *piv, const uint64_t *tail_ptr,
                        uint32_t n_nodes, uint64_t n_entries, const uint32_t *items, uint32_t *out, cudaStream_t st, int n_sm) {
    if (n_nodes == 0 || n_entries == 0) return;
    const uint64_t groups = (n_entries + kTailI - 1) / kTailI;
    const uint32_t n_seg = query_segments(groups, n_words, n_sm);
    const uint64_t seg_words = ((n_words + n_seg - 1) / n_seg + kQueryStep - 1) / kQueryStep * kQueryStep;
    if (n_seg > 1) SG_CUDA_TRY(cudaMemsetAsync(out, 0, n_entries * 4, st));
    uint32_t search_step = 1;   // 32 steps of it cover the nodes
    while ((uint64_t)search_step * 32 < n_nodes) search_step *= 32;
    const uint64_t blocks = std::min<uint64_t>((groups * n_seg + 7) / 8, (uint64_t)n_sm * 64);
    tail_count_kernel<<<(unsigned)blocks, 256, 0, st>>>(rows, row_stride, n_words, arena, arena_stride, slot, piv,
                                                        tail_ptr, n_nodes, items, out, n_seg, seg_words, search_step);
    SG_CUDA_TRY(cudaGetLastError());
}

void launch_queries(const QueryBatch &qb, cudaStream_t st, int n_sm) {
    if (qb.n_q == 0) return;
    const uint32_t n_seg = query_segments(qb.n_q, qb.n_words, n_sm);
    const uint64_t seg_words =
        std::max<uint64_t>(1, ((qb.n_words + n_seg - 1) / n_seg + kQueryStep - 1) / kQueryStep) * kQueryStep;
    if (n_seg > 1) SG_CUDA_TRY(cudaMemsetAsync(qb.out, 0, qb.n_q * 4, st));
    const uint64_t blocks = std::min<uint64_t>((qb.n_q * n_seg + 7) / 8, (uint64_t)n_sm * 64);
    query_kernel<<<(unsigned)blocks, 256, 0, st>>>(qb, n_seg, seg_words);
    SG_CUDA_TRY(cudaGetLastError());
}

// ---------------------------------------------------------------- streamed batch supports
// Supports of CSR candidates straight from L2/HBM: a warp owns one segment of
// one candidate's rows.  A step covers kStreamU x 64 words, two rows at a time
// (eight 16-byte loads in flight per lane), and rows are read only where the
// AND of the rows before them still has a bit.  With more than one segment the
// warps add into out, which holds zeros (an empty candidate's support comes
// from its first segment).  Short segments fill the chip
// when candidates are few and keep its last wave short: over 1,000,000
// transactions 300 candidates take 23 us and 3,000 130 us (one warp per candidate:
// 384 and 420 us), 200,000 run at 22 TB/s from L1 and L2.
constexpr int kStreamU = 4;
constexpr uint32_t kStreamStep = 64 * kStreamU;   // words a warp covers per step

struct StreamBatch {
    const uint64_t *rows;
    uint64_t stride, n_words;
    uint32_t d;
    const uint64_t *cand_ptr;
    const uint32_t *items;
    uint64_t n;                       // candidates (entries of index, when given)
    const uint64_t *n_device;         // when set, the count is read on the device
    const uint32_t *index;            // optional: entry j is candidate index[j]
    uint64_t n_txn;
    uint64_t seg_words;               // multiple of 2
    uint32_t n_seg;
    uint32_t *out;
};

__global__ void __launch_bounds__(256) cand_stream_kernel(StreamBatch sb) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t total = (sb.n_device ? *sb.n_device : sb.n) * sb.n_seg;
    for (uint64_t q = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; q < total; q += n_warps) {
        const uint64_t j = q / sb.n_seg;
        const uint64_t c = sb.index ? sb.index[j] : j, seg = q - j * sb.n_seg;
        const uint64_t a = sb.cand_ptr[c], k = sb.cand_ptr[c + 1] - a;
        uint32_t acc = 0;
        if (k == 0) {
            acc = seg == 0 ? (uint32_t)sb.n_txn : 0u;
        } else {
            // the first 32 items travel in the lanes
            const uint32_t mine = lane < k ? sb.items[a + lane] : 0u;
            bool bad = mine >= sb.d;
            for (uint64_t i = 32 + lane; i < k; i += 32) bad |= sb.items[a + i] >= sb.d;
            if (!__any_sync(0xffffffffu, bad)) {
                const uint64_t w0 = seg * sb.seg_words, w1 = min(sb.n_words, w0 + sb.seg_words);
                uint32_t part = 0;
                for (uint64_t base = w0; base < w1; base += kStreamStep) {
                    const uint64_t *at = sb.rows + base + 2 * lane;
                    uint4 v[kStreamU];
                    const uint64_t *r0 = at + (uint64_t)__shfl_sync(0xffffffffu, mine, 0) * sb.stride;
#pragma unroll
                    for (int u = 0; u < kStreamU; ++u)
                        v[u] = base + 64 * u + 2 * lane < w1 ? ld_nc_v4(r0 + 64 * u) : make_uint4(0, 0, 0, 0);
                    for (uint64_t i = 1; i < k; i += 2) {
                        const uint64_t i2 = i + 1 < k ? i + 1 : i;   // an odd count ANDs its last row twice
                        const uint32_t x = i < 32 ? __shfl_sync(0xffffffffu, mine, (int)i) : sb.items[a + i];
                        const uint32_t y = i2 < 32 ? __shfl_sync(0xffffffffu, mine, (int)i2) : sb.items[a + i2];
                        const uint64_t *rx = at + (uint64_t)x * sb.stride, *ry = at + (uint64_t)y * sb.stride;
                        uint4 p[kStreamU], o[kStreamU];
                        bool any = false;
#pragma unroll
                        for (int u = 0; u < kStreamU; ++u) {
                            const bool live = (v[u].x | v[u].y | v[u].z | v[u].w) != 0;
                            p[u] = o[u] = make_uint4(0, 0, 0, 0);
                            if (live) {
                                p[u] = ld_nc_v4(rx + 64 * u);
                                o[u] = ld_nc_v4(ry + 64 * u);
                            }
                            any |= live;
                        }
#pragma unroll
                        for (int u = 0; u < kStreamU; ++u) v[u] = and4(v[u], and4(p[u], o[u]));
                        if (!__any_sync(0xffffffffu, any)) break;
                    }
#pragma unroll
                    for (int u = 0; u < kStreamU; ++u) part += popc4(v[u]);
                }
                acc = warp_sum(part);
            }
        }
        if (lane == 0) {
            if (sb.n_seg == 1) sb.out[c] = acc;
            else if (acc) atomicAdd(&sb.out[c], acc);
        }
    }
}

// All n candidates (index null), or the listed ones, whose outputs hold zeros.
static void launch_cand_stream(StreamBatch sb, cudaStream_t st, int n_sm) {
    const uint64_t warps = (uint64_t)n_sm * 128;   // four times what the chip holds at once: short tails
    const uint64_t most = std::max<uint64_t>(1, (sb.n_words + kStreamStep - 1) / kStreamStep);
    if (sb.n_device) {
        sb.n_seg = (uint32_t)std::min<uint64_t>(8, most);
    } else {
        if (sb.n == 0) return;
        sb.n_seg = (uint32_t)std::min<uint64_t>(most, std::max<uint64_t>(1, warps / sb.n));
        if (sb.n_seg > 1) SG_CUDA_TRY(cudaMemsetAsync(sb.out, 0, sb.n * 4, st));
    }
    sb.seg_words = ((sb.n_words + sb.n_seg - 1) / sb.n_seg + kStreamStep - 1) / kStreamStep * kStreamStep;
    const uint64_t blocks =
        sb.n_device ? (uint64_t)n_sm * 8 : std::min<uint64_t>((sb.n * sb.n_seg + 7) / 8, (uint64_t)n_sm * 64);
    cand_stream_kernel<<<(unsigned)blocks, 256, 0, st>>>(sb);
    SG_CUDA_TRY(cudaGetLastError());
}

// ---------------------------------------------------------------- staged batch supports
// Candidate records: 8 x uint16 row ids; 0xffff marks unused slots and an
// all-0xffff record marks a candidate whose support was written elsewhere.
constexpr uint16_t kRecNone = 0xffffu;
constexpr uint32_t kStagedRowsPerBox = 256;
constexpr uint32_t kStagedWords = 16;   // words per row per chunk (128 bytes)

__global__ void prep_records_kernel(const uint64_t *__restrict__ cand_ptr, const uint32_t *__restrict__ cand_items,
                                    uint64_t n, uint32_t d, uint64_t n_txn, uint4 *__restrict__ recs,
                                    uint32_t *__restrict__ ovf_list, unsigned long long *__restrict__ ovf_count,
                                    uint32_t *__restrict__ out) {
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = cand_ptr[c], b = cand_ptr[c + 1];
        const uint64_t k = b - a;
        uint32_t h[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
        if (k == 0) {
            out[c] = (uint32_t)n_txn;
        } else if (k > 8) {
            const unsigned long long slot = atomicAdd(ovf_count, 1ull);
            ovf_list[slot] = (uint32_t)c;
            out[c] = 0;
        } else {
            bool zero = false;
            uint16_t it[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) it[i] = kRecNone;
            for (uint64_t i = 0; i < k; ++i) {
                const uint32_t x = cand_items[a + i];
                if (x >= d) zero = true;
                it[i] = (uint16_t)x;
            }
            if (zero) {
                out[c] = 0;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) h[i] = (uint32_t)it[2 * i] | ((uint32_t)it[2 * i + 1] << 16);
            }
        }
        recs[c] = make_uint4(h[0], h[1], h[2], h[3]);
    }
}

// 8-lane transpose-reduce: lane l (of an aligned group of 8) enters with
// partials p[0..7] for 8 candidates and leaves with the group-wide sum of p[l].
__device__ __forceinline__ uint32_t treduce8(const uint32_t (&p)[8], uint32_t l) {
    uint32_t q[4], r[2];
    const bool h4 = l & 4, h2 = l & 2, h1 = l & 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t send = h4 ? p[k] : p[k + 4];
        const uint32_t keep = h4 ? p[k + 4] : p[k];
        q[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t send = h2 ? q[k] : q[k + 2];
        const uint32_t keep = h2 ? q[k + 2] : q[k];
        r[k] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const uint32_t send = h1 ? r[0] : r[1];
    const uint32_t keep = h1 ? r[1] : r[0];
    return keep + __shfl_xor_sync(0xffffffffu, send, 1);
}

// Each CTA owns `cpc` consecutive candidates and sweeps the whole transaction
// range in chunks of 16 words (1024 transactions).  Per chunk, TMA copies the
// 128-byte slice of every bitmap row into shared memory (rows r*128 bytes
// apart); a group of 8 lanes then evaluates one candidate at a time, each
// lane ANDing a 16-byte piece of the k rows, so a warp reads 4 rows x 128
// contiguous bytes per step (4 conflict-free wavefronts).  Partial popcounts
// of 8 candidates are transpose-reduced into one register per lane, which
// accumulates across chunks: each support is written once, at the end.
template <int THREADS, int SMAX>
__global__ void __launch_bounds__(THREADS, 1)
    k1_staged_kernel(const __grid_constant__ CUtensorMap bm_map, uint32_t n_boxes, uint64_t n_words,
                     const uint4 *__restrict__ recs, uint64_t n_cand, uint32_t cpc, uint32_t *__restrict__ out,
                     uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr uint32_t G = THREADS / 8;             // groups of 8 lanes
    uint8_t *chunk = smem;                           // n_boxes * 256 rows * 128 B
    const uint32_t chunk_bytes = n_boxes * kStagedRowsPerBox * kStagedWords * 8;
    uint4 *rec_s = reinterpret_cast<uint4 *>(smem + chunk_bytes);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + chunk_bytes + (size_t)cpc * 16);

    const uint32_t tid = threadIdx.x;
    const uint32_t g = tid >> 3, l = tid & 7;
    const uint64_t base = (uint64_t)blockIdx.x * cpc;
    if (base >= n_cand) return;
    const uint64_t left = n_cand - base;
    const uint32_t ncta = left < cpc ? (uint32_t)left : cpc;

    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    for (uint32_t i = tid; i < ncta; i += THREADS) rec_s[i] = recs[base + i];
    __syncthreads();

    uint32_t acc[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) acc[s] = 0;
    const uint32_t n_sets = (ncta + 8 * G - 1) / (8 * G);
    const uint64_t n_chunks = (n_words + kStagedWords - 1) / kStagedWords;
    uint32_t phase = 0;
    for (uint64_t ch = 0; ch < n_chunks; ++ch) {
        if (tid == 0) {
            mbar_arrive_expect_tx(bar, chunk_bytes);
            for (uint32_t b = 0; b < n_boxes; ++b)
                tma_load_2d(chunk + (size_t)b * kStagedRowsPerBox * kStagedWords * 8, &bm_map,
                            (int32_t)(ch * kStagedWords), (int32_t)(b * kStagedRowsPerBox), bar);
        }
        const bool ok = mbar_wait_bounded(bar, phase, err);
        phase ^= 1;
        if (__syncthreads_or(!ok)) {
            // give in-flight copies one more bounded chance to land before leaving
            mbar_wait_bounded(bar, phase ^ 1, err);
            return;
        }
#pragma unroll
        for (int s = 0; s < SMAX; ++s) {
            if ((uint32_t)s < n_sets) {
                uint32_t p[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t c = ((uint32_t)s * 8 + j) * G + g;
                    uint32_t v = 0;
                    if (c < ncta) {
                        const uint4 r = rec_s[c];
                        const uint32_t h[4] = {r.x, r.y, r.z, r.w};
                        uint32_t it0 = h[0] & 0xffffu;
                        if (it0 != kRecNone) {
                            uint4 m = *reinterpret_cast<const uint4 *>(chunk + (size_t)it0 * 128 + l * 16);
#pragma unroll
                            for (int k = 1; k < 8; ++k) {
                                const uint32_t it = (h[k >> 1] >> ((k & 1) * 16)) & 0xffffu;
                                if (it == kRecNone) break;
                                m = and4(m, *reinterpret_cast<const uint4 *>(chunk + (size_t)it * 128 + l * 16));
                            }
                            v = popc4(m);
                        }
                    }
                    p[j] = v;
                }
                acc[s] += treduce8(p, l);
            }
        }
        __syncthreads();  // every group is done with this chunk before TMA overwrites it
    }
#pragma unroll
    for (int s = 0; s < SMAX; ++s) {
        const uint32_t c = ((uint32_t)s * 8 + l) * G + g;
        if ((uint32_t)s < n_sets && c < ncta) {
            const uint32_t it0 = rec_s[c].x & 0xffffu;
            if (it0 != kRecNone) out[base + c] = acc[s];
        }
    }
}

// 4-lane transpose-reduce: lane l (of an aligned group of 4) enters with
// partials p[0..3] for 4 candidates and leaves with the group-wide sum of p[l].
__device__ __forceinline__ uint32_t treduce4(const uint32_t (&p)[4], uint32_t l) {
    uint32_t q[2];
    const bool h2 = l & 2, h1 = l & 1;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t send = h2 ? p[k] : p[k + 2];
        const uint32_t keep = h2 ? p[k + 2] : p[k];
        q[k] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const uint32_t send = h1 ? q[0] : q[1];
    const uint32_t keep = h1 ? q[1] : q[0];
    return keep + __shfl_xor_sync(0xffffffffu, send, 1);
}

// k1_staged_kernel with groups of 4 lanes: each lane ANDs 32 bytes of a row
// (two 16-byte pieces, 64 bytes apart), so a candidate's record is decoded by
// 4 lanes instead of 8 and a warp evaluates 8 candidates per step.  Even
// groups read the row's first half first and odd groups its second half
// first: the two groups of an 8-lane phase of a 128-bit shared load then hit
// disjoint banks.
template <int THREADS, int SMAX>
__global__ void __launch_bounds__(THREADS, 1)
    k1_staged4_kernel(const __grid_constant__ CUtensorMap bm_map, uint32_t n_boxes, uint64_t n_words,
                      const uint4 *__restrict__ recs, uint64_t n_cand, uint32_t cpc, uint32_t *__restrict__ out,
                      uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr uint32_t G = THREADS / 4;             // groups of 4 lanes
    uint8_t *chunk = smem;                           // n_boxes * 256 rows * 128 B
    const uint32_t chunk_bytes = n_boxes * kStagedRowsPerBox * kStagedWords * 8;
    uint4 *rec_s = reinterpret_cast<uint4 *>(smem + chunk_bytes);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + chunk_bytes + (size_t)cpc * 16);

    const uint32_t tid = threadIdx.x;
    const uint32_t g = tid >> 2, l = tid & 3;
    const uint32_t off_a = ((g & 1) ? 64u : 0u) + l * 16, off_b = ((g & 1) ? 0u : 64u) + l * 16;
    const uint64_t base = (uint64_t)blockIdx.x * cpc;
    if (base >= n_cand) return;
    const uint64_t left = n_cand - base;
    const uint32_t ncta = left < cpc ? (uint32_t)left : cpc;

    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    for (uint32_t i = tid; i < ncta; i += THREADS) rec_s[i] = recs[base + i];
    __syncthreads();

    uint32_t acc[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) acc[s] = 0;
    const uint32_t n_sets = (ncta + 4 * G - 1) / (4 * G);
    const uint64_t n_chunks = (n_words + kStagedWords - 1) / kStagedWords;
    uint32_t phase = 0;
    for (uint64_t ch = 0; ch < n_chunks; ++ch) {
        if (tid == 0) {
            mbar_arrive_expect_tx(bar, chunk_bytes);
            for (uint32_t b = 0; b < n_boxes; ++b)
                tma_load_2d(chunk + (size_t)b * kStagedRowsPerBox * kStagedWords * 8, &bm_map,
                            (int32_t)(ch * kStagedWords), (int32_t)(b * kStagedRowsPerBox), bar);
        }
        const bool ok = mbar_wait_bounded(bar, phase, err);
        phase ^= 1;
        if (__syncthreads_or(!ok)) {
            // give in-flight copies one more bounded chance to land before leaving
            mbar_wait_bounded(bar, phase ^ 1, err);
            return;
        }
#pragma unroll
        for (int s = 0; s < SMAX; ++s) {
            if ((uint32_t)s < n_sets) {
                uint32_t p[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t c = ((uint32_t)s * 4 + j) * G + g;
                    uint32_t v = 0;
                    if (c < ncta) {
                        const uint4 r = rec_s[c];
                        const uint32_t h[4] = {r.x, r.y, r.z, r.w};
                        const uint32_t it0 = h[0] & 0xffffu;
                        if (it0 != kRecNone) {
                            const uint8_t *row = chunk + (size_t)it0 * 128;
                            uint4 ma = *reinterpret_cast<const uint4 *>(row + off_a);
                            uint4 mb = *reinterpret_cast<const uint4 *>(row + off_b);
#pragma unroll
                            for (int k = 1; k < 8; ++k) {
                                const uint32_t it = (h[k >> 1] >> ((k & 1) * 16)) & 0xffffu;
                                if (it == kRecNone) break;
                                const uint8_t *rk = chunk + (size_t)it * 128;
                                ma = and4(ma, *reinterpret_cast<const uint4 *>(rk + off_a));
                                mb = and4(mb, *reinterpret_cast<const uint4 *>(rk + off_b));
                            }
                            v = popc4(ma) + popc4(mb);
                        }
                    }
                    p[j] = v;
                }
                acc[s] += treduce4(p, l);
            }
        }
        __syncthreads();  // every group is done with this chunk before TMA overwrites it
    }
#pragma unroll
    for (int s = 0; s < SMAX; ++s) {
        const uint32_t c = ((uint32_t)s * 4 + l) * G + g;
        if ((uint32_t)s < n_sets && c < ncta) {
            const uint32_t it0 = rec_s[c].x & 0xffffu;
            if (it0 != kRecNone) out[base + c] = acc[s];
        }
    }
}

// ---------------------------------------------------------------- sorted batch supports
// Candidates are counting-sorted by key = (k - 1) * 4096 + first item, so that
// (a) the four 8-lane groups of a warp almost always share k and run one fully
// unrolled, branch-free K-load AND (unused record slots point at an all-ones
// row in shared memory), and (b) consecutive candidates of a group usually
// share their first item, whose 16-byte piece then stays in registers.
// Sorted record: item0 in bits 0..11 and k in bits 12..15 of .x, items 1..7
// as 16-bit fields; pad items = the all-ones row index.
constexpr uint32_t kSortItemMax = 4096;
constexpr uint32_t kSortBins = 8 * kSortItemMax;
constexpr uint32_t kSortCompactMax = 1024;  // 10-bit ids in the 12-byte sorted records

__global__ void sort_count_kernel(const uint64_t *__restrict__ cand_ptr, const uint32_t *__restrict__ cand_items,
                                  uint64_t n, uint32_t d, uint64_t n_txn, uint32_t *__restrict__ bins,
                                  uint32_t *__restrict__ ovf_list, unsigned long long *__restrict__ ovf_count,
                                  uint32_t *__restrict__ out) {
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = cand_ptr[c], b = cand_ptr[c + 1];
        const uint64_t k = b - a;
        if (k == 0) {
            out[c] = (uint32_t)n_txn;
        } else if (k > 8) {
            ovf_list[atomicAdd(ovf_count, 1ull)] = (uint32_t)c;
            out[c] = 0;
        } else {
            uint32_t mn = 0xffffffffu;
            bool zero = false;
            for (uint64_t i = a; i < b; ++i) {
                const uint32_t x = cand_items[i];
                zero |= x >= d;
                mn = min(mn, x);
            }
            if (zero) out[c] = 0;
            else atomicAdd(&bins[(uint32_t)(k - 1) * kSortItemMax + mn], 1u);
        }
    }
}

// Exclusive scan of the bins in place (one CTA of 1024 threads); total -> *n_valid.
__global__ void __launch_bounds__(1024) sort_scan_kernel(uint32_t *__restrict__ bins, uint64_t *__restrict__ n_valid) {
    constexpr uint32_t per = kSortBins / 1024;
    __shared__ uint32_t part[1024];
    const uint32_t t = threadIdx.x;
    uint32_t s = 0;
    for (uint32_t i = 0; i < per; ++i) s += bins[t * per + i];
    part[t] = s;
    __syncthreads();
    for (uint32_t o = 1; o < 1024; o <<= 1) {
        const uint32_t v = t >= o ? part[t - o] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    uint32_t run = t ? part[t - 1] : 0u;
    for (uint32_t i = 0; i < per; ++i) {
        const uint32_t v = bins[t * per + i];
        bins[t * per + i] = run;
        run += v;
    }
    if (t == 1023) *n_valid = part[1023];
}

// Sorted record (12 bytes, ids < 1024): lo = items 0..5 as 10-bit fields and
// k in bits 60..63; hi = items 6..7 as 10-bit fields.  Slots beyond k repeat
// item 0 (AND is idempotent), so no padding row is needed.
__global__ void sort_scatter_kernel(const uint64_t *__restrict__ cand_ptr, const uint32_t *__restrict__ cand_items,
                                    uint64_t n, uint32_t d, uint32_t *__restrict__ cursor,
                                    uint64_t *__restrict__ rec_lo, uint32_t *__restrict__ rec_hi,
                                    uint32_t *__restrict__ perm) {
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = cand_ptr[c], b = cand_ptr[c + 1];
        const uint64_t k = b - a;
        if (k == 0 || k > 8) continue;
        uint32_t it[8];
        uint32_t mn = 0xffffffffu, at = 0;
        bool zero = false;
        for (uint64_t i = a; i < b; ++i) {
            const uint32_t x = cand_items[i];
            zero |= x >= d;
            if (x < mn) { mn = x; at = (uint32_t)(i - a); }
            it[i - a] = x;
        }
        if (zero) continue;
        // the smallest item goes first (it is the sort key and the reused row)
        it[at] = it[0];
        it[0] = mn;
        for (uint64_t i = k; i < 8; ++i) it[i] = mn;
        const uint32_t pos = atomicAdd(&cursor[(uint32_t)(k - 1) * kSortItemMax + mn], 1u);
        uint64_t lo = (uint64_t)k << 60;
#pragma unroll
        for (int i = 0; i < 6; ++i) lo |= (uint64_t)it[i] << (10 * i);
        rec_lo[pos] = lo;
        rec_hi[pos] = it[6] | (it[7] << 10);
        perm[pos] = (uint32_t)c;
    }
}

__device__ __forceinline__ uint32_t rec_item(uint64_t lo, uint32_t hi, int i) {
    return i < 6 ? (uint32_t)(lo >> (10 * i)) & 1023u : (hi >> (10 * (i - 6))) & 1023u;
}

template <int K>
__device__ __forceinline__ uint4 and_tail(const uint8_t *base, uint64_t lo, uint32_t hi, uint4 m) {
#pragma unroll
    for (int i = 1; i < K; ++i) m = and4(m, *reinterpret_cast<const uint4 *>(base + (size_t)rec_item(lo, hi, i) * 128));
    return m;
}

// Same chunk pipeline as k1_staged_kernel.  Group g owns a contiguous run of
// the CTA's sorted candidates, so consecutive candidates usually share k
// (one unrolled K-load AND per warp, K = the warp's largest k) and their
// first item, whose 16-byte piece stays in registers.  Slots past a group's
// run issue no shared loads.
template <int THREADS, int SMAX>
__global__ void __launch_bounds__(THREADS, 1)
    k1_sorted_kernel(const __grid_constant__ CUtensorMap bm_map, uint32_t n_boxes, uint64_t n_words,
                     const uint64_t *__restrict__ rec_lo, const uint32_t *__restrict__ rec_hi,
                     const uint32_t *__restrict__ perm, const uint64_t *__restrict__ n_valid, uint32_t cpc,
                     uint32_t *__restrict__ out, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr uint32_t G = THREADS / 8;
    const uint32_t chunk_bytes = n_boxes * kStagedRowsPerBox * kStagedWords * 8;
    uint8_t *chunk = smem;
    uint64_t *lo_s = reinterpret_cast<uint64_t *>(smem + chunk_bytes);
    uint32_t *hi_s = reinterpret_cast<uint32_t *>(lo_s + cpc);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + chunk_bytes + (size_t)cpc * 12 + 16 - ((size_t)cpc * 12) % 16);

    const uint32_t tid = threadIdx.x, g = tid >> 3, l = tid & 7;
    const uint64_t nv = *n_valid;
    const uint64_t base = (uint64_t)blockIdx.x * cpc;
    if (base >= nv) return;
    const uint32_t ncta = (uint32_t)min((uint64_t)cpc, nv - base);
    const uint32_t per_g = (ncta + G - 1) / G;
    const uint32_t g_lo = min(g * per_g, ncta), g_hi = min(g_lo + per_g, ncta);
    const uint32_t n_sets = (per_g + 7) / 8;

    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    for (uint32_t i = tid; i < ncta; i += THREADS) {
        lo_s[i] = rec_lo[base + i];
        hi_s[i] = rec_hi[base + i];
    }
    __syncthreads();

    uint32_t acc[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) acc[s] = 0;
    const uint64_t n_chunks = (n_words + kStagedWords - 1) / kStagedWords;
    const uint8_t *lane_base = chunk + l * 16;
    uint32_t phase = 0;
    for (uint64_t ch = 0; ch < n_chunks; ++ch) {
        if (tid == 0) {
            mbar_arrive_expect_tx(bar, chunk_bytes);
            for (uint32_t b = 0; b < n_boxes; ++b)
                tma_load_2d(chunk + (size_t)b * kStagedRowsPerBox * kStagedWords * 8, &bm_map,
                            (int32_t)(ch * kStagedWords), (int32_t)(b * kStagedRowsPerBox), bar);
        }
        const bool ok = mbar_wait_bounded(bar, phase, err);
        phase ^= 1;
        if (__syncthreads_or(!ok)) {
            mbar_wait_bounded(bar, phase ^ 1, err);
            return;
        }
#pragma unroll
        for (int s = 0; s < SMAX; ++s) {
            if ((uint32_t)s < n_sets) {
                uint32_t p[8];
                uint32_t cur0 = 0xffffffffu;
                uint4 row0 = make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t c = g_lo + (uint32_t)s * 8 + j;
                    const bool valid = c < g_hi;
                    uint64_t lo = 0;
                    uint32_t hi = 0;
                    if (valid) {
                        lo = lo_s[c];
                        hi = hi_s[c];
                    }
                    const uint32_t k = (uint32_t)(lo >> 60);
                    const uint32_t kmax = __reduce_max_sync(0xffffffffu, k);
                    uint32_t v = 0;
                    if (valid) {
                        const uint32_t it0 = (uint32_t)lo & 1023u;
                        if (it0 != cur0) {
                            row0 = *reinterpret_cast<const uint4 *>(lane_base + (size_t)it0 * 128);
                            cur0 = it0;
                        }
                        uint4 m = row0;
                        switch (kmax) {
                            case 2: m = and_tail<2>(lane_base, lo, hi, m); break;
                            case 3: m = and_tail<3>(lane_base, lo, hi, m); break;
                            case 4: m = and_tail<4>(lane_base, lo, hi, m); break;
                            case 5: m = and_tail<5>(lane_base, lo, hi, m); break;
                            case 6: m = and_tail<6>(lane_base, lo, hi, m); break;
                            case 7: m = and_tail<7>(lane_base, lo, hi, m); break;
                            case 8: m = and_tail<8>(lane_base, lo, hi, m); break;
                            default: break;
                        }
                        v = popc4(m);
                    }
                    p[j] = v;
                }
                acc[s] += treduce8(p, l);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int s = 0; s < SMAX; ++s) {
        const uint32_t c = g_lo + (uint32_t)s * 8 + l;
        if ((uint32_t)s < n_sets && c < g_hi) out[perm[base + c]] = acc[s];
    }
}

constexpr int kStagedThreads = 1024;
constexpr int kStagedSmax = 8;
constexpr int kStagedSmax4 = 8;   // 4-lane groups: 8 sets x 4 candidates x 256 groups = 8,192
constexpr int kSortedSmax = 8;
constexpr uint32_t kSortedMaxCpc = kStagedThreads / 8 * 8 * kSortedSmax;  // 8192

size_t sorted_smem_bytes(uint32_t d, uint32_t cpc) {
    const uint32_t n_boxes = (d + kStagedRowsPerBox - 1) / kStagedRowsPerBox;
    return (size_t)n_boxes * kStagedRowsPerBox * kStagedWords * 8 + (size_t)cpc * 12 + 16 + 64;
}
constexpr uint32_t kStagedMaxCpc = kStagedThreads / 8 * 8 * kStagedSmax;  // 8192

size_t staged_smem_bytes(uint32_t d, uint32_t cpc) {
    const uint32_t n_boxes = (d + kStagedRowsPerBox - 1) / kStagedRowsPerBox;
    return (size_t)n_boxes * kStagedRowsPerBox * kStagedWords * 8 + (size_t)cpc * 16 + 64;
}

bool encode_bitmap_map(CUtensorMap *map, const uint64_t *bitmaps, uint32_t d, uint64_t n_words, uint64_t row_stride) {
    using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !p)
            return false;
        fn = reinterpret_cast<EncodeFn>(p);
    }
    if ((reinterpret_cast<uintptr_t>(bitmaps) & 15) || (row_stride & 1)) return false;
    cuuint64_t dims[2] = {(cuuint64_t)n_words, (cuuint64_t)d};
    cuuint64_t strides[1] = {(cuuint64_t)row_stride * 8};
    cuuint32_t box[2] = {kStagedWords, kStagedRowsPerBox};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<uint64_t *>(bitmaps), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// The kernel of an AUTO call (map: the rows can be staged by TMA); the lines are in support_rule.h.
static SupportKernel auto_kernel(uint64_t n_cand, uint32_t d, uint64_t n_words, bool map) {
    if (!map || d == 0 || support_streams(n_cand, d, n_words)) return SUPPORT_STREAM;
    if (pair_supported(d, n_cand) && support_pairs(n_cand, d, n_words)) return SUPPORT_PAIR;
    return lane_supported(d) ? SUPPORT_LANE_TM : SUPPORT_STAGED4;
}

size_t support_scratch_bytes(uint64_t n_cand, uint32_t d, uint64_t n_words, const SupportPlan &plan,
                             uint64_t hbm_budget) {
    const size_t base = support_scratch_bytes_for(n_cand);
    if (!pair_supported(d, n_cand)) return base;
    const size_t with_pair = align256(base) + pair_scratch_bytes(n_cand, d);
    const bool pair = plan.kernel == SUPPORT_PAIR ||
                      (plan.kernel == SUPPORT_AUTO && with_pair <= hbm_budget / 8 &&
                       auto_kernel(n_cand, d, n_words, true) == SUPPORT_PAIR);
    return pair ? with_pair : base;
}

int support_batch_device(const uint64_t *bitmaps, uint32_t d, uint64_t n_words, uint64_t row_stride,
                         uint64_t n_txn, const uint64_t *cand_ptr, const uint32_t *cand_items, uint64_t n_cand,
                         uint32_t *out, const SupportScratch &scratch, const SupportPlan &plan,
                         const CUtensorMap *map, uint32_t *dev_err, cudaStream_t st, int n_sm, uint64_t *launches,
                         cudaEvent_t *ev) {
    if (n_cand == 0) return 0;
    auto mark = [&](int i) {
        if (ev) SG_CUDA_TRY(cudaEventRecord(ev[i], st));
    };
    const uint64_t n_words_even = (n_words + 1) & ~1ull;
    // default grid: one wave of CTAs for the sorted kernel (its 12-byte records leave room
    // for ~6,600 candidates per CTA), two for the staged kernel
    auto pick_cpc = [&](uint32_t cap, size_t (*smem_fn)(uint32_t, uint32_t), uint32_t waves) -> uint32_t {
        const uint64_t ctas_target = (uint64_t)n_sm * std::max<uint32_t>(1, plan.waves ? plan.waves : waves);
        uint32_t cpc = plan.cands_per_cta;
        if (cpc == 0) cpc = (uint32_t)std::min<uint64_t>(cap, (n_cand + ctas_target - 1) / ctas_target);
        cpc = std::max<uint32_t>(1, std::min(cpc, cap));
        while (cpc > 1 && smem_fn(d, cpc) > 227 * 1024) cpc = cpc * 3 / 4;
        return smem_fn(d, cpc) <= 227 * 1024 ? cpc : 0;
    };
    StreamBatch cs{};
    cs.rows = bitmaps; cs.stride = row_stride; cs.n_words = n_words_even; cs.d = d;
    cs.cand_ptr = cand_ptr; cs.items = cand_items; cs.n = n_cand; cs.n_txn = n_txn; cs.out = out;
    int kind = plan.kernel;
    if (map == nullptr || d == 0) kind = SUPPORT_STREAM;
    // AUTO falls through to the shared-memory lane form, then STAGED4, when a layout does not
    // fit (1M candidates x 1,024 rows: 22.3 ms with records in TMEM, 23.2 in shared memory, staged
    // with 4-lane groups 30.0, with 8-lane groups 30.9, sorted 30.8 - 46)
    const bool gated = kind == SUPPORT_AUTO;
    if (kind == SUPPORT_AUTO) kind = auto_kernel(n_cand, d, n_words_even, map != nullptr);
    const uint32_t *gate = nullptr;
    if (kind == SUPPORT_PAIR) {
        uint32_t *ovf_l = nullptr;
        unsigned long long *ovf_c = nullptr;
        const size_t at = align256(support_scratch_bytes_for(n_cand));   // the lane kernels' scratch comes first
        mark(0);
        if (scratch.bytes > at &&
            pair_supports_device(map, bitmaps, d, n_words_even, row_stride, cand_ptr, cand_items, n_cand, n_txn, out,
                                 static_cast<char *>(scratch.base) + at, scratch.bytes - at, gated, dev_err, st, n_sm,
                                 &gate, &ovf_l, &ovf_c, launches, ev) == 0) {
            StreamBatch tail = cs;
            tail.n_device = reinterpret_cast<const uint64_t *>(ovf_c);
            tail.index = ovf_l;
            launch_cand_stream(tail, st, n_sm);
            if (launches) *launches += 1;
            if (!gated) {
                mark(3);
                return 0;
            }
        }
        kind = lane_supported(d) ? SUPPORT_LANE_TM : SUPPORT_STAGED4;
    }
    if (kind == SUPPORT_LANE || kind == SUPPORT_LANE_TM) {
        uint32_t *ovf_l = nullptr;
        unsigned long long *ovf_c = nullptr;
        // after a gated pair call: these kernels run when it found the data dense.  The host does not
        // know, so the count's time spans both, from the pair kernel's first event to the end of this one
        if (!gate) mark(0);
        cudaEvent_t *lane_ev = gate ? nullptr : ev;
        int rc = -1;
        if (kind == SUPPORT_LANE_TM)
            rc = lane_tm_supports_device(map, d, n_words_even, cand_ptr, cand_items, n_cand, n_txn, out,
                                         scratch.base, scratch.bytes, plan.waves ? plan.waves : 1, dev_err, st, n_sm,
                                         &ovf_l, &ovf_c, launches, lane_ev, gate);
        if (rc != 0)
            rc = lane_supports_device(map, d, n_words_even, cand_ptr, cand_items, n_cand, n_txn, out, scratch.base,
                                      scratch.bytes, kind == SUPPORT_LANE && plan.waves ? plan.waves : 2, dev_err, st,
                                      n_sm, &ovf_l, &ovf_c, launches, lane_ev, gate);
        if (rc == 0) {
            if (gate) mark(2);
            cs.n_device = reinterpret_cast<const uint64_t *>(ovf_c);
            cs.index = ovf_l;
            launch_cand_stream(cs, st, n_sm);
            mark(3);
            if (launches) *launches += 1;
            return 0;
        }
        if (scratch.bytes < support_scratch_bytes_for(n_cand)) return -1;
        kind = SUPPORT_STAGED4;
    }
    if (kind == SUPPORT_SORTED && d > kSortCompactMax) kind = SUPPORT_STAGED;
    if ((kind == SUPPORT_STAGED || kind == SUPPORT_STAGED4) && d > 65535) kind = SUPPORT_STREAM;
    uint32_t cpc = 0;
    if (kind == SUPPORT_SORTED) {
        cpc = pick_cpc(kSortedMaxCpc, sorted_smem_bytes, 1);
        if (!cpc) kind = SUPPORT_STREAM;
    } else if (kind == SUPPORT_STAGED || kind == SUPPORT_STAGED4) {
        cpc = pick_cpc(kStagedMaxCpc, staged_smem_bytes, 2);
        if (!cpc) kind = SUPPORT_STREAM;
    }
    if (kind == SUPPORT_STREAM) {
        mark(0);
        mark(1);
        launch_cand_stream(cs, st, n_sm);
        mark(2);
        mark(3);
        if (launches) *launches += 1;
        return 0;
    }
    if (scratch.bytes < support_scratch_bytes_for(n_cand)) return -1;
    uint8_t *sb = static_cast<uint8_t *>(scratch.base);
    uint4 *recs = reinterpret_cast<uint4 *>(sb);
    uint32_t *ovf = reinterpret_cast<uint32_t *>(sb + align256(n_cand * 16));
    uint32_t *perm = reinterpret_cast<uint32_t *>(sb + align256(n_cand * 16) + align256(n_cand * 4));
    uint32_t *bins = reinterpret_cast<uint32_t *>(sb + align256(n_cand * 16) + 2 * align256(n_cand * 4));
    unsigned long long *ovf_n = reinterpret_cast<unsigned long long *>(
        sb + align256(n_cand * 16) + 2 * align256(n_cand * 4) + align256(kSupportSortBins * 4));
    uint64_t *n_valid = reinterpret_cast<uint64_t *>(ovf_n + 1);
    const uint32_t n_boxes = (d + kStagedRowsPerBox - 1) / kStagedRowsPerBox;
    const unsigned prep_blocks = (unsigned)std::min<uint64_t>((n_cand + 255) / 256, (uint64_t)n_sm * 16);
    const uint64_t ctas = (n_cand + cpc - 1) / cpc;
    mark(0);
    SG_CUDA_TRY(cudaMemsetAsync(ovf_n, 0, 8, st));
    if (kind == SUPPORT_SORTED) {
        SG_CUDA_TRY(cudaMemsetAsync(bins, 0, kSupportSortBins * 4, st));
        sort_count_kernel<<<prep_blocks, 256, 0, st>>>(cand_ptr, cand_items, n_cand, d, n_txn, bins, ovf, ovf_n, out);
        SG_CUDA_TRY(cudaGetLastError());
        sort_scan_kernel<<<1, 1024, 0, st>>>(bins, n_valid);
        SG_CUDA_TRY(cudaGetLastError());
        uint64_t *rec_lo = reinterpret_cast<uint64_t *>(recs);
        uint32_t *rec_hi = reinterpret_cast<uint32_t *>(rec_lo + n_cand);
        sort_scatter_kernel<<<prep_blocks, 256, 0, st>>>(cand_ptr, cand_items, n_cand, d, bins, rec_lo, rec_hi, perm);
        SG_CUDA_TRY(cudaGetLastError());
        const size_t smem = sorted_smem_bytes(d, cpc);
        auto kern = k1_sorted_kernel<kStagedThreads, kSortedSmax>;
        SG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        mark(1);
        kern<<<(unsigned)ctas, kStagedThreads, smem, st>>>(*map, n_boxes, n_words_even, rec_lo, rec_hi, perm, n_valid,
                                                           cpc, out, dev_err);
        SG_CUDA_TRY(cudaGetLastError());
        mark(2);
        if (launches) *launches += 4;
    } else {
        prep_records_kernel<<<prep_blocks, 256, 0, st>>>(cand_ptr, cand_items, n_cand, d, n_txn, recs, ovf, ovf_n,
                                                         out);
        SG_CUDA_TRY(cudaGetLastError());
        const size_t smem = staged_smem_bytes(d, cpc);
        auto kern = kind == SUPPORT_STAGED4 ? k1_staged4_kernel<kStagedThreads, kStagedSmax4>
                                            : k1_staged_kernel<kStagedThreads, kStagedSmax>;
        SG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        mark(1);
        kern<<<(unsigned)ctas, kStagedThreads, smem, st>>>(*map, n_boxes, n_words_even, recs, n_cand, cpc, out,
                                                           dev_err);
        SG_CUDA_TRY(cudaGetLastError());
        mark(2);
        if (launches) *launches += 2;
    }
    // candidates with more than 8 items
    cs.n_device = reinterpret_cast<const uint64_t *>(ovf_n);
    cs.index = ovf;
    launch_cand_stream(cs, st, n_sm);
    mark(3);
    if (launches) *launches += 1;
    return 0;
}

// ---------------------------------------------------------------- wait self-test
// An mbarrier that nothing ever arrives at: every thread's bounded wait runs
// out, records DEVERR_MBAR_TIMEOUT and returns.  No copy or MMA is issued, so
// nothing is in flight when the CTA leaves.
__global__ void wait_probe_kernel(uint32_t *err) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    mbar_wait_bounded(&bar, 0, err);
}

void launch_wait_probe(uint32_t *err, cudaStream_t st) {
    wait_probe_kernel<<<1, 32, 0, st>>>(err);
    SG_CUDA_TRY(cudaGetLastError());
}

// ---------------------------------------------------------------- projected databases
// A row restricted to the transactions of a root row, packed in their order.  A
// block takes 256 words of the root: where its transactions start is the sum of the
// blocks' popcounts before it (projection_sums_kernel), where its words' start a
// scan.  The move masks of the compress of a root word, after H. S. Warren,
// Hacker's Delight, 2nd ed., section 7-4 (six steps, step i shifting the bits under
// mask i right by 2^i), depend on the root alone: they stay in registers while the
// block goes through its items, eight at a time, packing into shared memory; whole
// output words leave as plain stores, the two it shares with its neighbours by an
// atomic on the cleared row.  (A launch of one CTA for the starts, masks kept in
// memory and read again for each item, and an L2 atomic per input word took 18 + 3
// + 31 us a root (31,250 words, 320 items on average), 74 ms with the clearing in a
// 2,000,000-transaction search of 633 roots and their candidate pools; this way 57,
// with the listed form below for sparse roots 47.)
constexpr int kProjWords = 256;    // root words per block
constexpr int kProjItems = 8;      // items packed between two barriers
constexpr int kProjGroup = 32;     // items per block

// blocks [0, n_chunks): sums[b] = set bits of the root's words [256 b, 256 (b+1));
// the blocks after them clear one item's output row each
__global__ void __launch_bounds__(kProjWords) projection_sums_kernel(const uint64_t *__restrict__ root, uint64_t n_words,
                                                                    uint32_t n_chunks, uint32_t *__restrict__ sums,
                                                                    const uint32_t *__restrict__ items,
                                                                    uint64_t *__restrict__ out, uint64_t out_stride,
                                                                    uint64_t out_words) {
    if (blockIdx.x >= n_chunks) {
        uint64_t *row = out + (uint64_t)items[blockIdx.x - n_chunks] * out_stride;
        for (uint64_t w = 2 * threadIdx.x; w < out_words; w += 2 * kProjWords)
            *reinterpret_cast<ulonglong2 *>(row + w) = make_ulonglong2(0, 0);
        return;
    }
    __shared__ uint32_t part[kProjWords / 32];
    const uint64_t w = (uint64_t)blockIdx.x * kProjWords + threadIdx.x;
    const uint32_t c = __reduce_add_sync(0xffffffffu, w < n_words ? (uint32_t)popc64(root[w]) : 0u);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (uint32_t i = 0; i < kProjWords / 32; ++i) t += part[i];
        sums[blockIdx.x] = t;
    }
}

// Where a chunk's set bits start in the packed row (base: the chunks before), where
// this thread's word starts in the chunk, and the chunk's total.
__device__ __forceinline__ void chunk_positions(uint32_t c, const uint32_t *sums, uint32_t chunk, uint32_t t,
                                                uint32_t lane, uint32_t wid, uint32_t *s_part, uint32_t *s_base,
                                                uint32_t &base, uint32_t &mine, uint32_t &tot) {
    uint32_t incl = c, before = 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += x;
    }
    for (uint32_t b = t; b < chunk; b += kProjWords) before += sums[b];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 31) s_part[wid] = incl;
    if (lane == 0) s_base[wid] = before;
    __syncthreads();
    base = tot = 0;
    mine = incl - c;
#pragma unroll
    for (uint32_t i = 0; i < kProjWords / 32; ++i) {
        base += s_base[i];
        if (i < wid) mine += s_part[i];
        tot += s_part[i];
    }
}

__global__ void __launch_bounds__(kProjWords) project_rows_kernel(const uint64_t *__restrict__ rows, uint64_t stride,
                                                                 uint64_t n_words, const uint64_t *__restrict__ root,
                                                                 const uint32_t *__restrict__ sums,
                                                                 const uint32_t *__restrict__ items, uint32_t n_items,
                                                                 unsigned long long *__restrict__ out,
                                                                 uint64_t out_stride) {
    constexpr uint32_t kBuf = kProjWords + 1;   // output words a block touches at most
    __shared__ unsigned long long buf[kProjItems][kBuf + 1];
    __shared__ uint32_t s_part[kProjWords / 32], s_base[kProjWords / 32];
    const uint32_t t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const uint64_t w = (uint64_t)blockIdx.x * kProjWords + t;
    const uint64_t m = w < n_words ? root[w] : 0;
    const uint32_t c = popc64(m);
    uint32_t base, mine, tot;
    chunk_positions(c, sums, blockIdx.x, t, lane, wid, s_part, s_base, base, mine, tot);
    if (tot == 0) return;
    const uint32_t first = base >> 6, n_out = ((base + tot - 1) >> 6) - first + 1;
    const uint32_t pos = base + mine - (first << 6);   // of the word's first bit, in the block's buffer
    const bool own_first = (base & 63) == 0, own_last = ((base + tot) & 63) == 0;
    uint64_t mv[6];
    {
        uint64_t x = m, mk = ~m << 1;   // ones at positions whose lower neighbour is a zero of m
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            uint64_t mp = mk ^ (mk << 1);   // parallel suffix (prefix xor towards the high end)
            mp ^= mp << 2;
            mp ^= mp << 4;
            mp ^= mp << 8;
            mp ^= mp << 16;
            mp ^= mp << 32;
            mv[i] = mp & x;                 // bits that move by 2^i in this step
            x = (x ^ mv[i]) | (mv[i] >> (1 << i));
            mk &= ~mp;
        }
    }
    const uint32_t g0 = blockIdx.y * kProjGroup, g1 = min(n_items, g0 + kProjGroup);
    for (uint32_t g = g0; g < g1; g += kProjItems) {
        const uint32_t n = min((uint32_t)kProjItems, g1 - g);
        uint64_t x[kProjItems];
#pragma unroll
        for (uint32_t i = 0; i < kProjItems; ++i)
            x[i] = i < n && m ? rows[(uint64_t)items[g + i] * stride + w] & m : 0;
#pragma unroll
        for (uint32_t i = 0; i < kProjItems; ++i)
            for (uint32_t k = t; k <= n_out; k += kProjWords) buf[i][k] = 0;
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < kProjItems; ++i) {
            uint64_t v = x[i];
            if (v == 0) continue;
#pragma unroll
            for (int k = 0; k < 6; ++k) v = (v & ~mv[k]) | ((v & mv[k]) >> (1 << k));
            const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32), sh = pos & 31;
            uint32_t *to = reinterpret_cast<uint32_t *>(buf[i]) + (pos >> 5);
            const uint32_t a = lo << sh, b = __funnelshift_l(lo, hi, sh), e = __funnelshift_l(hi, 0u, sh);
            if (a) atomicOr(to, a);
            if (b) atomicOr(to + 1, b);
            if (e) atomicOr(to + 2, e);
        }
        __syncthreads();
        for (uint32_t i = 0; i < n; ++i) {
            unsigned long long *dst = out + (uint64_t)items[g + i] * out_stride + first;
            for (uint32_t k = t; k < n_out; k += kProjWords) {
                const unsigned long long v = buf[i][k];
                if ((k > 0 || own_first) && (k + 1 < n_out || own_last)) dst[k] = v;
                else if (v) atomicOr(dst + k, v);
            }
        }
        __syncthreads();
    }
}

// A sparse root's transactions are listed instead, and a warp packs 1,024 of them
// per item: each lane fetches the bits at 32 of its positions into one word and the
// warp transposes the words (180 instructions per 1,024 output bits, against about
// 70 for every 32 words of the whole row above).
constexpr int kListItems = 8;      // items per warp

__global__ void __launch_bounds__(kProjWords) projection_list_kernel(const uint64_t *__restrict__ root, uint64_t n_words,
                                                                    const uint32_t *__restrict__ sums,
                                                                    uint32_t *__restrict__ list, uint32_t n_list) {
    __shared__ uint32_t s_part[kProjWords / 32], s_base[kProjWords / 32];
    const uint32_t t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const uint64_t w = (uint64_t)blockIdx.x * kProjWords + t;
    uint32_t base, at, tot;
    uint64_t m = w < n_words ? root[w] : 0;
    chunk_positions(popc64(m), sums, blockIdx.x, t, lane, wid, s_part, s_base, base, at, tot);
    at += base;
    for (; m; m &= m - 1, ++at)
        if (at < n_list) list[at] = (uint32_t)(w * 64) + (__ffsll((long long)m) - 1);
}

__global__ void __launch_bounds__(256) project_listed_kernel(const uint64_t *__restrict__ rows, uint64_t stride,
                                                             uint64_t n_words, const uint32_t *__restrict__ list,
                                                             uint32_t n_list,
                                                             const uint32_t *__restrict__ items, uint32_t n_items,
                                                             uint64_t *__restrict__ out, uint64_t out_stride,
                                                             uint64_t out_words) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t unit = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);   // 1,024 output bits
    if (unit * 16 >= out_words) return;
    const uint32_t first = (uint32_t)(unit * 1024);
    const uint32_t g1 = min(n_items, (blockIdx.y + 1) * kListItems);
    if (unit * 1024 >= n_list) {   // past the packed bits: zeros
        for (uint32_t g = blockIdx.y * kListItems; g < g1; ++g)
            if (unit * 32 + lane < 2 * out_words)
                reinterpret_cast<uint32_t *>(out + (uint64_t)items[g] * out_stride)[unit * 32 + lane] = 0;
        return;
    }
    uint32_t pos[32];
#pragma unroll
    for (uint32_t i = 0; i < 32; ++i) {
        const uint64_t at = (uint64_t)first + i * 32 + lane;
        pos[i] = at < n_list ? list[at] : 0xffffffffu;
        if ((pos[i] >> 6) >= n_words) pos[i] = 0xffffffffu;
    }
#pragma unroll 1
    for (uint32_t g = blockIdx.y * kListItems; g < g1; ++g) {
        const uint32_t e = items[g];
        const uint32_t *src = reinterpret_cast<const uint32_t *>(rows + (uint64_t)e * stride);
        uint32_t bits = 0;   // bit i: of position pos[i]
#pragma unroll
        for (uint32_t i0 = 0; i0 < 32; i0 += 16) {
            uint32_t v[16];
#pragma unroll
            for (uint32_t i = 0; i < 16; ++i) v[i] = pos[i0 + i] != 0xffffffffu ? __ldg(src + (pos[i0 + i] >> 5)) : 0u;
#pragma unroll
            for (uint32_t i = 0; i < 16; ++i) bits = __funnelshift_r(bits, __funnelshift_r(v[i], 0u, pos[i0 + i]), 1);
        }
        const uint32_t word = transpose32(bits, lane);
        const uint64_t to = unit * 32 + lane;
        if (to < 2 * out_words) reinterpret_cast<uint32_t *>(out + (uint64_t)e * out_stride)[to] = word;
    }
}

uint64_t projection_chunks(uint64_t n_words) { return (n_words + kProjWords - 1) / kProjWords; }
// By instructions the two meet at about 12 set bits a word.
bool projection_listed(uint64_t n_set, uint64_t n_words) { return n_set <= 10 * n_words; }

void launch_projection(const uint64_t *rows, uint64_t stride, uint64_t n_words, uint32_t root_row, uint64_t n_set,
                       const uint32_t *items, uint32_t n_items, uint32_t *sums, uint32_t *list, uint64_t *out,
                       uint64_t out_stride, uint64_t out_words, cudaStream_t st) {
    if (n_items == 0 || out_words == 0) return;
    const uint64_t *root = rows + (uint64_t)root_row * stride;
    const uint32_t chunks = (uint32_t)projection_chunks(n_words);
    const bool listed = projection_listed(n_set, n_words);
    const uint32_t clear = listed ? 0 : n_items;   // the listed kernel writes whole rows
    if (chunks + clear) {
        projection_sums_kernel<<<chunks + clear, kProjWords, 0, st>>>(root, n_words, chunks, sums, items, out,
                                                                      out_stride, out_words);
        SG_CUDA_TRY(cudaGetLastError());
    }
    if (listed) {
        if (chunks) {
            projection_list_kernel<<<chunks, kProjWords, 0, st>>>(root, n_words, sums, list, (uint32_t)n_set);
            SG_CUDA_TRY(cudaGetLastError());
        }
        const uint64_t units = (out_words + 15) / 16;
        project_listed_kernel<<<dim3((unsigned)((units + 7) / 8), (n_items + kListItems - 1) / kListItems), 256, 0, st>>>(
            rows, stride, n_words, list, (uint32_t)n_set, items, n_items, out, out_stride, out_words);
    } else if (chunks) {
        project_rows_kernel<<<dim3(chunks, (n_items + kProjGroup - 1) / kProjGroup), kProjWords, 0, st>>>(
            rows, stride, n_words, root, sums, items, n_items, reinterpret_cast<unsigned long long *>(out), out_stride);
    }
    SG_CUDA_TRY(cudaGetLastError());
}

// ---------------------------------------------------------------- miner helpers
// Masks of new nodes: mask(child) = mask(parent) AND the listed rows.  A warp takes
// 256 words of one child, four 16-byte pieces per lane in flight.  (One 16-byte
// piece per thread behind a 64-bit division: 22 ms of a 2,000,000-transaction
// search, 11 this way, and 5 with masks for expanding nodes alone.)
__global__ void __launch_bounds__(256) child_mask_kernel(uint64_t *__restrict__ arena, uint64_t astride, uint64_t n_words,
                                                        const uint64_t *__restrict__ rows, uint64_t rstride,
                                                        const uint64_t *__restrict__ ptr,
                                                        const uint32_t *__restrict__ items,
                                                        const uint32_t *__restrict__ parent_slot,
                                                        const uint32_t *__restrict__ child_slot, uint32_t n,
                                                        uint32_t n_steps) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t total = (uint64_t)n * n_steps;
    for (uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; i < total; i += n_warps) {
        const uint32_t c = (uint32_t)(i / n_steps);
        const uint64_t w = (i - (uint64_t)c * n_steps) * kQueryStep + 2 * lane;
        const uint32_t ps = parent_slot[c];
        const uint64_t a = ptr[c], b = ptr[c + 1];
        const uint64_t *from = ps != kNoSlot ? arena + (uint64_t)ps * astride + w : nullptr;
        uint64_t *to = arena + (uint64_t)child_slot[c] * astride + w;
        uint4 r[kQueryU];
#pragma unroll
        for (uint32_t u = 0; u < kQueryU; ++u)
            r[u] = from && w + 64 * u < n_words ? *reinterpret_cast<const uint4 *>(from + 64 * u)
                                                : make_uint4(~0u, ~0u, ~0u, ~0u);
        for (uint64_t j = a; j < b; ++j) {
            const uint64_t *row = rows + (uint64_t)items[j] * rstride + w;
#pragma unroll
            for (uint32_t u = 0; u < kQueryU; ++u)
                if (w + 64 * u < n_words) r[u] = and4(r[u], ld_nc_v4(row + 64 * u));
        }
#pragma unroll
        for (uint32_t u = 0; u < kQueryU; ++u)
            if (w + 64 * u < n_words) *reinterpret_cast<uint4 *>(to + 64 * u) = r[u];
    }
}

void launch_child_masks(uint64_t *arena, uint64_t arena_stride, uint64_t n_words, const uint64_t *rows,
                        uint64_t row_stride, const uint64_t *ptr, const uint32_t *items, const uint32_t *parent_slot,
                        const uint32_t *child_slot, uint32_t n, cudaStream_t st, int n_sm) {
    if (n == 0 || n_words == 0) return;
    const uint32_t n_steps = (uint32_t)((n_words + kQueryStep - 1) / kQueryStep);
    const unsigned blocks = (unsigned)std::min<uint64_t>(((uint64_t)n * n_steps + 7) / 8, (uint64_t)n_sm * 32);
    child_mask_kernel<<<blocks, 256, 0, st>>>(arena, arena_stride, n_words, rows, row_stride, ptr, items, parent_slot,
                                              child_slot, n, n_steps);
    SG_CUDA_TRY(cudaGetLastError());
}

__global__ void pool_append_kernel(unsigned long long *__restrict__ pool, uint64_t pstride,
                                   const uint64_t *__restrict__ set_ptr, const uint32_t *__restrict__ set_items,
                                   uint64_t first, uint32_t n_sets, const uint64_t *__restrict__ set_col) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n_sets; s += gridDim.x * blockDim.x) {
        const uint64_t m = set_col ? set_col[s] : first + s;
        for (uint64_t i = set_ptr[s]; i < set_ptr[s + 1]; ++i)
            atomicOr(&pool[(uint64_t)set_items[i] * pstride + (m >> 6)], 1ull << (m & 63));
    }
}

void launch_pool_append(uint64_t *pool_rows, uint64_t pool_stride, const uint64_t *set_ptr, const uint32_t *set_items,
                        uint64_t first_member, uint32_t n_sets, cudaStream_t st, const uint64_t *set_col) {
    if (n_sets == 0) return;
    const unsigned blocks = std::min<unsigned>((n_sets + 255) / 256, 1024);
    pool_append_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<unsigned long long *>(pool_rows), pool_stride,
                                               set_ptr, set_items, first_member, n_sets, set_col);
    SG_CUDA_TRY(cudaGetLastError());
}

}  // namespace sg
