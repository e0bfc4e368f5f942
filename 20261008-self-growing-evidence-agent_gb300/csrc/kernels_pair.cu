// kernels_pair.cu -- batched supports of many candidates, grouped by their two rarest items.
//
// Reference counterpart: the AND-popcount counting of kernel_bitmap.cu:412-442
// (one candidate per launch there) and of the wave engine, kernel_bmma.cu:603-768.
//
// For sparse data.  Most of what a support count reads it reads for nothing:
// once the AND of the first rows is empty over a stretch of transactions, the
// other rows cannot matter there, and two candidates that share items read and
// AND the same rows twice.  So the candidates' items are put in ascending order
// of support, the candidates are grouped by their first two items, and a lane
// counts a group of up to eight candidates: it ANDs the pair's 1,024-transaction
// slices once, keeps a bit per 32-bit word that is not empty, and reads the
// candidates' further rows, rarest first, only at those words.
//
// Steps (all on the device, no host synchronisation):
//   row supports (sampled), ranks       pair_sup_kernel, pair_rank_kernel
//   is the data sparse enough?          pair_sample_kernel, pair_gate_kernel
//   records, pair histogram             pair_records_kernel
//   groups per size, group numbers      pair_sizes_kernel, pair_assign_kernel
//   records in group order              pair_scatter_kernel
//   counting                            pair_lane_kernel
//   supports to the caller's order      pair_out_kernel
//
// The counting kernel keeps the chunk pipeline of k1_lane_tm_kernel
// (kernels_lane.cu): the rows' 128-byte slices of a chunk staged by TMA in a
// ring of 32-KB box slots, lane q of a phase reading piece i XOR q at step i
// (conflict-free), and the groups' row ids in tensor memory.  Groups of one
// size fill sets of 32 (one per lane); sets are dealt round-robin to the CTAs,
// largest first, and inside a CTA to the four TMEM quadrants, whose warps take
// them from a shared counter once per chunk.  Counts of a chunk go to the
// group-ordered totals with one coalesced reduction per candidate that has any.
//
// Bound: shared-memory wavefronts and instruction issue, about equally.
// Measured, 1,048,576 transactions x 1,024 rows (2 - 20% dense), 1,000,000
// candidates of 3..8 items: 13.4 ms a call against 22.4 for k1_lane_tm_kernel,
// which reads every row (600,000 candidates: 10.0 / 14.8; 300,000: 7.8 / 9.0).
// Groups of up to 4, 6 and 8: 14.0, 13.8 and 13.4 ms.  ncu at 200,000 transactions:
// 65 wavefronts and 230 warp instructions per 32 candidates and chunk (176
// wavefronts for every row), shared-memory pipe 49%, issue slots 52%, the rest the
// chunk boundaries.  Counting a pair group with a warp straight from L2 instead
// took 14.1 ms for 600,000 candidates.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "support_rule.h"
#include "tcgen05.cuh"

namespace sg {
namespace {

constexpr uint32_t kPairItems = 16;       // items of a record (longer candidates are streamed)
constexpr uint32_t kPairGroup = 8;        // candidates of a group
constexpr uint32_t kPairBoxRows = 256;
constexpr uint32_t kPairWords = 16;       // words per row per chunk
constexpr uint32_t kPairBoxBytes = kPairBoxRows * kPairWords * 8;   // 32 KB
constexpr int kPairThreads = 1024;
constexpr uint32_t kPairQuadSets = 96;    // sets a quadrant's table holds
constexpr uint32_t kPairSamples = 1024, kPairSampleChunks = 16;
constexpr uint32_t kNoRow = 0xffffffffu;

// Items 0..15 as 16-bit rows in ascending support; slots past the last repeat
// it.  Rows take 11 bits: the top four bits of slot 0 hold the item count - 1.
struct PairRec {
    uint4 lo, hi;
};

// Counters of one call (device).
struct PairCtl {
    uint32_t dense;                      // the gate: 1 = too dense for this path
    uint32_t sampled, live, items;       // words sampled, how many were not empty, their candidates' items
    uint32_t groups[kPairGroup + 1];     // groups of each size
    uint32_t cursor[kPairGroup + 1];
    unsigned long long ovf_n;            // candidates with more items than a record holds
};

struct PairScratch {
    PairCtl *ctl;
    uint32_t *sup, *rank;      // d each
    uint32_t *table;           // d * d: candidates per pair
    uint2 *base;               // d * d: numbers of its first full group and of its last group
    PairRec *rec, *sorted;     // n and n_slots
    uint32_t *ord;             // n: ordinal inside the pair
    uint32_t *head, *next2;    // n_slots: a group's pair (slot of its candidate 0); a candidate's third and fourth rows
    uint32_t *perm, *total;    // n_slots: candidate (kNoRow: none) and its count
    uint32_t *ovf;             // n
    uint64_t n_slots;
    size_t bytes;
};

// Slots: the candidates, and up to 31 empty lanes in the last set of each size.
constexpr uint64_t pair_slots(uint64_t n) { return n + 32 * (kPairGroup * (kPairGroup + 1) / 2); }

PairScratch pair_layout(void *base, uint64_t n, uint32_t d) {
    PairScratch s{};
    size_t at = 0;
    auto take = [&](size_t b) {
        void *p = base ? static_cast<char *>(base) + at : nullptr;
        at += align256(b);
        return p;
    };
    s.n_slots = pair_slots(n);
    s.ctl = static_cast<PairCtl *>(take(sizeof(PairCtl)));
    s.sup = static_cast<uint32_t *>(take((size_t)d * 4));
    s.rank = static_cast<uint32_t *>(take((size_t)d * 4));
    s.table = static_cast<uint32_t *>(take((size_t)d * d * 4));
    s.base = static_cast<uint2 *>(take((size_t)d * d * 8));
    s.rec = static_cast<PairRec *>(take(n * sizeof(PairRec)));
    s.sorted = static_cast<PairRec *>(take(s.n_slots * sizeof(PairRec)));
    s.ord = static_cast<uint32_t *>(take(n * 4));
    s.head = static_cast<uint32_t *>(take(s.n_slots * 4));
    s.next2 = static_cast<uint32_t *>(take(s.n_slots * 4));
    s.perm = static_cast<uint32_t *>(take(s.n_slots * 4));
    s.total = static_cast<uint32_t *>(take(s.n_slots * 4));
    s.ovf = static_cast<uint32_t *>(take(n * 4));
    s.bytes = at;
    return s;
}

// Bits of every row in evenly spread pieces, a sixteenth of its words: the ranks
// only choose which rows are read first.
constexpr uint32_t kSupPiece = 64, kSupEvery = 16;   // words
__global__ void __launch_bounds__(256) pair_sup_kernel(const uint64_t *__restrict__ rows, uint64_t stride,
                                                       uint64_t n_words, uint32_t d, uint32_t *__restrict__ sup) {
    const uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (e >= d) return;
    const uint64_t *row = rows + (uint64_t)e * stride;
    uint32_t c = 0;
    for (uint64_t w = 2 * lane; w < n_words; w += kSupPiece * kSupEvery) c += popc4(ld_nc_v4(row + w));
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) sup[e] = c;
}

// rank[e]: position of row e in ascending (support, row) order; a warp per row.
__global__ void pair_rank_kernel(const uint32_t *__restrict__ sup, uint32_t d, uint32_t *__restrict__ rank) {
    const uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (e >= d) return;
    const uint32_t s = sup[e];
    uint32_t c = 0;
    for (uint32_t f = lane; f < d; f += 32) c += sup[f] < s || (sup[f] == s && f < e);
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) rank[e] = c;
}

__device__ __forceinline__ uint32_t rec_a(uint32_t w) { return w & 0x0fffu; }
__device__ __forceinline__ uint32_t rec_b(uint32_t w) { return w >> 16; }
__device__ __forceinline__ uint32_t rec_k(uint32_t w) { return ((w >> 12) & 15u) + 1; }

// Table entry of a pair: the pairs with the most common first rows come first, so
// the lanes of a set have about as many live words each and a CTA's long sets
// are taken early.
__device__ __forceinline__ uint64_t pair_index(const PairScratch &s, uint32_t ab, uint32_t d) {
    return (uint64_t)(d - 1 - s.rank[rec_a(ab)]) * d + (d - 1 - s.rank[rec_b(ab)]);
}

// The record of a candidate of 1..16 known rows; false when a row is unknown.
__device__ __forceinline__ bool make_record(const uint32_t *__restrict__ items, uint32_t k, uint32_t d,
                                            const uint32_t *__restrict__ rank, PairRec &r) {
    uint32_t key[kPairItems];   // rank << 16 | row, unused slots last
    bool known = true;
#pragma unroll
    for (uint32_t i = 0; i < kPairItems; ++i) {
        key[i] = 0xffffffffu;
        if (i < k) {
            const uint32_t x = items[i];
            known &= x < d;
            if (x < d) key[i] = rank[x] << 16 | x;
        }
    }
    if (!known) return false;
#pragma unroll
    for (uint32_t i = 1; i < kPairItems; ++i) {
        if (i < k) {
#pragma unroll
            for (uint32_t j = i; j > 0; --j) {
                const uint32_t lo = min(key[j - 1], key[j]), hi = max(key[j - 1], key[j]);
                key[j - 1] = lo;
                key[j] = hi;
            }
        }
    }
    uint32_t w[kPairItems / 2], last = key[0];
#pragma unroll
    for (uint32_t i = 0; i < kPairItems; ++i) {
        if (i < k) last = key[i];
        if (i & 1) w[i >> 1] |= last << 16;
        else w[i >> 1] = last & 0xffffu;
    }
    r.lo = make_uint4(w[0] | (k - 1) << 12, w[1], w[2], w[3]);
    r.hi = make_uint4(w[4], w[5], w[6], w[7]);
    return true;
}

// One thread per candidate: its record, and its ordinal among the candidates of
// its pair.  Empty candidates, unknown ids and candidates of more than 16 items
// are settled here (ord = ~0) or listed.
__global__ void __launch_bounds__(256) pair_records_kernel(const uint64_t *__restrict__ cand_ptr,
                                                           const uint32_t *__restrict__ items, uint64_t n, uint32_t d,
                                                           uint64_t n_txn, PairScratch s, uint32_t *__restrict__ out) {
    if (s.ctl->dense) return;
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = cand_ptr[c], k = cand_ptr[c + 1] - a;
        out[c] = k == 0 ? (uint32_t)n_txn : 0u;
        s.ord[c] = 0xffffffffu;
        if (k > kPairItems) s.ovf[atomicAdd(&s.ctl->ovf_n, 1ull)] = (uint32_t)c;
        if (k == 0 || k > kPairItems) continue;
        PairRec r;
        if (!make_record(items + a, (uint32_t)k, d, s.rank, r)) continue;
        s.rec[c] = r;
        s.ord[c] = atomicAdd(&s.table[pair_index(s, r.lo.x, d)], 1u);
    }
}

// The gate: how many 32-bit words of a pair's AND hold a bit, over candidates and
// chunks spread evenly over the call.  A warp per (candidate, chunk): one word
// of 64 bits for every other lane.
__global__ void __launch_bounds__(256) pair_sample_kernel(const uint64_t *__restrict__ rows, uint64_t stride,
                                                          uint64_t n_words, const uint64_t *__restrict__ cand_ptr,
                                                          const uint32_t *__restrict__ items, uint64_t n, uint32_t d,
                                                          PairScratch s) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t si = w / kPairSampleChunks, ci = w % kPairSampleChunks;
    if (si >= kPairSamples) return;
    const uint64_t c = n * si / kPairSamples;
    const uint64_t a = cand_ptr[c], k = cand_ptr[c + 1] - a;
    PairRec r;
    if (k == 0 || k > kPairItems || !make_record(items + a, (uint32_t)k, d, s.rank, r)) return;
    const uint32_t ab = r.lo.x;
    const uint64_t chunks = (n_words + kPairWords - 1) / kPairWords;
    const uint64_t at = (chunks * ci / kPairSampleChunks) * kPairWords + (lane >> 1);
    uint64_t v = 0;
    if (at < n_words) v = rows[(uint64_t)rec_a(ab) * stride + at] & rows[(uint64_t)rec_b(ab) * stride + at];
    const uint32_t half = lane & 1 ? (uint32_t)(v >> 32) : (uint32_t)v;
    const uint32_t live = __popc(__ballot_sync(0xffffffffu, half != 0));
    if (lane == 0) {
        atomicAdd(&s.ctl->live, live);
        atomicAdd(&s.ctl->sampled, 32u);
        atomicAdd(&s.ctl->items, (uint32_t)k);
    }
}

__global__ void pair_gate_kernel(PairCtl *ctl, uint64_t n, uint32_t d) {
    ctl->dense = pair_dense(ctl->live, ctl->sampled, ctl->items, n, d);
}

// Groups of each size over all pairs: cnt / kPairGroup full ones, and one of the rest.
__global__ void __launch_bounds__(256) pair_sizes_kernel(PairScratch s, uint64_t pairs) {
    __shared__ uint32_t num[kPairGroup + 1];
    if (s.ctl->dense) return;
    if (threadIdx.x <= kPairGroup) num[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < pairs; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = s.table[i];
        if (c >= kPairGroup) atomicAdd(&num[kPairGroup], c / kPairGroup);
        if (c % kPairGroup) atomicAdd(&num[c % kPairGroup], 1u);
    }
    __syncthreads();
    if (threadIdx.x <= kPairGroup && num[threadIdx.x]) atomicAdd(&s.ctl->groups[threadIdx.x], num[threadIdx.x]);
}

// Group numbers inside each size: a tile of 256 pairs reserves its runs with one
// atomic per size.
__global__ void __launch_bounds__(256) pair_assign_kernel(PairScratch s, uint64_t pairs) {
    __shared__ uint32_t num[kPairGroup + 1], first[kPairGroup + 1];
    if (s.ctl->dense) return;
    for (uint64_t i0 = (uint64_t)blockIdx.x * 256; i0 < pairs; i0 += (uint64_t)gridDim.x * 256) {
        if (threadIdx.x <= kPairGroup) num[threadIdx.x] = 0;
        __syncthreads();
        const uint64_t i = i0 + threadIdx.x;
        const uint32_t c = i < pairs ? s.table[i] : 0;
        uint32_t full = 0, rest = 0;
        if (c >= kPairGroup) full = atomicAdd(&num[kPairGroup], c / kPairGroup);
        if (c % kPairGroup) rest = atomicAdd(&num[c % kPairGroup], 1u);
        __syncthreads();
        if (threadIdx.x <= kPairGroup && num[threadIdx.x])
            first[threadIdx.x] = atomicAdd(&s.ctl->cursor[threadIdx.x], num[threadIdx.x]);
        __syncthreads();
        if (c)
            s.base[i] = make_uint2(c >= kPairGroup ? first[kPairGroup] + full : 0,
                                   c % kPairGroup ? first[c % kPairGroup] + rest : 0);
        __syncthreads();
    }
}

// First set and first slot of size g (sizes descend; a set is 32 groups of one size).
__device__ __forceinline__ void size_start(const PairCtl *ctl, uint32_t g, uint32_t &set, uint32_t &slot) {
    set = slot = 0;
    for (uint32_t h = kPairGroup; h > g; --h) {
        const uint32_t sets = (ctl->groups[h] + 31) / 32;
        set += sets;
        slot += sets * h * 32;
    }
}

__global__ void __launch_bounds__(256) pair_scatter_kernel(PairScratch s, uint64_t n, uint32_t d) {
    if (s.ctl->dense) return;
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t o = s.ord[c];
        if (o == 0xffffffffu) continue;
        const PairRec r = s.rec[c];
        const uint64_t pair = pair_index(s, r.lo.x, d);
        const uint32_t cnt = s.table[pair];
        const uint2 base = s.base[pair];
        const bool in_full = o < cnt / kPairGroup * kPairGroup;
        const uint32_t size = in_full ? kPairGroup : cnt % kPairGroup;
        const uint32_t group = in_full ? base.x + o / kPairGroup : base.y, j = o % kPairGroup;
        uint32_t set, slot;
        size_start(s.ctl, size, set, slot);
        slot += (group / 32) * size * 32 + j * 32 + (group & 31);
        s.sorted[slot] = r;
        s.perm[slot] = (uint32_t)c;
        s.total[slot] = 0;
        if (j == 0) s.head[slot] = rec_a(r.lo.x) | (r.lo.x & 0xffff0000u);
        // rows three and four (a short candidate repeats its last row); bit 15: more rows follow
        s.next2[slot] = r.lo.y | (rec_k(r.lo.x) > 4 ? 0x8000u : 0u);
    }
}

__device__ __forceinline__ uint32_t lds32(const uint8_t *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ uint32_t tm_ld1_async(uint32_t taddr) {
    uint32_t v;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr) : "memory");
    return v;
}

// Shared-memory offset of a row's slice: chunk = first box's offset in the ring
// plus the lane's rotation; the ring wraps at ring bytes.
__device__ __forceinline__ uint32_t row_at(uint32_t row, uint32_t chunk, uint32_t ring) {
    const uint32_t t = (row << 7) + chunk;
    return min(t, t - ring);
}

// A group's pair over half of its slice of a chunk, pieces 0..3 of the lane's rotated
// order or, with oa and ob moved by 64 (XOR), pieces 4..7: bit w of the result is set when
// 32-bit word w of the half (piece w / 4) holds a bit.
__device__ __forceinline__ uint32_t pair_words(const uint8_t *smem, uint32_t oa, uint32_t ob) {
    uint32_t z = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        const uint4 x = *reinterpret_cast<const uint4 *>(smem + (oa ^ (i << 4)));
        const uint4 y = *reinterpret_cast<const uint4 *>(smem + (ob ^ (i << 4)));
        if (x.x & y.x) z |= 1u << (4 * i);
        if (x.y & y.y) z |= 2u << (4 * i);
        if (x.z & y.z) z |= 4u << (4 * i);
        if (x.w & y.w) z |= 8u << (4 * i);
    }
    return z;
}

// The G candidates of every lane's group at the lane's live words z.  tcols:
// their TMEM columns (third and fourth row each); slot: the set's first slot
// plus the lane.
template <int G>
__device__ __forceinline__ void count_words(uint32_t tcols, const uint8_t *smem, uint32_t oa, uint32_t ob, uint32_t z,
                                            uint32_t chunk, uint32_t ring, uint64_t slot, const PairScratch &s) {
    uint32_t cd[G], oc[G], od[G], more = 0;
#pragma unroll
    for (int g = 0; g < G; ++g) cd[g] = tm_ld1_async(tcols + g);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int g = 0; g < G; ++g) {
        asm volatile("" : "+r"(cd[g]));   // not before the wait
        oc[g] = row_at(cd[g] & 0x07ffu, chunk, ring);
        od[g] = row_at(cd[g] >> 16, chunk, ring);
        more |= ((cd[g] >> 15) & 1u) << g;
    }
    // the words where the first four rows still have a bit
    uint32_t hit[G];
#pragma unroll
    for (int g = 0; g < G; ++g) hit[g] = 0;
    while (z) {
        const uint32_t w = (uint32_t)__ffs((int)z) - 1, bit = 1u << w, sh = w << 2;
        z &= z - 1;
        const uint32_t p = lds32(smem + (oa ^ sh)) & lds32(smem + (ob ^ sh));
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (p & lds32(smem + (oc[g] ^ sh)) & lds32(smem + (od[g] ^ sh))) hit[g] |= bit;
    }
    __syncwarp();
    // few words get here: count them, with the record's other rows (from L1/L2)
#pragma unroll
    for (int g = 0; g < G; ++g) {
        uint32_t tot = 0;
        while (hit[g]) {
            const uint32_t sh = ((uint32_t)__ffs((int)hit[g]) - 1) << 2;
            hit[g] &= hit[g] - 1;
            uint32_t v = lds32(smem + (oa ^ sh)) & lds32(smem + (ob ^ sh)) & lds32(smem + (oc[g] ^ sh)) &
                         lds32(smem + (od[g] ^ sh));
            if ((more >> g) & 1u) {
                const uint16_t *it = reinterpret_cast<const uint16_t *>(s.sorted + slot + 32 * g);
                const uint32_t k = (__ldg(it) >> 12) + 1u;
                for (uint32_t i = 4; i < k && v; ++i)
                    v &= lds32(smem + (row_at(__ldg(it + i), chunk, ring) ^ sh));
            }
            tot += __popc(v);
        }
        if (tot) atomicAdd(s.total + slot + 32 * g, tot);
    }
}

__global__ void __launch_bounds__(kPairThreads, 1)
    pair_lane_kernel(const __grid_constant__ CUtensorMap bm_map, uint32_t n_boxes, uint32_t n_ring, uint64_t n_words,
                     PairScratch s, uint32_t tm_cols, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)n_ring * kPairBoxBytes);   // one per ring slot
    unsigned long long *issued_s = reinterpret_cast<unsigned long long *>(full + n_ring);
    uint32_t *ctr = reinterpret_cast<uint32_t *>(issued_s + 1);      // [quadrant][chunk parity]
    uint32_t *tslot = ctr + 8;
    uint32_t *slot0 = tslot + 1;                                     // [quadrant][set]: first slot
    uint16_t *cols = reinterpret_cast<uint16_t *>(slot0 + 4 * kPairQuadSets);   // column << 4 | size
    uint32_t *nq_s = reinterpret_cast<uint32_t *>(cols + 4 * kPairQuadSets);    // sets of each quadrant
    if (s.ctl->dense) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3;
    const uint32_t G = gridDim.x, cta = blockIdx.x;

    if (warp == 0) tmem_alloc(tslot, tm_cols);
    if (tid == 0) {
        for (uint32_t i = 0; i < n_ring; ++i) mbar_init(&full[i], 1);
        fence_mbar_init();
        for (int i = 0; i < 8; ++i) ctr[i] = 0;
        *issued_s = 0;
    }
    if (tid >= 32 && tid < 36) {   // this CTA's sets, quadrant by quadrant
        const uint32_t q = tid - 32;
        uint32_t m = 0, col = 0, size = kPairGroup, set_lo = 0, slot_lo = 0;
        uint32_t sets = (s.ctl->groups[size] + 31) / 32;
        for (uint64_t set = cta + (uint64_t)q * G; m < kPairQuadSets; set += 4ull * G) {
            while (size && set >= set_lo + sets) {
                set_lo += sets;
                slot_lo += sets * size * 32;
                --size;
                sets = size ? (s.ctl->groups[size] + 31) / 32 : 0;
            }
            if (!size || col + 1 + size > tm_cols) break;   // (the host's bound on the columns rules the second out)
            slot0[q * kPairQuadSets + m] = slot_lo + (uint32_t)(set - set_lo) * size * 32;
            cols[q * kPairQuadSets + m] = (uint16_t)(col << 4 | size);
            col += 1 + size;
            ++m;
        }
        nq_s[q] = m;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot, tq = tbase + ((quad * 32u) << 16);
    const uint32_t nq = nq_s[quad];
    const uint32_t *my_slot0 = slot0 + quad * kPairQuadSets;
    const uint16_t *my_cols = cols + quad * kPairQuadSets;
    for (uint32_t m = warp >> 2; m < nq; m += 8) {
        const uint32_t at = my_cols[m], size = at & 15u, taddr = tq + (at >> 4);
        const uint64_t slot = (uint64_t)my_slot0[m] + lane;
        for (uint32_t g = 0; g <= size; ++g) {
            const uint32_t v = g == 0 ? s.head[slot] : s.next2[slot + 32 * (g - 1)];
            asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr + g), "r"(v) : "memory");
        }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");

    const uint32_t rot = (lane & 7) << 4, ring = n_ring * kPairBoxBytes;
    const uint64_t n_chunks = (n_words + kPairWords - 1) / kPairWords;
    const uint64_t total = n_chunks * n_boxes;
    bool ok = true;
    for (uint64_t ch = 0; ch < n_chunks; ++ch) {
        if (tid == 0) {
            // a ring slot is free once the chunk of its last box is done: every chunk before ch is
            uint64_t b = *issued_s;
            const uint64_t lim = min(total, ch * n_boxes + n_ring);
            for (; b < lim; ++b) {
                const uint32_t sl = (uint32_t)(b % n_ring);
                mbar_arrive_expect_tx(&full[sl], kPairBoxBytes);
                tma_load_2d(smem + (size_t)sl * kPairBoxBytes, &bm_map, (int32_t)((b / n_boxes) * kPairWords),
                            (int32_t)((b % n_boxes) * kPairBoxRows), &full[sl]);
            }
            *issued_s = b;
        }
        for (uint32_t b = 0; b < n_boxes && ok; ++b) {
            const uint64_t g = ch * n_boxes + b;
            ok = mbar_wait_bounded(&full[g % n_ring], (uint32_t)((g / n_ring) & 1), err);
        }
        tc_fence_before();
        if (__syncthreads_or(!ok)) {
            ok = false;   // the same for every thread: the paths below hold warp-wide TMEM operations
            break;
        }
        tc_fence_after();
        const uint32_t chunk = ((uint32_t)((ch * n_boxes) % n_ring) << 15) + rot;
        uint32_t *my_ctr = ctr + quad * 2 + (uint32_t)(ch & 1);
        // work units: a set's first and second half of the slice (shorter units even out the warps' ends)
        uint32_t m = 0;
        if (lane == 0) m = atomicAdd(my_ctr, 1u);
        m = __shfl_sync(0xffffffffu, m, 0);
        while (m < 2 * nq) {
            const uint32_t at = my_cols[m >> 1], taddr = tq + (at >> 4), size = at & 15u;
            const uint64_t slot = (uint64_t)my_slot0[m >> 1] + lane;
            const uint32_t here = chunk ^ ((m & 1) << 6);
            uint32_t ab = tm_ld1_async(taddr);
            if (lane == 0) m = atomicAdd(my_ctr, 1u);   // the next unit's number, while this one is counted
            asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(ab)::"memory");
            const bool used = ab != kNoRow;
            if (!used) ab = 0;
            const uint32_t oa = row_at(ab & 0xffffu, here, ring), ob = row_at(ab >> 16, here, ring);
            uint32_t z = pair_words(smem, oa, ob);
            if (!used) z = 0;
            if (__any_sync(0xffffffffu, z)) {
                uint32_t first = 0;
                if (size >= 4) {
                    count_words<4>(taddr + 1, smem, oa, ob, z, here, ring, slot, s);
                    first = 4;
                }
                for (; first + 2 <= size; first += 2)
                    count_words<2>(taddr + 1 + first, smem, oa, ob, z, here, ring, slot + 32 * first, s);
                if (first < size)
                    count_words<1>(taddr + 1 + first, smem, oa, ob, z, here, ring, slot + 32 * first, s);
            }
            m = __shfl_sync(0xffffffffu, m, 0);
        }
        __syncthreads();   // every warp is done with this chunk's ring slots
        if (tid < 4) ctr[tid * 2 + (uint32_t)(ch & 1)] = 0;   // next used by chunk ch + 2
    }
    if (!ok) {
        // a wait ran out: let the copies still in flight land (bounded) before the
        // CTA's shared memory goes away
        const uint64_t b1 = *issued_s;
        for (uint64_t b = b1 > n_ring ? b1 - n_ring : 0; b < b1; ++b)
            mbar_wait_bounded(&full[b % n_ring], (uint32_t)((b / n_ring) & 1), err);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tbase, tm_cols);
    }
}

__global__ void __launch_bounds__(256) pair_out_kernel(PairScratch s, uint32_t *__restrict__ out) {
    if (s.ctl->dense) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < s.n_slots; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = s.perm[i];
        if (c != kNoRow) out[c] = s.total[i];
    }
}

size_t pair_smem_bytes(uint32_t n_ring) {
    return (size_t)n_ring * kPairBoxBytes + (size_t)n_ring * 8 + 8 + 9 * 4 + 4 * kPairQuadSets * 6 + 4 * 4 + 64;
}

}  // namespace

bool pair_supported(uint32_t d, uint64_t n_cand) {
    // the rows' 32-KB boxes of one chunk fit the ring; sets fit the quadrants' tables at up to 8 CTAs per SM
    return d > 0 && d <= 7 * kPairBoxRows && n_cand <= (1ull << 24);
}
size_t pair_scratch_bytes(uint64_t n_cand, uint32_t d) { return pair_layout(nullptr, n_cand, d).bytes; }

int pair_supports_device(const CUtensorMap *map, const uint64_t *bitmaps, uint32_t d, uint64_t n_words,
                         uint64_t row_stride, const uint64_t *cand_ptr, const uint32_t *cand_items, uint64_t n_cand,
                         uint64_t n_txn, uint32_t *out, void *scratch, size_t scratch_bytes, bool gated,
                         uint32_t *dev_err, cudaStream_t st, int n_sm, const uint32_t **dense, uint32_t **ovf_list,
                         unsigned long long **ovf_count, uint64_t *launches, cudaEvent_t *ev) {
    if (!pair_supported(d, n_cand) || n_cand == 0) return -1;
    const PairScratch s = pair_layout(scratch, n_cand, d);
    if (s.bytes > scratch_bytes) return -1;
    const uint32_t n_boxes = (d + kPairBoxRows - 1) / kPairBoxRows;
    uint32_t n_ring = 0;
    while (pair_smem_bytes(n_ring + 1) <= 227 * 1024) ++n_ring;
    if (n_ring < n_boxes) return -1;
    // CTAs: one per SM while every quadrant's sets (at most n / 32 + 8 of them over the grid, dealt
    // evenly) fit its table, and their columns (1 + size each, at most 2 n / 32 + 52) its 512
    uint32_t waves = 1;
    const uint64_t most_sets = n_cand / 32 + kPairGroup, most_cols = 2 * (n_cand / 32) + 52;
    while (most_sets / (4ull * n_sm * waves) + 1 > kPairQuadSets ||
           most_cols / (4ull * n_sm * waves) + 2 + kPairGroup > 512)
        ++waves;
    const uint64_t pairs = (uint64_t)d * d;
    const unsigned pair_blocks = (unsigned)std::min<uint64_t>((pairs + 255) / 256, (uint64_t)n_sm * 8);
    const unsigned cand_blocks = (unsigned)std::min<uint64_t>((n_cand + 255) / 256, (uint64_t)n_sm * 8);
    SG_CUDA_TRY(cudaMemsetAsync(s.ctl, 0, sizeof(PairCtl), st));
    SG_CUDA_TRY(cudaMemsetAsync(s.table, 0, pairs * 4, st));
    SG_CUDA_TRY(cudaMemsetAsync(s.head, 0xff, s.n_slots * 4, st));
    SG_CUDA_TRY(cudaMemsetAsync(s.perm, 0xff, s.n_slots * 4, st));
    pair_sup_kernel<<<(d + 7) / 8, 256, 0, st>>>(bitmaps, row_stride, n_words, d, s.sup);
    SG_CUDA_TRY(cudaGetLastError());
    pair_rank_kernel<<<(d + 7) / 8, 256, 0, st>>>(s.sup, d, s.rank);
    SG_CUDA_TRY(cudaGetLastError());
    if (gated) {
        pair_sample_kernel<<<kPairSamples * kPairSampleChunks / 8, 256, 0, st>>>(bitmaps, row_stride, n_words, cand_ptr,
                                                                                      cand_items, n_cand, d, s);
        SG_CUDA_TRY(cudaGetLastError());
        pair_gate_kernel<<<1, 1, 0, st>>>(s.ctl, n_cand, d);
        SG_CUDA_TRY(cudaGetLastError());
    }
    pair_records_kernel<<<cand_blocks, 256, 0, st>>>(cand_ptr, cand_items, n_cand, d, n_txn, s, out);
    SG_CUDA_TRY(cudaGetLastError());
    pair_sizes_kernel<<<pair_blocks, 256, 0, st>>>(s, pairs);
    SG_CUDA_TRY(cudaGetLastError());
    pair_assign_kernel<<<pair_blocks, 256, 0, st>>>(s, pairs);
    SG_CUDA_TRY(cudaGetLastError());
    pair_scatter_kernel<<<cand_blocks, 256, 0, st>>>(s, n_cand, d);
    SG_CUDA_TRY(cudaGetLastError());
    const size_t smem = pair_smem_bytes(n_ring);
    SG_CUDA_TRY(cudaFuncSetAttribute(pair_lane_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (ev) SG_CUDA_TRY(cudaEventRecord(ev[1], st));
    pair_lane_kernel<<<(unsigned)n_sm * waves, kPairThreads, smem, st>>>(*map, n_boxes, n_ring, n_words, s, 512, dev_err);
    SG_CUDA_TRY(cudaGetLastError());
    if (ev) SG_CUDA_TRY(cudaEventRecord(ev[2], st));
    pair_out_kernel<<<cand_blocks, 256, 0, st>>>(s, out);
    SG_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += gated ? 10 : 8;
    *dense = &s.ctl->dense;
    *ovf_list = s.ovf;
    *ovf_count = &s.ctl->ovf_n;
    return 0;
}

}  // namespace sg
