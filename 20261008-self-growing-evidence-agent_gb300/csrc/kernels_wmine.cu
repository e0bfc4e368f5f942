// kernels_wmine.cu -- batched per-window MFI mining on the ring.
//
// The reference mines one window per engine process (code/pipeline/
// skab_spike.py:61-80 builds the windows; the engines' DFS is
// kernel_bitmap.cu:841-894); its result for a window is the MFI set of that
// window's transactions at the window's floor, which these kernels reproduce.
//
// Representation.  Items are the ring's dense ids 0..d-1 (d <= 64*MW); an
// itemset is an MW-word mask.  A task's base database is the window's
// transactions that contain the task's required items, found through the ring's
// vertical rows; their item masks are read from the ring's horizontal masks.
// wvtask_kernel (the default) turns them into vertical rows, one bit per entry
// per item, and keeps one tidset per search level: counts are AND-popcounts of
// the level's tidset with the item rows.  wtask_kernel
// (SGFIM_F_WINDOWS_HORIZONTAL) instead stacks each level's projected database as
// entries, restricted to the level's tail.
//
// Search.  Depth-first over the set-enumeration tree, one node at a time per
// warp, children in ascending (support, id) order -- the order under which a
// candidate found later is never a proper superset of one found earlier in
// the same subtree: child j's subtree lacks item f_i of every earlier sibling
// i < j, which all candidates of sibling i contain.  Every node applies
//   counts  c_e = |t(H u {e})|, e in T       (ballot popcounts over entries)
//   PEP     c_e == sup(H) (and >= thr)       -> e joins H
//   leaf    F = {e : thr <= c_e < sup(H)} empty: H is a candidate
//   HUT     H u F inside a known MFI          -> nothing new below
//   FHUT    |t(H u F)| >= thr                  -> H u F is the only candidate
// and candidates are checked against the MFIs found so far that contain the
// node's head (the "local MFI" list: the parent's list filtered to members
// containing the child's head, plus everything found inside the parent's
// subtree, which contains the parent's head by construction).
//
// Work split.  A window shorter than 64 transactions is one task: its warp
// searches the whole tree and its pool is the exact MFI set.  Longer windows
// are split at the root: wroot_kernel counts the root and sorts its frequent
// tail f_0..f_{k-1}; task (w, j) searches child j's subtree alone.  The
// costliest children are expanded the same way (wsub_kernel) and their children
// become the tasks, the costliest of these once more.  Tasks share no pool, so a
// candidate of one subtree may sit inside a candidate of an earlier subtree
// in depth-first order (never of a later one, by the argument above);
// the wfilter kernels remove exactly those with a vertical bitmap of the window's
// candidates, and wgather_kernel writes the kept candidates in window order.
//
// Work is distributed by atomic counters (costliest tasks first); every
// loop is bounded by list lengths, and any capacity overflow (entry stack,
// local-MFI stack, pool, depth, filter scratch) marks the window for the
// host-driven wave miner instead of producing a partial result.
#include <cstddef>

#include "common.cuh"
#include "kernels.h"

namespace sg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

template <int MW> struct Mask {
    uint64_t w[MW];
};

template <int MW> __device__ __forceinline__ uint64_t m_word(const Mask<MW> &m, uint32_t i) {
    // arithmetic selection: no indexable copy of m
    uint64_t r = 0;
#pragma unroll
    for (int k = 0; k < MW; ++k) r |= m.w[k] & (0ull - (uint64_t)((uint32_t)k == i));
    return r;
}
template <int MW> __device__ __forceinline__ bool m_has(const Mask<MW> &m, uint32_t e) {
    return (m_word(m, e >> 6) >> (e & 63)) & 1ull;
}
template <int MW> __device__ __forceinline__ void m_set(Mask<MW> &m, uint32_t e) {
    const uint64_t bit = 1ull << (e & 63);
#pragma unroll
    for (int k = 0; k < MW; ++k) m.w[k] |= bit & (0ull - (uint64_t)((uint32_t)k == (e >> 6)));
}
template <int MW> __device__ __forceinline__ bool m_nz(const Mask<MW> &m) {
    uint64_t x = 0;
#pragma unroll
    for (int i = 0; i < MW; ++i) x |= m.w[i];
    return x != 0;
}
// a subset of b
template <int MW> __device__ __forceinline__ bool m_sub(const Mask<MW> &a, const Mask<MW> &b) {
    uint64_t x = 0;
#pragma unroll
    for (int i = 0; i < MW; ++i) x |= a.w[i] & ~b.w[i];
    return x == 0;
}
template <int MW> __device__ __forceinline__ Mask<MW> m_and(const Mask<MW> &a, const Mask<MW> &b) {
    Mask<MW> r;
#pragma unroll
    for (int i = 0; i < MW; ++i) r.w[i] = a.w[i] & b.w[i];
    return r;
}
template <int MW> __device__ __forceinline__ Mask<MW> m_zero() {
    Mask<MW> r;
#pragma unroll
    for (int i = 0; i < MW; ++i) r.w[i] = 0;
    return r;
}
// 16-byte vector accesses: every mask array is 16-byte aligned (MW even)
template <int MW> __device__ __forceinline__ Mask<MW> m_load(const uint64_t *p) {
    static_assert(MW % 2 == 0, "mask width must be even");
    Mask<MW> r;
#pragma unroll
    for (int i = 0; i < MW; i += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p + i);
        r.w[i] = v.x;
        r.w[i + 1] = v.y;
    }
    return r;
}
template <int MW> __device__ __forceinline__ void m_store(uint64_t *p, const Mask<MW> &m) {
#pragma unroll
    for (int i = 0; i < MW; i += 2) *reinterpret_cast<ulonglong2 *>(p + i) = make_ulonglong2(m.w[i], m.w[i + 1]);
}
template <int MW> __device__ __forceinline__ Mask<MW> warp_or(const Mask<MW> &m) {
    Mask<MW> r;
#pragma unroll
    for (int i = 0; i < MW; ++i) {
        const uint32_t lo = __reduce_or_sync(kFull, (uint32_t)m.w[i]);
        const uint32_t hi = __reduce_or_sync(kFull, (uint32_t)(m.w[i] >> 32));
        r.w[i] = ((uint64_t)hi << 32) | lo;
    }
    return r;
}

// Per-level record of the search stack (global memory, one stack per warp).
template <int MW> struct alignas(16) WLevel {
    uint64_t hp[MW];        // head after PEP
    uint64_t list_off;      // first entry of this node's projected database
    uint32_t list_n;
    uint32_t lm_off, lm_n;  // local-MFI list (pool indices)
    uint32_t entry;         // pool size when the node was entered
    uint32_t k, j;          // frequent tail size, next child
    uint32_t end;           // children to search: k, or a task's part of them
    uint8_t f[128];         // frequent tail, ascending (support, id)
    uint32_t c[128];        // supports of f
};

// An expanded node of a split window: its root (wroot_kernel), or a child of an
// expanded node that is split again (wsub_kernel).  Its children are tasks, or
// expanded in turn.
template <int MW> struct alignas(16) WRoot {
    uint64_t hp[MW];        // head after PEP (items in every transaction of the node)
    uint64_t cand[MW];      // the node's only MFI when it is terminal
    uint32_t cand_sup;
    uint32_t has_cand;      // 1: the subtree's MFIs are {cand}; 0: the children (k of them) hold them
    uint32_t k;
    uint32_t pad;
    uint8_t f[128];
    uint32_t c[128];
    uint64_t req[MW];       // the items that were chosen on the way here: the node's transactions hold them
};

// the host reads these fields of the root records (ring.cu)
static_assert(offsetof(WRoot<2>, cand) == 16 && offsetof(WRoot<2>, cand_sup) == 32 &&
                  offsetof(WRoot<2>, has_cand) == 36 && offsetof(WRoot<2>, k) == 40 &&
                  offsetof(WRoot<2>, f) == 48 && offsetof(WRoot<2>, c) == 176,
              "root record layout read by sgfim_ring_mine_windows");

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The search stack holds itemsets of up to kWDepth - 1 items.
constexpr int kWDepth = 48;
// chunks of 32 entries loaded before any is processed (memory-level parallelism)
constexpr int kU = 4;

// One projected-database entry: ring slot (start + i) of the window, or entry
// i of the warp's stack.
template <int MW> __device__ __forceinline__ const uint64_t *entry_ptr(bool ring, const WMineParams &p, uint64_t start,
                                                                      const uint64_t *lists, uint64_t off, uint32_t i) {
    return ring ? p.hm + ((start + i) & p.cap_mask) * MW : lists + (off + i) * MW;
}

// c_e over the database (lane 0 accumulates into the warp's counters cnt[128]).
template <int MW>
__device__ __forceinline__ void count_items(bool ring, const WMineParams &p, uint64_t start, const uint64_t *lists,
                                            uint64_t off, uint32_t n, const Mask<MW> &T, uint32_t *cnt,
                                            uint32_t lane) {
    for (uint32_t q = lane; q < 128; q += 32) cnt[q] = 0;
    __syncwarp();
    for (uint32_t b = 0; b < n; b += 32 * kU) {
        Mask<MW> m[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t i = b + u * 32 + lane;
            m[u] = i < n ? m_and(m_load<MW>(entry_ptr<MW>(ring, p, start, lists, off, i)), T) : m_zero<MW>();
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const Mask<MW> om = warp_or(m[u]);
#pragma unroll
            for (int ww = 0; ww < MW; ++ww) {
                const uint64_t mine = m[u].w[ww];
                uint64_t x = om.w[ww];
                while (x) {
                    const uint32_t bit = __ffsll((long long)x) - 1;
                    x &= x - 1;
                    const uint32_t c = __popc(__ballot_sync(kFull, (mine >> bit) & 1ull));
                    if (lane == 0) cnt[ww * 64 + bit] += c;
                }
            }
        }
    }
    __syncwarp();
}

// PEP items P and frequent tail F of a node from its counts.
template <int MW>
__device__ __forceinline__ void classify(const Mask<MW> &T, const uint32_t *cnt, uint32_t d, uint32_t thr, uint32_t sup,
                                         uint32_t lane, Mask<MW> &P, Mask<MW> &F) {
    P = m_zero<MW>();
    F = m_zero<MW>();
#pragma unroll
    for (int q = 0; q < 2 * MW; ++q) {
        const uint32_t e = q * 32 + lane;
        const bool inT = e < d && ((T.w[q >> 1] >> ((q & 1) * 32 + lane)) & 1ull);
        const uint32_t c = inT ? cnt[e] : 0;
        const uint32_t bp = __ballot_sync(kFull, inT && c >= thr && c == sup);
        const uint32_t bf = __ballot_sync(kFull, inT && c >= thr && c < sup);
        P.w[q >> 1] |= (uint64_t)bp << ((q & 1) * 32);
        F.w[q >> 1] |= (uint64_t)bf << ((q & 1) * 32);
    }
}

// |{entries containing F}|
template <int MW>
__device__ __forceinline__ uint32_t count_superset(bool ring, const WMineParams &p, uint64_t start,
                                                   const uint64_t *lists, uint64_t off, uint32_t n,
                                                   const Mask<MW> &F, uint32_t lane) {
    uint32_t cf = 0;
    for (uint32_t b = 0; b < n; b += 32 * kU) {
        bool h[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t i = b + u * 32 + lane;
            h[u] = i < n && m_sub(F, m_load<MW>(entry_ptr<MW>(ring, p, start, lists, off, i)));
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) cf += __popc(__ballot_sync(kFull, h[u]));
    }
    return cf;
}

// F sorted by (count, id) ascending into f[], c[] (the lanes own the 4*MW/2
// items lane, lane+32, ...; one pass over F compares against all of them).
template <int MW>
__device__ __forceinline__ void sort_tail(const Mask<MW> &F, const uint32_t *cnt, uint32_t lane, uint8_t *f,
                                          uint32_t *c) {
    uint32_t ce[2 * MW], rank[2 * MW];
#pragma unroll
    for (int q = 0; q < 2 * MW; ++q) {
        const uint32_t e = q * 32 + lane;
        ce[q] = ((F.w[q >> 1] >> ((q & 1) * 32 + lane)) & 1ull) ? cnt[e] : 0xffffffffu;
        rank[q] = 0;
    }
#pragma unroll
    for (int ww = 0; ww < MW; ++ww) {
        uint64_t x = F.w[ww];
        while (x) {
            const uint32_t e2 = ww * 64 + (__ffsll((long long)x) - 1);
            x &= x - 1;
            const uint32_t c2 = cnt[e2];
#pragma unroll
            for (int q = 0; q < 2 * MW; ++q) {
                const uint32_t e = q * 32 + lane;
                rank[q] += (c2 < ce[q]) || (c2 == ce[q] && e2 < e);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 2 * MW; ++q) {
        if (ce[q] != 0xffffffffu) {
            f[rank[q]] = (uint8_t)(q * 32 + lane);
            c[rank[q]] = ce[q];
        }
    }
}

// Child database: entries holding every item of req, restricted to Tc,
// non-empty, written at dst .. dst+cn of the warp's stack.  Returns cn, or
// 0xffffffff on overflow.
template <int MW>
__device__ __forceinline__ uint32_t build_child(bool ring, const WMineParams &p, uint64_t start, uint64_t *lists,
                                                uint64_t src_off, uint32_t src_n, const Mask<MW> &req,
                                                const Mask<MW> &Tc, uint64_t dst, uint32_t lane) {
    uint32_t cn = 0;
    for (uint32_t b = 0; b < src_n; b += 32 * kU) {
        Mask<MW> m[kU];
        bool keep[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t i = b + u * 32 + lane;
            m[u] = m_zero<MW>();
            keep[u] = false;
            if (i < src_n) {
                const Mask<MW> r = m_load<MW>(entry_ptr<MW>(ring, p, start, lists, src_off, i));
                m[u] = m_and(r, Tc);
                keep[u] = m_sub(req, r) && m_nz(m[u]);
            }
        }
        // the child's entries go after the source's: writes never touch entries still to be read
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t bal = __ballot_sync(kFull, keep[u]);
            const uint64_t pos = dst + cn + __popc(bal & ((1u << lane) - 1));
            if (keep[u] && pos < p.list_cap) m_store(lists + pos * MW, m[u]);
            cn += __popc(bal);
        }
    }
    return dst + cn > p.list_cap ? 0xffffffffu : cn;
}


// Tidset words a lane keeps in registers (tidsets of up to 128 words).
constexpr uint32_t kReg = 4;

// cnt[i] = popc(tidset AND row(items[i])), four items at a time, a lane per word;
// R: words per lane (0: the tidset is read from tid).  Two sums share a reduction
// while the database has fewer than 65,536 entries.
template <int R>
__device__ __forceinline__ void count_tail(const uint32_t *rows, uint32_t vw, uint32_t W, const uint32_t (&tr)[kReg],
                                           const uint32_t *tid, const uint8_t *items, uint32_t nt, bool two,
                                           uint32_t *cnt, uint32_t lane) {
#pragma unroll 1
    for (uint32_t i = 0; i < nt; i += 4) {
        const uint32_t *r[4];
        uint32_t a[4] = {0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < 4; ++u) r[u] = rows + (uint32_t)items[min(i + u, nt - 1)] * vw;
        if (R > 0) {
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (lane + 32 * k < W)
#pragma unroll
                    for (int u = 0; u < 4; ++u) a[u] += __popc(tr[k] & r[u][lane + 32 * k]);
        } else {
#pragma unroll 2
            for (uint32_t x = lane; x < W; x += 32) {
                const uint32_t v = tid[x];
#pragma unroll
                for (int u = 0; u < 4; ++u) a[u] += __popc(v & r[u][x]);
            }
        }
        if (two) {
            const uint32_t s = __reduce_add_sync(kFull, a[0] | a[1] << 16), t = __reduce_add_sync(kFull, a[2] | a[3] << 16);
            a[0] = s & 0xffffu;
            a[1] = s >> 16;
            a[2] = t & 0xffffu;
            a[3] = t >> 16;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = __reduce_add_sync(kFull, a[u]);
        }
        if (lane == 0) *reinterpret_cast<uint4 *>(cnt + i) = make_uint4(a[0], a[1], a[2], a[3]);
    }
}

// Support of the node's head with all k items, rarest first, or any number below
// thr once it falls below.
template <int R>
__device__ __forceinline__ uint32_t count_all(const uint32_t *rows, uint32_t vw, uint32_t W, const uint32_t (&tr)[kReg],
                                              const uint8_t *items, uint32_t k, uint32_t thr, uint32_t lane) {
    uint32_t v[R], cf = 0;
#pragma unroll
    for (int x = 0; x < R; ++x) v[x] = tr[x];
#pragma unroll 1
    for (uint32_t i = 0; i < k; i += 2) {
        const uint32_t *r0 = rows + (uint32_t)items[i] * vw, *r1 = rows + (uint32_t)items[min(i + 1, k - 1)] * vw;
        uint32_t a = 0;
#pragma unroll
        for (int x = 0; x < R; ++x)
            if (lane + 32 * x < W) {
                v[x] &= r0[lane + 32 * x] & r1[lane + 32 * x];
                a += __popc(v[x]);
            }
        cf = __reduce_add_sync(kFull, a);
        if (cf < thr) break;
    }
    return cf;
}

}  // namespace

// ------------------------------------------------------------------ expanded nodes
// Supports come from the ring's vertical rows: the node's transactions are the
// window's bit range ANDed with the rows of the items chosen so far (one row per
// item, 64 transactions per word), and an item's support is the popcount of that
// with its row.  A node's words are taken 128 at a time, four per lane.

namespace {

// The window's words of a node, four per lane from word b on: its bits in words
// b + lane + 32 u of the window.
template <int MW> struct NodeWords {
    uint64_t w0, nwd, m_first, m_last, cwm;
    const uint64_t *rows;
    uint64_t ring_words;
    __device__ NodeWords(const WMineParams &p, uint64_t start, uint32_t n) {
        // unwrapped words w0 .., masked at both ends; ring words: a power of two
        w0 = start >> 6;
        nwd = n ? ((start + n - 1) >> 6) - w0 + 1 : 0;
        m_first = ~0ull << (start & 63);
        m_last = n ? (~0ull >> (63 - ((start + n - 1) & 63))) : 0;
        cwm = p.ring_words - 1;
        rows = p.ring_rows;
        ring_words = p.ring_words;
    }
    __device__ __forceinline__ uint64_t word(uint32_t e, uint64_t i) const {
        return rows[(uint64_t)e * ring_words + ((w0 + i) & cwm)];
    }
    __device__ __forceinline__ void load(uint64_t b, const Mask<MW> &req, uint32_t lane, uint64_t (&v)[4]) const {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t i = b + lane + 32 * u;
            v[u] = 0;
            if (i < nwd) {
                v[u] = ~0ull;
                if (i == 0) v[u] &= m_first;
                if (i + 1 == nwd) v[u] &= m_last;
            }
        }
#pragma unroll
        for (int ww = 0; ww < MW; ++ww)
            for (uint64_t x = req.w[ww]; x; x &= x - 1) {
                const uint32_t e = ww * 64 + (__ffsll((long long)x) - 1);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (v[u]) v[u] &= word(e, b + lane + 32 * u);
            }
    }
};

// Finishes a node from its items' supports cnt[e], e in T: PEP, the frequent tail,
// FHUT over the node's words, and the record (one warp).
template <int MW>
__device__ __forceinline__ void finish_node(const WMineParams &p, const NodeWords<MW> &nw, const Mask<MW> &H,
                                            const Mask<MW> &T, const Mask<MW> &req, uint32_t sup, uint32_t thr,
                                            const uint32_t *cnt, uint32_t lane, WRoot<MW> &S) {
    Mask<MW> P, F;
    classify<MW>(T, cnt, p.d, thr, sup, lane, P, F);
    Mask<MW> Hp, cand;
    uint32_t k = 0;
#pragma unroll
    for (int i = 0; i < MW; ++i) {
        Hp.w[i] = H.w[i] | P.w[i];
        cand.w[i] = Hp.w[i];
        k += __popcll(F.w[i]);
    }
    uint32_t has = 0, csup = 0;
    if (k == 0) {
        has = m_nz(Hp) ? 1u : 0u;   // (a root without any item has no candidate)
        csup = sup;
    } else {
        // FHUT: transactions holding every item of F
        sort_tail<MW>(F, cnt, lane, S.f, S.c);
        __syncwarp();
        uint32_t acc = 0;
        for (uint64_t b = 0; b < nw.nwd; b += 128) {
            uint64_t v[4];
            nw.load(b, req, lane, v);
            for (uint32_t j = 0; j < k; ++j) {   // rarest first
                const uint32_t e = S.f[j];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (v[u]) v[u] &= nw.word(e, b + lane + 32 * u);
                if (!__any_sync(kFull, (v[0] | v[1] | v[2] | v[3]) != 0)) break;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) acc += __popcll(v[u]);
        }
        const uint32_t cf = __reduce_add_sync(kFull, acc);
        if (cf >= thr) {
            has = 1;
            csup = cf;
#pragma unroll
            for (int i = 0; i < MW; ++i) cand.w[i] |= F.w[i];
        }
    }
    if (lane < MW) {
        S.hp[lane] = m_word(Hp, lane);
        S.cand[lane] = m_word(cand, lane);
        S.req[lane] = m_word(req, lane);
    }
    if (lane == 0) {
        S.cand_sup = csup;
        S.has_cand = has;
        S.k = has ? 0 : k;
        S.pad = 0;
    }
    __syncwarp();
}

// acc[item] over the node's words for the items of T given by its bits: every
// warp of `warps` takes its share of the items.
template <int MW>
__device__ __forceinline__ void count_node(const NodeWords<MW> &nw, const Mask<MW> &T, const Mask<MW> &req,
                                           uint32_t first, uint32_t step, uint32_t *cnt, uint32_t lane) {
    for (uint64_t b = 0; b < nw.nwd || b == 0; b += 128) {
        uint64_t v[4];
        nw.load(b, req, lane, v);
        uint32_t at = 0;
#pragma unroll
        for (int ww = 0; ww < MW; ++ww)
            for (uint64_t x = T.w[ww]; x; x &= x - 1, ++at) {
                if (at % step != first) continue;
                const uint32_t e = ww * 64 + (__ffsll((long long)x) - 1);
                uint32_t acc = 0;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (v[u]) acc += __popcll(v[u] & nw.word(e, b + lane + 32 * u));
                acc = __reduce_add_sync(kFull, acc);
                if (lane == 0) cnt[e] = (b ? cnt[e] : 0u) + acc;
            }
    }
    __syncwarp();
}

}  // namespace

// Roots of split windows: a CTA of 8 warps per window, the items shared out (a
// warp per window left a batch of 45 windows on 45 warps: 0.55 ms, now 0.13).
constexpr int kRootThreads = 256;
template <int MW> __global__ void __launch_bounds__(kRootThreads) wroot_kernel(WMineParams p) {
    __shared__ uint32_t cnt[128];
    __shared__ uint32_t s_wi;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    WRoot<MW> *roots = reinterpret_cast<WRoot<MW> *>(p.roots);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_wi = atomicAdd(p.next + 1, 1u);
        __syncthreads();
        const uint32_t wi = s_wi;
        if (wi >= p.n_split) break;
        const uint32_t w = p.split_win[wi];
        const uint32_t n = p.lens[w];
        const NodeWords<MW> nw(p, p.starts[w], n);
        Mask<MW> T = m_zero<MW>();
        for (uint32_t e = 0; e < p.d; ++e) m_set(T, e);
        count_node<MW>(nw, T, m_zero<MW>(), wib, kRootThreads / 32, cnt, lane);
        __syncthreads();
        if (wib == 0)
            finish_node<MW>(p, nw, m_zero<MW>(), T, m_zero<MW>(), n, p.thrs[w] ? p.thrs[w] : 1, cnt, lane, roots[w]);
    }
}

// Children of expanded nodes that are expanded themselves: child sub_child[i] of
// record sub_parent[i] of `parents` (roots by window, or earlier records), a warp
// each, into subs[sub_out + i].  (Counted over the children's listed databases they
// took 2.0 ms in a batch of 45 windows, 0.25 ms this way.)
template <int MW> __global__ void __launch_bounds__(128) wsub_kernel(WMineParams p) {
    __shared__ uint32_t s_cnt[4][128];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t wib = threadIdx.x >> 5;
    uint32_t *cnt = s_cnt[wib];
    const WRoot<MW> *parents = reinterpret_cast<const WRoot<MW> *>(p.sub_parents);
    WRoot<MW> *subs = reinterpret_cast<WRoot<MW> *>(p.subs);
    for (;;) {
        uint32_t si = 0;
        if (lane == 0) si = atomicAdd(p.sub_next, 1u);
        si = __shfl_sync(kFull, si, 0);
        if (si >= p.n_sub) break;
        const uint32_t w = p.sub_win[si], j = p.sub_child[si];
        const WRoot<MW> &R = parents[p.sub_parent[si]];
        const uint32_t k = R.k;
        Mask<MW> T = m_zero<MW>();
        for (uint32_t q = j + 1 + lane; q < k; q += 32) m_set(T, R.f[q]);
        T = warp_or(T);
        Mask<MW> H = m_load<MW>(R.hp), req = m_load<MW>(R.req);
        m_set(H, R.f[j]);
        m_set(req, R.f[j]);
        const NodeWords<MW> nw(p, p.starts[w], p.lens[w]);
        count_node<MW>(nw, T, req, 0, 1, cnt, lane);
        finish_node<MW>(p, nw, H, T, req, R.c[j], p.thrs[w] ? p.thrs[w] : 1, cnt, lane, subs[p.sub_out + si]);
    }
}

// ------------------------------------------------------------------ tasks
template <int MW> __global__ void __launch_bounds__(128) wtask_kernel(WMineParams p) {
    __shared__ uint32_t s_cnt[4][128];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t wib = threadIdx.x >> 5;
    const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    uint32_t *cnt = s_cnt[wib];
    uint64_t *lists = p.lists + warp * (uint64_t)p.list_cap * MW;
    uint32_t *lmfi = p.lmfi + warp * (uint64_t)p.lmfi_cap;
    uint64_t *pool = p.pool_m + warp * (uint64_t)p.pool_cap * MW;
    uint32_t *pool_s = p.pool_s + warp * (uint64_t)p.pool_cap;
    WLevel<MW> *LV = reinterpret_cast<WLevel<MW> *>(p.levels) + warp * kWDepth;
    const WRoot<MW> *roots = reinterpret_cast<const WRoot<MW> *>(p.roots);
    const uint32_t d = p.d;

    for (;;) {
        uint32_t ti = 0;
        if (lane == 0) ti = atomicAdd(p.next, 1u);
        ti = __shfl_sync(kFull, ti, 0);
        if (ti >= p.n_tasks) break;
        const uint64_t t_begin = globaltimer_ns();
        const uint32_t t = p.task_order[ti];
        const uint32_t w = p.task_win[t];
        const uint32_t child = p.task_child[t];
        const uint32_t rec = p.task_rec[t];
        const uint64_t start = p.starts[w];
        const uint32_t n = p.lens[w];
        const uint32_t thr = p.thrs[w] ? p.thrs[w] : 1;
        int status = 0;
        uint32_t np = 0;
        uint64_t nodes = 0;

        // the task's first node: the whole window, or a child of an expanded node
        const bool ring0 = rec == kWholeWindow && child == kWholeWindow;
        Mask<MW> H = m_zero<MW>(), T = m_zero<MW>();
        uint32_t sup = n, list_n = n;
        bool done = false;   // an expanded node that is itself terminal: its one candidate
        if (ring0) {
            for (uint32_t e = 0; e < d; ++e) m_set(T, e);
        } else {
            const WRoot<MW> &R = rec == kWholeWindow ? roots[w] : reinterpret_cast<const WRoot<MW> *>(p.subs)[rec];
            if (child == kWholeWindow) {
                if (lane < MW) pool[lane] = R.cand[lane];
                if (lane == 0) pool_s[0] = R.cand_sup;
                np = 1;
                nodes = 1;
                done = true;
            } else {
                for (uint32_t q = child + 1 + lane; q < R.k; q += 32) m_set(T, R.f[q]);
                T = warp_or(T);
                H = m_load<MW>(R.hp);
                Mask<MW> req = m_load<MW>(R.req);
                m_set(req, R.f[child]);
                m_set(H, R.f[child]);
                sup = R.c[child];
                list_n = 0;
                if (m_nz(T)) {
                    list_n = build_child<MW>(true, p, start, lists, 0, n, req, T, 0, lane);
                    if (list_n == 0xffffffffu) status = 1;
                }
            }
        }
        int l = 0;
        uint64_t list_off = 0;
        uint32_t lm_off = 0, lm_n = 0, entry = 0;
        bool expand = true;

        while (status == 0 && !done) {
            if (expand) {
                expand = false;
                ++nodes;
                const bool ring = ring0 && l == 0;
                count_items<MW>(ring, p, start, lists, list_off, list_n, T, cnt, lane);
                Mask<MW> P, F;
                classify<MW>(T, cnt, d, thr, sup, lane, P, F);
                Mask<MW> Hp, Q;
                uint32_t k = 0;
#pragma unroll
                for (int i = 0; i < MW; ++i) {
                    Hp.w[i] = H.w[i] | P.w[i];
                    Q.w[i] = Hp.w[i] | F.w[i];
                    k += __popcll(F.w[i]);
                }
                // ---- is H u P u F inside a known MFI?  (local list; nothing was found since entry)
                bool hit = false;
                for (uint32_t b = 0; b < lm_n && !hit; b += 32 * kU) {
                    uint32_t idx[kU];
#pragma unroll
                    for (int u = 0; u < kU; ++u) {
                        const uint32_t i = b + u * 32 + lane;
                        idx[u] = i < lm_n ? lmfi[lm_off + i] : 0xffffffffu;
                    }
                    bool h = false;
#pragma unroll
                    for (int u = 0; u < kU; ++u)
                        if (idx[u] != 0xffffffffu) h |= m_sub(Q, m_load<MW>(pool + (uint64_t)idx[u] * MW));
                    hit = __any_sync(kFull, h);
                }
                if (k == 0 || hit) {
                    if (k == 0 && !hit && m_nz(Hp)) {
                        if (np >= p.pool_cap) { status = 1; break; }
                        if (lane < MW) pool[(uint64_t)np * MW + lane] = m_word(Hp, lane);
                        if (lane == 0) pool_s[np] = sup;
                        ++np;
                    }
                    if (l == 0) break;
                    --l;
                    __syncwarp();
                    continue;
                }
                // ---- FHUT: support of H u P u F
                const uint32_t cf = count_superset<MW>(ring, p, start, lists, list_off, list_n, F, lane);
                if (cf >= thr) {
                    if (np >= p.pool_cap) { status = 1; break; }
                    if (lane < MW) pool[(uint64_t)np * MW + lane] = m_word(Q, lane);
                    if (lane == 0) pool_s[np] = cf;
                    ++np;
                    if (l == 0) break;
                    --l;
                    __syncwarp();
                    continue;
                }
                // ---- record the node: frequent tail sorted by (support, id)
                WLevel<MW> &A = LV[l];
                sort_tail<MW>(F, cnt, lane, A.f, A.c);
                if (lane < MW) A.hp[lane] = m_word(Hp, lane);
                if (lane == 0) {
                    A.list_off = list_off;
                    A.list_n = list_n;
                    A.lm_off = lm_off;
                    A.lm_n = lm_n;
                    A.entry = entry;
                    A.k = k;
                    A.j = 0;
                }
                __syncwarp();
            }
            // ---- next child of level l, or up
            WLevel<MW> &A = LV[l];
            const uint32_t j = A.j, k = A.k;
            if (j >= k) {
                if (l == 0) break;
                --l;
                continue;
            }
            __syncwarp();
            if (lane == 0) A.j = j + 1;
            const uint32_t e = A.f[j];
            const uint32_t csup = A.c[j];
            Mask<MW> Tc = m_zero<MW>();
            for (uint32_t q = j + 1 + lane; q < k; q += 32) m_set(Tc, A.f[q]);
            Tc = warp_or(Tc);
            Mask<MW> Hc = m_load<MW>(A.hp);
            m_set(Hc, e);
            const bool pring = ring0 && l == 0;
            const uint64_t p_off = A.list_off;
            const uint32_t p_n = A.list_n;
            const uint64_t c_off = pring ? 0 : p_off + p_n;
            uint32_t cn = 0;
            if (m_nz(Tc)) {
                Mask<MW> req = m_zero<MW>();
                m_set(req, e);
                cn = build_child<MW>(pring, p, start, lists, p_off, p_n, req, Tc, c_off, lane);
                if (cn == 0xffffffffu) { status = 1; break; }
            }
            // child local-MFI list: members containing the child's head
            const uint32_t c_lm = A.lm_off + A.lm_n;
            const uint32_t p_lm_off = A.lm_off, p_lm_n = A.lm_n, p_entry = A.entry;
            const uint32_t n_src = p_lm_n + (np - p_entry);
            uint32_t ln = 0;
            for (uint32_t b = 0; b < n_src; b += 32 * kU) {
                uint32_t idx[kU];
                bool keep[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const uint32_t i = b + u * 32 + lane;
                    idx[u] = 0;
                    keep[u] = false;
                    if (i < n_src) idx[u] = i < p_lm_n ? lmfi[p_lm_off + i] : p_entry + (i - p_lm_n);
                }
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if (b + u * 32 + lane < n_src) keep[u] = m_sub(Hc, m_load<MW>(pool + (uint64_t)idx[u] * MW));
                // the child's list goes after the parent's: writes never touch indices still to be read
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const uint32_t bal = __ballot_sync(kFull, keep[u]);
                    const uint64_t pos = (uint64_t)c_lm + ln + __popc(bal & ((1u << lane) - 1));
                    if (keep[u] && pos < p.lmfi_cap) lmfi[pos] = idx[u];
                    ln += __popc(bal);
                }
            }
            if ((uint64_t)c_lm + ln > p.lmfi_cap) { status = 1; break; }
            if (l + 1 >= kWDepth) { status = 1; break; }
            __syncwarp();
            ++l;
            H = Hc;
            T = Tc;
            sup = csup;
            list_off = c_off;
            list_n = cn;
            lm_off = c_lm;
            lm_n = ln;
            entry = np;
            expand = true;
        }

        // ---- publish the task's candidates
        uint64_t off = 0;
        if (status == 0) {
            if (lane == 0) off = atomicAdd(p.out_pos, (unsigned long long)np);
            off = __shfl_sync(kFull, off, 0);
            if (off + np > p.out_cap) {
                status = 2;
            } else {
                __syncwarp();
                for (uint32_t i = lane; i < np * MW; i += 32) p.out_m[off * MW + i] = pool[i];
                for (uint32_t i = lane; i < np; i += 32) p.out_s[off + i] = pool_s[i];
            }
        }
        if (lane == 0) {
            p.task_off[t] = off;
            p.task_cnt[t] = status == 0 ? np : 0;
            p.task_status[t] = status;
            p.task_nodes[t] = nodes;
            if (p.task_ns) p.task_ns[t] = globaltimer_ns() - t_begin;
        }
        __syncwarp();
    }
}

namespace {

// Base database of a task: the window's transactions holding every item of req,
// found through the ring's vertical rows; their places, counted from the
// transaction the window's first word starts with, at at[0 ..), in no particular
// order.  Returns how many (at[] has room for the window's length).
template <int MW>
__device__ __forceinline__ uint32_t list_base(const NodeWords<MW> &nw, const Mask<MW> &req, uint32_t *at,
                                              uint32_t lane) {
    uint32_t cn = 0;
#pragma unroll 1
    for (uint64_t b = 0; b < nw.nwd; b += 128) {
        uint64_t v[4];
        nw.load(b, req, lane, v);
        uint32_t mine = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) mine += __popcll(v[u]);
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(kFull, incl, o);
            if (lane >= (uint32_t)o) incl += x;
        }
        uint32_t to = cn + incl - mine;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t at0 = (uint32_t)(b + lane + 32 * u) * 64;
#pragma unroll 1
            for (uint64_t x = v[u]; x; x &= x - 1) at[to++] = at0 + (__ffsll((long long)x) - 1);
        }
        cn += __shfl_sync(kFull, incl, 31);
    }
    __syncwarp();
    return cn;
}

// Vertical rows of a database of n0 transactions, by item id: bit i of word c of
// row e is set when entry 32c+i holds item e (rows of T0's items; vw a multiple of
// 4).  Four chunks of 32 entries at a time, so a row's words leave as one 16-byte
// store; the next four chunks' masks are on their way meanwhile.  (Each lane
// fetching the masks of its own words one by one, twice, took 90 to 330 us a task
// in a batch, most of the time of the tasks that search a handful of nodes; now 30 to 100 us.)
template <int MW>
__device__ __forceinline__ void build_rows(const WMineParams &p, const NodeWords<MW> &nw, const uint32_t *at,
                                           uint32_t n0, const Mask<MW> &T0, uint32_t *rows, uint32_t vw,
                                           uint32_t lane) {
    const uint32_t W = (n0 + 31) / 32;
    Mask<MW> next[4];
    auto fetch = [&](uint32_t c) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t i = (c + u) * 32 + lane;
            next[u] = i < n0 ? m_load<MW>(p.hm + (((nw.w0 << 6) + at[i]) & p.cap_mask) * MW) : m_zero<MW>();
        }
    };
    fetch(0);
#pragma unroll 1
    for (uint32_t c = 0; c < W; c += 4) {
        Mask<MW> m[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) m[u] = next[u];
        if (c + 4 < W) fetch(c + 4);
#pragma unroll
        for (int b = 0; b < 2 * MW; ++b) {
            const uint32_t want = (uint32_t)(T0.w[b >> 1] >> ((b & 1) * 32));
            if (!want) continue;
            uint32_t w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) w[u] = transpose32((uint32_t)(m[u].w[b >> 1] >> ((b & 1) * 32)), lane);
            if ((want >> lane) & 1u)
                *reinterpret_cast<uint4 *>(rows + (uint64_t)(b * 32 + lane) * vw + c) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    __syncwarp();
}

}  // namespace

// Resident CTAs per SM the register allocation is fitted to.  Measured with tails as masks on the
// 4,096 service windows: 6 (80 registers, 3,648 warps) 337 ms, 7 (72 registers,
// 4,176 warps, the workspace budget's limit) 338 ms with a longer makespan, 8
// (64 registers, spills) 358 ms -- more resident warps do not shorten the search.
#ifndef SGFIM_WVTASK_MIN_BLOCKS
#define SGFIM_WVTASK_MIN_BLOCKS 6
#endif

// A node's tail is a list in shared memory, ascending (support, id) in its parent.
// Counting runs with a lane per tidset word, four items at a time; the frequent
// items are packed, sorted by (support, id) (an item's place is the number of
// smaller keys) and become the node's record and its children's tails.  FHUT ANDs
// the rows rarest first and stops as soon as fewer than thr transactions are left.
// Bound by instruction issue and by fetching them (tidsets of 16 to 2,048 words:
// each item's count is a few loads and a reduction).  Item by item with 64-bit
// masks the node cost 2,000 instructions, now 1,060, and the code is 68 KB instead
// of 84.  45 windows of 512 to 65,536 transactions (floor 2%): 8.8 -> 6.5 ms;
// 768 windows: 69 -> 44 ms.  A child whose head and tail lie in a known MFI ends its
// parent's loop (2.15 -> 1.50 million nodes for 0.99 million MFIs; 37.1 -> 25.6
// million for 17.1), and a task may search several children of an expanded node:
// 6.5 -> 5.8 ms (the longest task; 2.4 ms a warp on average), 44 -> 36 ms.
template <int MW> __global__ void __launch_bounds__(128, SGFIM_WVTASK_MIN_BLOCKS) wvtask_kernel(WMineParams p) {
    constexpr uint32_t NI = 64 * MW;                        // items
    __shared__ __align__(16) uint32_t s_cnt[4][NI];
    __shared__ uint64_t s_key[4][NI];                       // (support, id) of the frequent items
    __shared__ uint8_t s_tail[4][NI], s_sort[4][NI];        // a node's tail; its frequent part, sorted
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t wib = threadIdx.x >> 5;
    const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    uint8_t *tail = s_tail[wib], *sorted = s_sort[wib];
    uint32_t *cnt = s_cnt[wib];
    uint64_t *keys = s_key[wib];
    uint32_t *at = reinterpret_cast<uint32_t *>(p.lists) + warp * (uint64_t)p.list_cap;
    uint32_t *lmfi = p.lmfi + warp * (uint64_t)p.lmfi_cap;
    uint64_t *pool = p.pool_m + warp * (uint64_t)p.pool_cap * MW;
    uint32_t *pool_s = p.pool_s + warp * (uint64_t)p.pool_cap;
    WLevel<MW> *LV = reinterpret_cast<WLevel<MW> *>(p.levels) + warp * kWDepth;
    const WRoot<MW> *roots = reinterpret_cast<const WRoot<MW> *>(p.roots);
    const uint32_t d = p.d;
    const uint32_t vw = p.v_words;
    uint32_t *vrows = p.vbuf + warp * (uint64_t)(128 + kWDepth) * vw;   // item e: vrows + e * vw
    uint32_t *vtid = vrows + (uint64_t)128 * vw;                        // level l: vtid + l * vw

    for (;;) {
        uint32_t ti = 0;
        if (lane == 0) ti = atomicAdd(p.next, 1u);
        ti = __shfl_sync(kFull, ti, 0);
        if (ti >= p.n_tasks) break;
        const uint64_t t_begin = globaltimer_ns();
        const uint32_t t = p.task_order[ti];
        const uint32_t w = p.task_win[t];
        const uint32_t child = p.task_child[t];
        const uint32_t rec = p.task_rec[t];
        const uint32_t n_child = p.task_n_child[t];
        const uint64_t start = p.starts[w];
        const uint32_t n = p.lens[w];
        const uint32_t thr = p.thrs[w] ? p.thrs[w] : 1;
        int status = 0;
        uint32_t np = 0;
        uint64_t nodes = 0;

        // the task's first node: the whole window, a child of an expanded node, or (n_child > 1)
        // an expanded node of whose children this task searches n_child
        const bool part = n_child > 1;
        Mask<MW> H = m_zero<MW>(), T0 = m_zero<MW>(), req = m_zero<MW>();
        uint32_t sup = n, list_n = n, nt = 0;
        bool done = false;               // an expanded node that is itself terminal: its one candidate
        const uint8_t *src = nullptr;    // where the first tail is listed (null: all items)
        if (rec == kWholeWindow && child == kWholeWindow) {
            nt = d;
        } else {
            const WRoot<MW> &R = rec == kWholeWindow ? roots[w] : reinterpret_cast<const WRoot<MW> *>(p.subs)[rec];
            if (child == kWholeWindow) {
                if (lane < MW) pool[lane] = R.cand[lane];
                if (lane == 0) pool_s[0] = R.cand_sup;
                np = 1;
                nodes = 1;
                done = true;
            } else {
                H = m_load<MW>(R.hp);
                req = m_load<MW>(R.req);
                src = R.f + child;
                nt = R.k - child;
                if (part) {   // the node is in the record: level 0, children from `child` on
                    WLevel<MW> &A = LV[0];
                    if (lane < MW) A.hp[lane] = R.hp[lane];
                    for (uint32_t i = lane; i < nt; i += 32) {
                        A.f[i] = src[i];
                        A.c[i] = R.c[child + i];
                    }
                    if (lane == 0) {
                        A.lm_off = A.lm_n = A.entry = 0;
                        A.k = nt;
                        A.end = n_child;
                        A.j = 0;
                    }
                } else {
                    m_set(req, R.f[child]);
                    m_set(H, R.f[child]);
                    sup = R.c[child];
                    ++src;
                    --nt;
                }
            }
        }
#pragma unroll 1
        for (uint32_t i = lane; i < nt; i += 32) {
            const uint32_t e = src ? src[i] : i;
            tail[i] = (uint8_t)e;
            m_set(T0, e);
        }
        T0 = warp_or(T0);
        const NodeWords<MW> nw(p, start, n);
        if (!done) {
            list_n = 0;
            if (nt) {
                if (n > p.list_cap) status = 1;
                else list_n = list_base<MW>(nw, req, at, lane);
            }
        }
        // ---- the task's database as vertical rows over its entries
        const uint32_t W = (list_n + 31) / 32;
        const bool small = W <= 32 * kReg, two = list_n < 65536;
        const uint32_t nk = (W + 31) / 32;   // words per lane
        uint32_t tr[kReg] = {0, 0, 0, 0};   // the node's tidset, when small
        if (status == 0 && !done) {
            if (((W + 3) & ~3u) > vw) {
                status = 1;
            } else {
                build_rows<MW>(p, nw, at, list_n, T0, vrows, vw, lane);
#pragma unroll 1
                for (uint32_t x = lane; x < W; x += 32) {
                    const uint32_t v = (x + 1 < W || (list_n & 31) == 0) ? 0xffffffffu : ((1u << (list_n & 31)) - 1);
                    vtid[x] = v;
#pragma unroll
                    for (uint32_t k = 0; k < kReg; ++k)
                        if (x == lane + 32 * k) tr[k] = v;
                }
                __syncwarp();
            }
        }
        int l = 0;
        uint32_t lm_off = 0, lm_n = 0, entry = 0;
        bool expand = !part;

        while (status == 0 && !done) {
            if (expand) {
                expand = false;
                ++nodes;
                const uint32_t *tid = vtid + (uint64_t)l * vw;
                // ---- supports of the tail's items
                if (nk <= 1) count_tail<1>(vrows, vw, W, tr, tid, tail, nt, two, cnt, lane);
                else if (nk <= 2) count_tail<2>(vrows, vw, W, tr, tid, tail, nt, two, cnt, lane);
                else if (small) count_tail<4>(vrows, vw, W, tr, tid, tail, nt, two, cnt, lane);
                else count_tail<0>(vrows, vw, W, tr, tid, tail, nt, two, cnt, lane);
                __syncwarp();
                // ---- PEP items P (they join H) and the frequent tail F
                Mask<MW> Pl = m_zero<MW>(), Fl = m_zero<MW>();
                uint32_t k = 0, any_p = 0;
#pragma unroll 1
                for (uint32_t b = 0; b < nt; b += 32) {
                    const bool in = b + lane < nt;
                    const uint32_t e = in ? tail[b + lane] : 0, c = in ? cnt[b + lane] : 0;
                    const bool isp = in && c >= thr && c == sup, isf = in && c >= thr && c < sup;
                    const uint32_t bal = __ballot_sync(kFull, isf);
                    any_p |= __ballot_sync(kFull, isp);
                    if (isp) m_set(Pl, e);
                    if (isf) {
                        m_set(Fl, e);
                        keys[k + __popc(bal & ((1u << lane) - 1))] = (uint64_t)c << 8 | e;
                    }
                    k += __popc(bal);
                }
                Mask<MW> Hp = H, Q;
                if (any_p) {
                    Pl = warp_or(Pl);
#pragma unroll
                    for (int i = 0; i < MW; ++i) Hp.w[i] |= Pl.w[i];
                }
                Q = Hp;
                if (k) {
                    Fl = warp_or(Fl);
#pragma unroll
                    for (int i = 0; i < MW; ++i) Q.w[i] |= Fl.w[i];
                }
                __syncwarp();
                // ---- is H u P u F inside a known MFI?  (local list; nothing was found since entry)
                bool hit = false;
#pragma unroll 1
                for (uint32_t b = 0; b < lm_n && !hit; b += 32 * kU) {
                    uint32_t idx[kU];
#pragma unroll
                    for (int u = 0; u < kU; ++u) {
                        const uint32_t i = b + u * 32 + lane;
                        idx[u] = i < lm_n ? lmfi[lm_off + i] : 0xffffffffu;
                    }
                    bool h = false;
#pragma unroll
                    for (int u = 0; u < kU; ++u)
                        if (idx[u] != 0xffffffffu) h |= m_sub(Q, m_load<MW>(pool + (uint64_t)idx[u] * MW));
                    hit = __any_sync(kFull, h);
                }
                if (k == 0 || hit) {
                    if (k == 0 && !hit && m_nz(Hp)) {
                        if (np >= p.pool_cap) { status = 1; break; }
                        if (lane < MW) pool[(uint64_t)np * MW + lane] = m_word(Hp, lane);
                        if (lane == 0) pool_s[np] = sup;
                        ++np;
                    }
                    if (l == 0) break;
                    --l;
                    __syncwarp();
                    continue;
                }
                // ---- F by (support, id): an item's place is the number of smaller keys
                WLevel<MW> &A = LV[l];
#pragma unroll 1
                for (uint32_t b = 0; b < k; b += 32) {
                    const uint64_t mine = b + lane < k ? keys[b + lane] : ~0ull;
                    uint32_t rank = 0;
#pragma unroll 2
                    for (uint32_t i = 0; i < k; ++i) rank += keys[i] < mine;
                    if (b + lane < k) {
                        sorted[rank] = (uint8_t)mine;
                        A.f[rank] = (uint8_t)mine;
                        A.c[rank] = (uint32_t)(mine >> 8);
                    }
                }
                __syncwarp();
                // ---- FHUT: support of H u P u F
                uint32_t cf = 0;
                if (nk <= 1) {
                    cf = count_all<1>(vrows, vw, W, tr, sorted, k, thr, lane);
                } else if (nk <= 2) {
                    cf = count_all<2>(vrows, vw, W, tr, sorted, k, thr, lane);
                } else if (small) {
                    cf = count_all<4>(vrows, vw, W, tr, sorted, k, thr, lane);
                } else {
#pragma unroll 1
                    for (uint32_t x = lane; x < W; x += 32) {
                        uint32_t v = tid[x];
#pragma unroll 1
                        for (uint32_t i = 0; i < k && v; ++i) v &= vrows[sorted[i] * vw + x];
                        cf += __popc(v);
                    }
                    cf = __reduce_add_sync(kFull, cf);
                }
                if (cf >= thr) {
                    if (np >= p.pool_cap) { status = 1; break; }
                    if (lane < MW) pool[(uint64_t)np * MW + lane] = m_word(Q, lane);
                    if (lane == 0) pool_s[np] = cf;
                    ++np;
                    if (l == 0) break;
                    --l;
                    __syncwarp();
                    continue;
                }
                // ---- record the node
                if (lane < MW) A.hp[lane] = m_word(Hp, lane);
                if (lane == 0) {
                    A.lm_off = lm_off;
                    A.lm_n = lm_n;
                    A.entry = entry;
                    A.k = A.end = k;
                    A.j = 0;
                }
                __syncwarp();
            }
            // ---- next child of level l, or up
            WLevel<MW> &A = LV[l];
            const uint32_t j = A.j, k = A.k;
            if (j >= A.end) {
                if (l == 0) break;
                --l;
                continue;
            }
            __syncwarp();
            if (lane == 0) A.j = j + 1;
            const uint32_t e = A.f[j];
            const uint32_t csup = A.c[j];
            Mask<MW> Hc = m_load<MW>(A.hp);
            m_set(Hc, e);
            nt = k - j - 1;
            Mask<MW> all = m_zero<MW>();   // the child's head and its whole tail
#pragma unroll 1
            for (uint32_t i = lane; i < nt; i += 32) {
                const uint32_t f = A.f[j + 1 + i];
                tail[i] = (uint8_t)f;
                m_set(all, f);
            }
            if (nt) all = warp_or(all);
#pragma unroll
            for (int i = 0; i < MW; ++i) all.w[i] |= Hc.w[i];
            // child local-MFI list: members containing the child's head.  One that contains its
            // tail too leaves nothing new below this child, nor below any later one: their heads
            // and tails are subsets of this one's.
            bool known = false;
            const uint32_t c_lm = A.lm_off + A.lm_n;
            const uint32_t p_lm_off = A.lm_off, p_lm_n = A.lm_n, p_entry = A.entry;
            const uint32_t n_src = p_lm_n + (np - p_entry);
            uint32_t ln = 0;
#pragma unroll 1
            for (uint32_t b = 0; b < n_src; b += 32 * kU) {
                uint32_t idx[kU];
                bool keep[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const uint32_t i = b + u * 32 + lane;
                    idx[u] = 0;
                    keep[u] = false;
                    if (i < n_src) idx[u] = i < p_lm_n ? lmfi[p_lm_off + i] : p_entry + (i - p_lm_n);
                }
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if (b + u * 32 + lane < n_src) {
                        const Mask<MW> m = m_load<MW>(pool + (uint64_t)idx[u] * MW);
                        keep[u] = m_sub(Hc, m);
                        known |= m_sub(all, m);
                    }
                // the child's list goes after the parent's: writes never touch indices still to be read
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const uint32_t bal = __ballot_sync(kFull, keep[u]);
                    const uint64_t pos = (uint64_t)c_lm + ln + __popc(bal & ((1u << lane) - 1));
                    if (keep[u] && pos < p.lmfi_cap) lmfi[pos] = idx[u];
                    ln += __popc(bal);
                }
            }
            if (__any_sync(kFull, known)) {
                if (l == 0) break;
                --l;
                __syncwarp();
                continue;
            }
            if (nt == 0) {   // the last child, alone: a candidate
                ++nodes;
                if (np >= p.pool_cap) { status = 1; break; }
                if (lane < MW) pool[(uint64_t)np * MW + lane] = m_word(Hc, lane);
                if (lane == 0) pool_s[np] = csup;
                ++np;
                __syncwarp();
                continue;
            }
            if ((uint64_t)c_lm + ln > p.lmfi_cap) { status = 1; break; }
            if (l + 1 >= kWDepth) { status = 1; break; }
            {
                // child tidset = parent tidset AND row(e)
                const uint32_t *ptid = vtid + (uint64_t)l * vw;
                uint32_t *ctid = vtid + (uint64_t)(l + 1) * vw;
                const uint32_t *row = vrows + e * vw;
                if (small) {
#pragma unroll
                    for (uint32_t x = 0; x < kReg; ++x)
                        if (lane + 32 * x < W) {
                            tr[x] = ptid[lane + 32 * x] & row[lane + 32 * x];
                            ctid[lane + 32 * x] = tr[x];
                        }
                } else {
#pragma unroll 1
                    for (uint32_t x = lane; x < W; x += 32) ctid[x] = ptid[x] & row[x];
                }
            }
            __syncwarp();
            ++l;
            H = Hc;
            sup = csup;
            lm_off = c_lm;
            lm_n = ln;
            entry = np;
            expand = true;
        }

        // ---- publish the task's candidates
        uint64_t off = 0;
        if (status == 0) {
            if (lane == 0) off = atomicAdd(p.out_pos, (unsigned long long)np);
            off = __shfl_sync(kFull, off, 0);
            if (off + np > p.out_cap) {
                status = 2;
            } else {
                __syncwarp();
#pragma unroll 1
                for (uint32_t i = lane; i < np * MW; i += 32) p.out_m[off * MW + i] = pool[i];
#pragma unroll 1
                for (uint32_t i = lane; i < np; i += 32) p.out_s[off + i] = pool_s[i];
            }
        }
        if (lane == 0) {
            p.task_off[t] = off;
            p.task_cnt[t] = status == 0 ? np : 0;
            p.task_status[t] = status;
            p.task_nodes[t] = nodes;
            if (p.task_ns) p.task_ns[t] = globaltimer_ns() - t_begin;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ cross-task filter
// The window's candidates in task order (subtrees in depth-first order) get a
// vertical bitmap rows[e][q] (wfilter_mark); candidate q of a task is dropped when
// the AND of its items' rows has a bit below the task's first candidate
// (wfilter_check).  keep[] is written per arena slot, kept[] per task.  Both take
// 256 candidates of one window at a time, so a large window is spread over the
// chip (a CTA per window: 45 windows on 45 SMs: 1.96 ms, now 0.41).
namespace {

constexpr int kFilterThreads = 256;

// The unit's window (binary search over the units' prefix) and its first candidate.
__device__ __forceinline__ uint32_t filter_window(const WFilterParams &p, uint32_t unit) {
    uint32_t lo = 0, hi = p.n_win - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (p.win_unit0[mid] <= unit) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// candidate q of a window (task order) -> its entry of the task lists
__device__ __forceinline__ uint32_t filter_entry(const WFilterParams &p, uint32_t wi, uint64_t q) {
    uint32_t lo = p.win_task0[wi], hi = p.win_task0[wi + 1] - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (p.task_first[mid] <= q) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

}  // namespace

// A warp turns 32 candidates' masks into a 32-bit word of every item's row, and
// counts the items' candidates and their first and last words.
template <int MW> __global__ void __launch_bounds__(kFilterThreads) wfilter_mark_kernel(WFilterParams p) {
    __shared__ uint32_t s_wi;
    __shared__ uint32_t s_freq[64 * MW], s_lo[64 * MW], s_hi[64 * MW];
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t unit = blockIdx.x; unit < p.n_units; unit += gridDim.x) {
        __syncthreads();
        if (threadIdx.x == 0) s_wi = filter_window(p, unit);
        for (uint32_t i = threadIdx.x; i < 64 * MW; i += kFilterThreads) {
            s_freq[i] = 0;
            s_lo[i] = 0xffffffffu;
            s_hi[i] = 0;
        }
        __syncthreads();
        const uint32_t wi = s_wi;
        const uint64_t M = p.win_total[wi];
        const uint64_t W = (M + 63) / 64;
        uint32_t *rows = reinterpret_cast<uint32_t *>(p.scratch + p.win_row0[wi]);
        const uint64_t q = (uint64_t)(unit - p.win_unit0[wi]) * kFilterThreads + threadIdx.x;
        Mask<MW> m = m_zero<MW>();
        if (q < M) {
            const uint32_t en = filter_entry(p, wi, q);
            m = m_load<MW>(p.out_m + (p.task_off[p.task_of[en]] + (q - p.task_first[en])) * MW);
        }
        const uint64_t wd = q >> 5;   // the warp's word
#pragma unroll
        for (int b = 0; b < 2 * MW; ++b) {
            const uint32_t v = transpose32((uint32_t)(m.w[b >> 1] >> ((b & 1) * 32)), lane);
            const uint32_t e = b * 32 + lane;
            if (e < p.d && wd < 2 * W) {
                rows[(uint64_t)e * (2 * W) + wd] = v;
                if (v) {
                    atomicAdd(&s_freq[e], __popc(v));
                    atomicMin(&s_lo[e], (uint32_t)(wd >> 1));
                    atomicMax(&s_hi[e], (uint32_t)(wd >> 1));
                }
            }
        }
        __syncthreads();
        uint32_t *st = p.win_stats + (uint64_t)wi * 3 * 64 * MW;
        for (uint32_t i = threadIdx.x; i < 64 * MW; i += kFilterThreads)
            if (s_freq[i]) {
                atomicAdd(st + i, s_freq[i]);
                atomicMax(st + 64 * MW + i, ~s_lo[i]);   // complemented: the table starts as zeros
                atomicMax(st + 2 * 64 * MW + i, s_hi[i]);
            }
    }
}

template <int MW> __global__ void __launch_bounds__(kFilterThreads) wfilter_check_kernel(WFilterParams p) {
    __shared__ uint32_t s_wi;
    __shared__ uint32_t s_freq[64 * MW];               // candidates holding each item
    __shared__ uint32_t s_lo[64 * MW], s_hi[64 * MW];  // first / last word of each item's row with a bit
    for (uint32_t unit = blockIdx.x; unit < p.n_units; unit += gridDim.x) {
        __syncthreads();
        if (threadIdx.x == 0) s_wi = filter_window(p, unit);
        __syncthreads();
        const uint32_t wi = s_wi;
        const uint32_t *st = p.win_stats + (uint64_t)wi * 3 * 64 * MW;
        for (uint32_t i = threadIdx.x; i < 64 * MW; i += kFilterThreads) {
            s_freq[i] = st[i];
            s_lo[i] = ~st[64 * MW + i];
            s_hi[i] = st[2 * 64 * MW + i];
        }
        __syncthreads();
        const uint64_t M = p.win_total[wi];
        const uint64_t W = (M + 63) / 64;
        const uint64_t *rows = p.scratch + p.win_row0[wi];
        const uint64_t q = (uint64_t)(unit - p.win_unit0[wi]) * kFilterThreads + threadIdx.x;
        if (q >= M) continue;
        const uint32_t en = filter_entry(p, wi, q);
        const uint32_t t = p.task_of[en];
        const uint64_t slot = p.task_off[t] + (q - p.task_first[en]);
        bool keep = true;
        const uint64_t lim = p.task_first[en];   // candidates of earlier subtrees: [0, lim)
        if (lim) {
            const Mask<MW> m = m_load<MW>(p.out_m + slot * MW);
            // the candidate's three rarest items drive the scan: their rows have the fewest bits,
            // and few words are left for the others (1.0 million candidates: 0.77 ms from the rarest
            // alone, 0.38 from three)
            uint32_t e1 = 0, e2 = 0, e3 = 0, b1 = 0xffffffffu, b2 = 0xffffffffu, b3 = 0xffffffffu;
#pragma unroll
            for (int ww = 0; ww < MW; ++ww) {
                uint64_t x = m.w[ww];
                while (x) {
                    const uint32_t e = ww * 64 + (__ffsll((long long)x) - 1), f = s_freq[e];
                    x &= x - 1;
                    if (f < b1) {
                        b3 = b2; e3 = e2;
                        b2 = b1; e2 = e1;
                        b1 = f; e1 = e;
                    } else if (f < b2) {
                        b3 = b2; e3 = e2;
                        b2 = f; e2 = e;
                    } else if (f < b3) {
                        b3 = f; e3 = e;
                    }
                }
            }
            if (b2 == 0xffffffffu) e2 = e1;   // fewer than three items
            if (b3 == 0xffffffffu) e3 = e1;
            const uint64_t wd_end = (lim + 63) / 64;
            const uint64_t hi = min(min((uint64_t)s_hi[e1], (uint64_t)min(s_hi[e2], s_hi[e3])) + 1, wd_end);
            const uint64_t lo = max(s_lo[e1], max(s_lo[e2], s_lo[e3]));
            const uint64_t *r1 = rows + (uint64_t)e1 * W, *r2 = rows + (uint64_t)e2 * W, *r3 = rows + (uint64_t)e3 * W;
            for (uint64_t wd = lo; wd < hi && keep; wd += 2) {
                uint64_t v[2];
                v[0] = r1[wd] & r2[wd] & r3[wd];
                v[1] = wd + 1 < hi ? r1[wd + 1] & r2[wd + 1] & r3[wd + 1] : 0;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (!v[u]) continue;
                    const uint64_t at = wd + u;
                    if (at * 64 + 64 > lim) v[u] &= (1ull << (lim - at * 64)) - 1;
#pragma unroll
                    for (int ww = 0; ww < MW; ++ww) {
                        uint64_t x = m.w[ww];
                        while (x && v[u]) {
                            const uint32_t e = ww * 64 + (__ffsll((long long)x) - 1);
                            x &= x - 1;
                            v[u] &= rows[(uint64_t)e * W + at];
                        }
                    }
                    keep &= v[u] == 0;
                }
            }
        }
        if (!keep) {
            p.keep[slot] = 0;
            atomicSub(&p.task_kept[t], 1u);
        }
    }
}

// ------------------------------------------------------------------ gather
// One warp per task: its kept candidates, in emission order, to dst.
template <int MW> __global__ void __launch_bounds__(128) wgather_kernel(WGatherParams p) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t t = warp; t < p.n_tasks; t += n_warps) {
        const uint64_t src = p.task_off[t];
        const uint32_t n = p.task_cnt[t];
        uint64_t dst = p.task_dst[t];
        if (dst == ~0ull) continue;
        for (uint32_t b = 0; b < n; b += 32) {
            const uint32_t i = b + lane;
            const bool keep = i < n && (!p.keep || p.keep[src + i]);
            const uint32_t bal = __ballot_sync(kFull, keep);
            if (keep) {
                const uint64_t pos = dst + __popc(bal & ((1u << lane) - 1));
                m_store<MW>(p.dst_m + pos * MW, m_load<MW>(p.out_m + (src + i) * MW));
                p.dst_s[pos] = p.out_s[src + i];
            }
            dst += __popc(bal);
        }
    }
}

int wmine_depth() { return kWDepth; }

int wtask_blocks_per_sm(bool vertical) {
    int blocks = 0;
    if (vertical) SG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, wvtask_kernel<2>, 128, 0));
    else SG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, wtask_kernel<2>, 128, 0));
    return blocks > 0 ? blocks : 1;
}
size_t wmine_level_bytes(int mw) { return mw == 2 ? sizeof(WLevel<2>) * kWDepth : 0; }
size_t wmine_root_bytes(int mw) { return mw == 2 ? sizeof(WRoot<2>) : 0; }

void launch_wroot(const WMineParams &p, int mw, unsigned blocks, cudaStream_t st) {
    if (mw != 2) throw CudaError(cudaErrorInvalidValue, "batched window miner supports 2 mask words", __FILE__, __LINE__);
    wroot_kernel<2><<<blocks, kRootThreads, 0, st>>>(p);
    SG_CUDA_TRY(cudaGetLastError());
}
void launch_wsub(const WMineParams &p, int mw, unsigned blocks, cudaStream_t st) {
    if (mw != 2) throw CudaError(cudaErrorInvalidValue, "batched window miner supports 2 mask words", __FILE__, __LINE__);
    wsub_kernel<2><<<blocks, 128, 0, st>>>(p);
    SG_CUDA_TRY(cudaGetLastError());
}
void launch_wtask(const WMineParams &p, int mw, unsigned blocks, cudaStream_t st) {
    if (mw != 2) throw CudaError(cudaErrorInvalidValue, "batched window miner supports 2 mask words", __FILE__, __LINE__);
    if (p.vbuf)
        wvtask_kernel<2><<<blocks, 128, 0, st>>>(p);
    else
        wtask_kernel<2><<<blocks, 128, 0, st>>>(p);
    SG_CUDA_TRY(cudaGetLastError());
}
int wfilter_unit() { return kFilterThreads; }

void launch_wfilter(const WFilterParams &p, int mw, unsigned blocks, cudaStream_t st) {
    if (mw != 2) throw CudaError(cudaErrorInvalidValue, "batched window miner supports 2 mask words", __FILE__, __LINE__);
    wfilter_mark_kernel<2><<<blocks, kFilterThreads, 0, st>>>(p);
    wfilter_check_kernel<2><<<blocks, kFilterThreads, 0, st>>>(p);
    SG_CUDA_TRY(cudaGetLastError());
}
void launch_wgather(const WGatherParams &p, int mw, unsigned blocks, cudaStream_t st) {
    if (mw != 2) throw CudaError(cudaErrorInvalidValue, "batched window miner supports 2 mask words", __FILE__, __LINE__);
    wgather_kernel<2><<<blocks, 128, 0, st>>>(p);
    SG_CUDA_TRY(cudaGetLastError());
}

}  // namespace sg
