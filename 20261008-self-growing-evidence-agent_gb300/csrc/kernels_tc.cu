// kernels_tc.cu -- co-occurrence on the 5th-generation tensor cores (tcgen05).
//
// C[i][j] = popc(bv_i & bv_j) is the dot product of two 0/1 vectors.  Bits
// are expanded to fp8 e4m3 bytes (1.0 = 0x38, 0.0 = 0x00; both exact) inside
// the kernel and multiplied with tcgen05.mma .kind::f8f6f4, accumulating in
// fp32 in tensor memory: every partial sum is an integer below 2^24 (a CTA
// covers at most 2^20 transactions per split), so fp32 holds it exactly.
// The reference does this product with b1 AND-POPC wmma fragments
// (code/engine_tensorfim/code/microbench/bmma_bench.cu:99-152); GB300 has no
// b1 tcgen05 kind and its int8 tensor rate is cut, hence e4m3.
//
// Tiling: a CTA owns one upper-triangle 128 x 128 tile (rows bi, columns bj)
// and a slice of the transactions.  Per stage, 256 threads expand a 256-bit
// slice of 128 + 128 rows into two 128B-swizzled K-major atoms per operand
// (row r, byte b at r*128 + ((b/16) ^ (r%8))*16 + b%16), fence the async
// proxy, and one thread issues 8 MMAs of K=32; tcgen05.commit arrives on the
// stage's mbarrier when the tensor core is done reading it.  The epilogue
// reads the 128 x 128 fp32 accumulator from TMEM (tcgen05.ld 32x32b) and
// adds the integer counts into C (and its mirror) with atomics.
#include <algorithm>

#include "common.cuh"
#include "cooc_plan.h"
#include "kernels.h"
#include "tcgen05.cuh"

namespace sg {

namespace {

constexpr int kTcThreads = 256;
constexpr int kTcStages = 2;
constexpr int kTcAtom = 128 * 128;             // one 128-row x 128-byte swizzle atom
constexpr int kTcOperand = 2 * kTcAtom;        // two atoms along K per operand
constexpr int kTcStageBytes = 2 * kTcOperand;  // A and B
constexpr uint32_t kTcCols = 128;              // TMEM columns (fp32 accumulators)

// Instruction descriptor, kind::f8f6f4: D = f32 (bits 4-5 = 1), A = B = e4m3
// (bits 7-9, 10-12 = 0), both K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
constexpr uint32_t kTcIdesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(kTcIdesc), "r"(acc)
        : "memory");
}

// 4 bits -> 4 bytes of e4m3 (0x38 = 1.0 where the bit is set).
__device__ __forceinline__ uint32_t nib4(uint32_t n) { return ((n * 0x00204081u) & 0x01010101u) * 0x38u; }

// Expand 128 bits (two u64) into one 128-byte swizzled row of an atom.
__device__ __forceinline__ void expand_row(uint8_t *atom, uint32_t r, uint64_t lo, uint64_t hi) {
    uint8_t *row = atom + r * 128;
    const uint32_t x = r & 7;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint64_t w = c < 4 ? lo : hi;
        const uint32_t bits = (uint32_t)(w >> ((c & 3) * 16)) & 0xffffu;
        const uint4 v = make_uint4(nib4(bits & 15), nib4((bits >> 4) & 15), nib4((bits >> 8) & 15), nib4(bits >> 12));
        *reinterpret_cast<uint4 *>(row + ((c ^ x) << 4)) = v;
    }
}

// Bit slices arrive by TMA (box 4 words x 128 rows per operand) into a ring of
// kTcRing slots issued kTcRing steps ahead; expansion reads them from shared
// memory, and the two fp8 stages alternate so that expanding step i+1
// overlaps the tensor core's MMAs on step i.
constexpr int kTcRing = 6;
constexpr int kTcBitTile = 128 * 32;       // one operand's bit slice: 128 rows x 4 words
constexpr int kTcBitSlot = 2 * kTcBitTile;

__global__ void __launch_bounds__(kTcThreads, 1)
    cooc_tc_kernel(const __grid_constant__ CUtensorMap bm_map, uint64_t n_words, uint32_t d, uint32_t n_tiles,
                   uint64_t words_per_split, uint32_t *__restrict__ out, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mma_bar[kTcStages];
    __shared__ uint64_t bit_bar[kTcRing];
    __shared__ uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    uint32_t t = blockIdx.x, bi = 0;
    while (t >= n_tiles - bi) { t -= n_tiles - bi; ++bi; }
    const uint32_t bj = bi + t;
    const uint64_t w_begin = (uint64_t)blockIdx.y * words_per_split;
    const uint64_t w_end = min(n_words, w_begin + words_per_split);
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = base + (size_t)kTcStages * kTcStageBytes;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(kTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s) mbar_init(&mma_bar[s], 1);
        for (int s = 0; s < kTcRing; ++s) mbar_init(&bit_bar[s], 1);
        mbar_init(&done_bar, 1);
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    const uint64_t n_steps = w_begin < w_end ? (w_end - w_begin + 3) / 4 : 0;  // 4 words = 256 bits per step
    auto issue = [&](uint64_t step) {
        const uint32_t slot = (uint32_t)(step % kTcRing);
        uint8_t *dst = ring + (size_t)slot * kTcBitSlot;
        mbar_arrive_expect_tx(&bit_bar[slot], kTcBitSlot);
        const int32_t x = (int32_t)(w_begin + step * 4);
        tma_load_2d(dst, &bm_map, x, (int32_t)(bi * 128), &bit_bar[slot]);
        tma_load_2d(dst + kTcBitTile, &bm_map, x, (int32_t)(bj * 128), &bit_bar[slot]);
    };
    if (tid == 0)
        for (uint64_t sidx = 0; sidx < n_steps && sidx < (uint64_t)kTcRing; ++sidx) issue(sidx);
    bool ok = true;
    for (uint64_t it = 0; it < n_steps; ++it) {
        const uint32_t slot = (uint32_t)(it % kTcRing);
        const uint32_t s = (uint32_t)(it % kTcStages);
        uint8_t *stage = base + (size_t)s * kTcStageBytes;
        ok = mbar_wait_bounded(&bit_bar[slot], (uint32_t)((it / kTcRing) & 1), err);
        if (ok && it >= kTcStages)
            ok = mbar_wait_bounded(&mma_bar[s], (uint32_t)((it / kTcStages - 1) & 1), err);
        if (__syncthreads_or(!ok)) break;
        {
            // thread -> one row of A (tid < 128) or B (tid >= 128): 4 words from the ring
            const uint32_t r = tid & 127;
            const uint8_t *src = ring + (size_t)slot * kTcBitSlot + (tid < 128 ? 0 : kTcBitTile) + r * 32;
            const uint4 x0 = *reinterpret_cast<const uint4 *>(src);
            const uint4 x1 = *reinterpret_cast<const uint4 *>(src + 16);
            uint8_t *op = stage + (tid < 128 ? 0 : kTcOperand);
            expand_row(op, r, (uint64_t)x0.x | ((uint64_t)x0.y << 32), (uint64_t)x0.z | ((uint64_t)x0.w << 32));
            expand_row(op + kTcAtom, r, (uint64_t)x1.x | ((uint64_t)x1.y << 32),
                       (uint64_t)x1.z | ((uint64_t)x1.w << 32));
        }
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_addr(stage), b0 = smem_addr(stage + kTcOperand);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t off = (uint32_t)(k >> 2) * kTcAtom + (uint32_t)(k & 3) * 32;
                tc_mma(tmem, smem_desc_sw128(a0 + off), smem_desc_sw128(b0 + off), (it > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit(&mma_bar[s]);
            // every thread has read this ring slot: refill it kTcRing steps ahead
            if (it + kTcRing < n_steps) issue(it + kTcRing);
        }
    }
    // wait for every MMA before reading the accumulator
    if (tid == 0 && n_steps > 0) tc_commit(&done_bar);
    __syncthreads();
    if (ok && n_steps > 0) ok = mbar_wait_bounded(&done_bar, 0, err);
    tc_fence_after();
    if (__syncthreads_or(!ok) == 0 && n_steps > 0 && warp < 4) {
        const uint32_t lane_base = warp * 32;
        const uint32_t row = bi * 128 + lane_base + (tid & 31);
#pragma unroll 1
        for (uint32_t cb = 0; cb < kTcCols; cb += 32) {
            uint32_t v[32];
            const uint32_t taddr = tmem + (lane_base << 16) + cb;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(taddr));
            tmem_wait_ld(v);
            if (row < d) {
#pragma unroll
                for (int q = 0; q < 32; ++q) {
                    const uint32_t col = bj * 128 + cb + q;
                    const uint32_t cnt = (uint32_t)__uint_as_float(v[q]);
                    if (col < d && cnt) {
                        atomicAdd(&out[(uint64_t)row * d + col], cnt);
                        if (bi != bj) atomicAdd(&out[(uint64_t)col * d + row], cnt);
                    }
                }
            }
        }
    }
    if (!ok) {
        // let copies still in flight land before the CTA's shared memory goes away
        for (int sidx = 0; sidx < kTcRing; ++sidx) mbar_wait_bounded(&bit_bar[sidx], 0, err);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
    }
}

// ---------------------------------------------------------------- 256 x 256 blocks
// The same product with a CTA per upper-triangle 256 x 256 block.  Per step
// (128 transactions) the bit slices of the block's 256 A rows and 256 B rows
// are expanded into one 128B-swizzled K-major atom per operand (B's atom is
// 256 rows tall), and per K = 32 substep two MMAs M = 128 (the two halves of
// A) x N = 256 accumulate into two 256-column fp32 accumulators (all 512 TMEM
// columns).  Each expanded slice feeds twice the MMA work of the 128 x 128
// form, and a diagonal block expands its rows once and uses them as A and B.
//
// Warp roles, coordinated by mbarriers only (no CTA-wide barrier per step):
//   warps 0..15  expansion: a row of A (warps 0..7) or of B (8..15) per thread
//                (half a row of the shared operand on the diagonal); wait ring_full and
//                stage_empty, expand, fence the async proxy, arrive on
//                stage_full and ring_empty (one arrival per warp).  A ring slot is released
//                behind the stores that used its bits: released behind the loads alone, a
//                diagonal block now and then expanded rows of the step that refilled the
//                slot (14 of 50,000 calls had wrong counts);
//   warp 16      one thread issues the MMAs of a step once stage_full completes
//                and commits them to stage_empty;
//   warp 17      one thread keeps the TMA ring of bit slices (2 words x 256
//                rows per operand, 16-byte rows read row-wise) kT2Ring steps ahead.
// Three 64-KB stages let the expansion run two steps ahead of the tensor core.
constexpr int kT2Rows = 256;
constexpr int kT2ExpWarps = 16;
constexpr int kT2Threads = 32 * (kT2ExpWarps + 2);
constexpr int kT2Cols = 512;                        // two 128 x 256 fp32 accumulators
constexpr int kT2AtomA = 256 * 128;                 // A: 256 rows x 128 B (two M halves)
constexpr int kT2AtomB = 256 * 128;                 // B: 256 rows x 128 B
constexpr int kT2StageBytes = kT2AtomA + kT2AtomB;  // 64 KB
constexpr int kT2Stages = 3;
constexpr int kT2Ring = 4;
constexpr int kT2BitBox = 256 * 16;                 // one operand's slice: 256 rows x 2 words
constexpr int kT2BitSlot = 2 * kT2BitBox;
constexpr uint32_t kT2Idesc = (1u << 4) | ((256u >> 3) << 17) | ((128u >> 4) << 24);   // D f32, e4m3, N=256, M=128

__device__ __forceinline__ void tc_mma_n256(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(kT2Idesc), "r"(acc)
        : "memory");
}

// Expand 64 bits (chunks 4*half .. 4*half+3 of a 128-byte swizzled row).
__device__ __forceinline__ void expand_half(uint8_t *atom, uint32_t r, uint32_t half, uint64_t w) {
    uint8_t *row = atom + r * 128;
    const uint32_t x = r & 7;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t bits = (uint32_t)(w >> (c * 16)) & 0xffffu;
        const uint4 v = make_uint4(nib4(bits & 15), nib4((bits >> 4) & 15), nib4((bits >> 8) & 15), nib4(bits >> 12));
        *reinterpret_cast<uint4 *>(row + (((half * 4 + c) ^ x) << 4)) = v;
    }
}

__global__ void __launch_bounds__(kT2Threads, 1)
    cooc_tc256_kernel(const __grid_constant__ CUtensorMap bm_map, uint64_t n_words, uint32_t d, uint32_t n_blocks,
                      uint64_t words_per_split, uint32_t *__restrict__ out, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t ring_full[kT2Ring], ring_empty[kT2Ring], stage_full[kT2Stages], stage_empty[kT2Stages];
    __shared__ uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t failed;              // a role gave up on a wait: the others stop
    __shared__ unsigned long long issued_n;           // ring steps issued (producer)
    uint32_t t = blockIdx.x, bi = 0;
    while (t >= n_blocks - bi) { t -= n_blocks - bi; ++bi; }
    const uint32_t bj = bi + t;
    const bool diag = bi == bj;
    const uint64_t w_begin = (uint64_t)blockIdx.y * words_per_split;
    const uint64_t w_end = min(n_words, w_begin + words_per_split);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = base + (size_t)kT2Stages * kT2StageBytes;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(kT2Cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kT2Ring; ++s) {
            mbar_init(&ring_full[s], 1);
            mbar_init(&ring_empty[s], kT2ExpWarps);
        }
        for (int s = 0; s < kT2Stages; ++s) {
            mbar_init(&stage_full[s], kT2ExpWarps);
            mbar_init(&stage_empty[s], 1);
        }
        mbar_init(&done_bar, 1);
        fence_mbar_init();
        failed = 0;
        issued_n = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint64_t n_steps = w_begin < w_end ? (w_end - w_begin + 1) / 2 : 0;   // 2 words = 128 bits per step

    if (warp < kT2ExpWarps) {
        // ---- expansion
        // warps 0..7: row tid of A; warps 8..15: row tid - 256 of B (on the diagonal,
        // half tid >> 8 of row tid & 255 of the shared operand)
        const uint32_t r = tid & 255, sel = tid >> 8;
        for (uint64_t it = 0; it < n_steps; ++it) {
            if (__any_sync(0xffffffffu, failed != 0)) break;   // the same decision for the whole warp
            const uint32_t slot = (uint32_t)(it % kT2Ring), s = (uint32_t)(it % kT2Stages);
            uint8_t *stage = base + (size_t)s * kT2StageBytes;
            bool ok = mbar_wait_bounded(&ring_full[slot], (uint32_t)((it / kT2Ring) & 1), err);
            uint4 a = make_uint4(0, 0, 0, 0);
            if (ok) {
                const uint8_t *src = ring + (size_t)slot * kT2BitSlot + r * 16;
                if (!diag) {
                    a = *reinterpret_cast<const uint4 *>(src + sel * kT2BitBox);
                } else {
                    const uint2 hw = *reinterpret_cast<const uint2 *>(src + sel * 8);
                    a.x = hw.x;
                    a.y = hw.y;
                }
            }
            if (ok && it >= kT2Stages)
                ok = mbar_wait_bounded(&stage_empty[s], (uint32_t)((it / kT2Stages - 1) & 1), err);
            if (!__all_sync(0xffffffffu, ok)) {
                failed = 1;
                break;
            }
            if (!diag)
                expand_row(stage + sel * kT2AtomA, r, (uint64_t)a.x | ((uint64_t)a.y << 32),
                           (uint64_t)a.z | ((uint64_t)a.w << 32));
            else
                expand_half(stage, r, sel, (uint64_t)a.x | ((uint64_t)a.y << 32));
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&stage_full[s]);
                mbar_arrive(&ring_empty[slot]);   // the slot's bits have been used (not only asked for)
            }
        }
    } else if (warp == kT2ExpWarps) {
        // ---- MMA issue (one thread)
        if (lane == 0) {
            for (uint64_t it = 0; it < n_steps && !failed; ++it) {
                const uint32_t s = (uint32_t)(it % kT2Stages);
                if (!mbar_wait_bounded(&stage_full[s], (uint32_t)((it / kT2Stages) & 1), err)) {
                    failed = 1;
                    break;
                }
                tc_fence_after();
                uint8_t *stage = base + (size_t)s * kT2StageBytes;
                const uint32_t a0 = smem_addr(stage), b0 = diag ? a0 : smem_addr(stage + kT2AtomA);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        tc_mma_n256(tmem + (uint32_t)h * 256u,
                                    smem_desc_sw128(a0 + (uint32_t)h * 128u * 128u + k * 32),
                                    smem_desc_sw128(b0 + k * 32), (it > 0 || k > 0) ? 1u : 0u);
                }
                tc_commit(&stage_empty[s]);
            }
            // every MMA issued so far, also after a failed wait (they still read the stages)
            if (n_steps > 0) tc_commit(&done_bar);
        }
    } else {
        // ---- TMA producer (one thread)
        if (lane == 0) {
            const uint32_t slot_bytes = diag ? kT2BitBox : kT2BitSlot;
            for (uint64_t it = 0; it < n_steps && !failed; ++it) {
                const uint32_t slot = (uint32_t)(it % kT2Ring);
                if (it >= kT2Ring &&
                    !mbar_wait_bounded(&ring_empty[slot], (uint32_t)((it / kT2Ring - 1) & 1), err)) {
                    failed = 1;
                    break;
                }
                uint8_t *dst = ring + (size_t)slot * kT2BitSlot;
                mbar_arrive_expect_tx(&ring_full[slot], slot_bytes);
                const int32_t x = (int32_t)(w_begin + it * 2);
                tma_load_2d(dst, &bm_map, x, (int32_t)(bi * kT2Rows), &ring_full[slot]);
                if (!diag) tma_load_2d(dst + kT2BitBox, &bm_map, x, (int32_t)(bj * kT2Rows), &ring_full[slot]);
                issued_n = it + 1;
            }
        }
    }
    __syncthreads();
    bool ok = !failed;
    if (n_steps > 0 && !mbar_wait_bounded(&done_bar, 0, err)) ok = false;
    tc_fence_after();
    if (__syncthreads_or(!ok) == 0 && n_steps > 0 && warp < kT2ExpWarps) {
        // warp w reads the 32 TMEM lanes of quadrant w % 4 in accumulator (w / 4) % 2,
        // columns 128 * (w / 8) .. +127
        const uint32_t q = warp & 3, h = (warp >> 2) & 1, c0 = (warp >> 3) * 128;
        const uint32_t row = bi * kT2Rows + h * 128 + q * 32 + lane;
#pragma unroll 1
        for (uint32_t cb = c0; cb < c0 + 128; cb += 32) {
            uint32_t v[32];
            const uint32_t taddr = tmem + ((q * 32) << 16) + h * 256 + cb;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(taddr));
            tmem_wait_ld(v);
            if (row < d) {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const uint32_t col = bj * kT2Rows + cb + c;
                    const uint32_t cnt = (uint32_t)__uint_as_float(v[c]);
                    if (col < d && cnt) {
                        atomicAdd(&out[(uint64_t)row * d + col], cnt);
                        if (!diag) atomicAdd(&out[(uint64_t)col * d + row], cnt);
                    }
                }
            }
        }
    }
    if (!ok) {
        // let the copies still in flight land before the CTA's shared memory goes
        // away: the last issued step of every ring slot, with its own phase
        const uint64_t g1 = issued_n;
        for (uint64_t g = g1 > (uint64_t)kT2Ring ? g1 - kT2Ring : 0; g < g1; ++g)
            mbar_wait_bounded(&ring_full[g % kT2Ring], (uint32_t)((g / kT2Ring) & 1), err);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kT2Cols) : "memory");
    }
}

// ---------------------------------------------------------------- fp4, 128 x 256 tiles
// The same product with 4-bit operands: tcgen05.mma kind::mxf4 (e2m1 with
// block scales) multiplies K = 64 transactions per instruction at twice the
// fp8 rate and half its bytes.  Every product is exactly 0 or 1 and the fp32 sums
// are the same exact integers.
//
// What the 256 x 256 form above is bound by is shared memory: per K = 32 it
// writes 16 KB of expanded operands and the MMAs read 24 KB (320 clocks) for 256
// clocks of tensor work.  Here A is expanded into tensor memory and only B goes
// through shared memory: per K = 64 with M = 128, N = 256, 8 KB written and 8 KB
// read (128 clocks) for 128 clocks of tensor work, and 6 KB of bit slices.  The
// expansion is cheaper too: the order of the transactions inside
// a K step does not matter as long as A and B share it, so a 32-bit word becomes
// four registers by shift and mask, register i holding bits i, i + 4, i + 8, ...
// as nibbles (5 instructions where the byte form needs 40).
//
// Bits arrive by TMA in rows of 64 bytes, two steps at a time.
//
// The work is cut into runs of transactions, all tiles of a run next to each
// other, so the CTAs that read the same rows read them at the same time (from L2:
// with a tile's runs next to each other the bitmaps came 4 times from HBM).  How it is cut
// and dealt is in cooc_plan.h; a CTA may end one tile and begin the next.  Counts are added to out and its
// mirror with coalesced atomics (the mirror through a shared-memory transpose).
// A diagonal tile's A rows are a half of its B rows: their bits are loaded once.
//
// Warp roles, as in the 256 x 256 form: two groups of 12 warps expand the even and
// the odd steps, a row per thread (eight warps B, four A), and all 24 read the
// accumulators at a tile's end; warp 24 issues the MMAs, warp 25 the TMA loads.
//
// Measured, 1,024 rows x 1,048,576 transactions: 0.30 ms a call (0.525 for the 256 x
// 256 form); tensor pipe 50%, and shared memory (expansion writes with their
// conflicts 310 clocks a step, the MMAs' reads 256, bit slices 200) about 75% of a
// step's 1,070 clocks.  Before: A through shared memory too 0.36 ms; a single group
// of 12 expansion warps 0.32; stage and phase divided out by the MMA thread every
// step 0.33.  No difference: 3 or 4 stages, 64- or 128-byte rows, 5 or 7 instructions
// per expanded word.
constexpr int kF4GroupWarps = 12;                        // warps that expand one step
constexpr int kF4ExpWarps = 2 * kF4GroupWarps;
constexpr int kF4Threads = 32 * (kF4ExpWarps + 2);
constexpr int kF4RowsA = 128, kF4RowsB = 256;
constexpr int kF4Words = 8;                              // 64-bit words of a double step: 512 transactions
constexpr int kF4StageBytes = kF4RowsB * 128;            // B, one step: 32 KB
constexpr int kF4Stages = 3;
constexpr int kF4Ring = 5;
constexpr int kF4RowBytes = kF4Words * 8;
constexpr int kF4RingBytes = (kF4RowsA + kF4RowsB) * kF4RowBytes;   // 24 KB
static_assert(kF4Words == 8 && kF4RowsA == 128 && kF4RowsB == 256, "f4_plan cuts the work for these tiles and steps");
constexpr int kF4Turn = 32 * 17;                         // words of a warp's 32 x 16 transpose buffer
constexpr uint32_t kF4ScaleCol = 256;                    // block scales: TMEM columns 256..319
constexpr uint32_t kF4ColA = 320;                        // A: 32 columns (256 values per row) per stage
// A, B e2m1; scale format ue8m0; N = 256, M = 128; K = 64
constexpr uint32_t kF4Idesc = (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);

// A from tensor memory, B from shared memory
__device__ __forceinline__ void tc_mma_f4(uint32_t tmem, uint32_t a, uint64_t bdesc, uint32_t scale_a,
                                          uint32_t scale_b, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%5], p;\n\t}" ::"r"(
            tmem),
        "r"(a), "l"(bdesc), "r"(kF4Idesc), "r"(scale_a), "r"(scale_b), "r"(acc)
        : "memory");
}

// 128 bits -> four 16-byte pieces (32 values each).  Piece i holds bits i, i + 4,
// i + 8, ... of the four words as nibbles: bits 0, 1 and 2 stay where they are and
// read as 0.5, 1 and 2, bit 3 moves to bit 2 (where it would be the sign).  The
// block scales (one per 32 values) make every product 1: 2 x 2 for piece 0, 1 x 1
// for piece 1, 1/2 x 1/2 for pieces 2 and 3.
__device__ __forceinline__ uint4 mask4(const uint4 &x, uint32_t m) {
    return make_uint4(x.x & m, x.y & m, x.z & m, x.w & m);
}
__device__ __forceinline__ void expand_f4(const uint4 &x, uint4 (&p)[4]) {
    p[0] = mask4(x, 0x11111111u);
    p[1] = mask4(x, 0x22222222u);
    p[2] = mask4(x, 0x44444444u);
    p[3] = mask4(make_uint4(x.x >> 1, x.y >> 1, x.z >> 1, x.w >> 1), 0x44444444u);
}
constexpr uint32_t kF4ScaleLow = 0x7f807f80u, kF4ScaleHigh = 0x7e7e7e7eu;   // pieces 0 and 1; 2 and 3 (ue8m0)

// 128 bits of a row -> 16 TMEM columns of e2m1 values.
__device__ __forceinline__ void tmem_st_f4(uint32_t taddr, const uint4 &x) {
    uint4 p[4];
    expand_f4(x, p);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(p[0].x), "r"(p[0].y), "r"(p[0].z), "r"(p[0].w), "r"(p[1].x), "r"(p[1].y), "r"(p[1].z), "r"(p[1].w),
        "r"(p[2].x), "r"(p[2].y), "r"(p[2].z), "r"(p[2].w), "r"(p[3].x), "r"(p[3].y), "r"(p[3].z), "r"(p[3].w)
        : "memory");
}

// 256 bits of a row -> its 128 bytes in stage ST; at[c]: address of piece c in stage 0.
template <int ST>
__device__ __forceinline__ void smem_st_f4(uint8_t *base, const uint32_t (&at)[8], const uint4 &x0, const uint4 &x1) {
    uint4 p[4];
    expand_f4(x0, p);
#pragma unroll
    for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4 *>(base + at[c] + ST * kF4StageBytes) = p[c];
    expand_f4(x1, p);
#pragma unroll
    for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4 *>(base + at[4 + c] + ST * kF4StageBytes) = p[c];
}

__global__ void __launch_bounds__(kF4Threads, 1)
    cooc_f4_kernel(const __grid_constant__ CUtensorMap bm_map, F4Work work, uint32_t *__restrict__ out, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t ring_full[kF4Ring], ring_empty[kF4Ring], stage_full[kF4Stages], stage_empty[kF4Stages];
    __shared__ uint64_t done_bar, free_bar;           // a tile's MMAs are done; its accumulators have been read
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t failed;              // a role gave up on a wait: the others stop
    __shared__ unsigned long long issued_n;           // ring steps issued (producer)
    const uint64_t limit = mbar_limit_ns(err);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = base + (size_t)kF4Stages * kF4StageBytes;
    uint32_t *turn = reinterpret_cast<uint32_t *>(base);   // transposes, while no stage is in use
    uint64_t g0, g1;
    f4_part(work, blockIdx.x, g0, g1);

    if (warp == 0) tmem_alloc(&tmem_slot, 512);
    if (tid == 0) {
        for (int i = 0; i < kF4Ring; ++i) {
            mbar_init(&ring_full[i], 1);
            mbar_init(&ring_empty[i], kF4ExpWarps);
        }
        for (int i = 0; i < kF4Stages; ++i) {
            mbar_init(&stage_full[i], kF4GroupWarps);
            mbar_init(&stage_empty[i], 1);
        }
        mbar_init(&done_bar, 1);
        mbar_init(&free_bar, kF4ExpWarps);
        fence_mbar_init();
        failed = 0;
        issued_n = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (warp < 4) {   // the scales, the same in every lane: A low, B low, A high, B high
        const uint32_t at = tmem + ((warp * 32u) << 16) + kF4ScaleCol;
#pragma unroll 1
        for (uint32_t c = 0; c < 64; ++c)
            asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(at + c),
                         "r"(c < 32 ? kF4ScaleLow : kF4ScaleHigh)
                         : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // every role walks the same units: ns double steps of a tile
    // (t: double steps of this CTA before the unit; double step t uses ring slot t % kF4Ring, its
    // steps 2t and 2t + 1 stages 2t % kF4Stages and the next)
    uint32_t t = 0;
    uint32_t mma_st = 0, mma_par = 0;                      // stage and phase of the next MMAs
    const uint64_t desc0 = smem_desc_sw128(smem_addr(base));
    uint32_t unit_n = 0;      // units of this CTA so far (done_bar and free_bar phases)
    bool ok = true;
    for (uint64_t g = g0; g < g1 && ok; ++unit_n) {
        uint32_t bi, bj;
        uint64_t step0;
        const uint64_t follow = f4_unit(work, g, bi, bj, step0);
        const uint32_t ns = (uint32_t)min(g1 - g, follow);
        const bool diag = (bi >> 1) == bj;   // A is half bi & 1 of B
        if (warp < kF4ExpWarps) {
            // ---- expansion: threads 0..255 B rows (shared memory), 256..383 A rows (tensor memory)
            // of the group whose turn the step is
            const uint32_t group = warp >= kF4GroupWarps ? 1u : 0u, r = tid - group * kF4GroupWarps * 32;
            const bool is_a = r >= kF4RowsB;
            const uint32_t src_row = is_a && diag ? r - kF4RowsB + (bi & 1) * kF4RowsA : r;
            // the bits' 16-byte pieces are swizzled by TMA: piece c of row r at c ^ (r / 2 % 4)
            const uint32_t sel = (src_row >> 1) & 3;
            const uint8_t *src = ring + src_row * kF4RowBytes;
            uint32_t at[8];
#pragma unroll
            for (uint32_t c = 0; c < 8; ++c) at[c] = r * 128 + ((c ^ (r & 7)) << 4);
            const uint32_t a_at = tmem + (((warp & 3) * 32u) << 16) + kF4ColA;
            for (uint32_t k = t; k < t + ns; ++k) {
                const uint32_t slot = k % kF4Ring, step = 2 * k + group, use = step / kF4Stages,
                               st = step - use * kF4Stages;
                ok = mbar_wait_limit(&ring_full[slot], (k / kF4Ring) & 1, limit, err);
                uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
                if (ok) {
                    x0 = *reinterpret_cast<const uint4 *>(src + slot * kF4RingBytes + (((group * 2) ^ sel) << 4));
                    x1 = *reinterpret_cast<const uint4 *>(src + slot * kF4RingBytes + (((group * 2 + 1) ^ sel) << 4));
                }
                if (ok && use) ok = mbar_wait_limit(&stage_empty[st], (use - 1) & 1, limit, err);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                if (!is_a) {
                    if (st == 0) smem_st_f4<0>(base, at, x0, x1);
                    else if (st == 1) smem_st_f4<1>(base, at, x0, x1);
                    else smem_st_f4<2>(base, at, x0, x1);
                    fence_proxy_async_smem();
                } else {
                    tc_fence_after();
                    tmem_st_f4(a_at + st * 32, x0);
                    tmem_st_f4(a_at + st * 32 + 16, x1);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&stage_full[st]);
                    mbar_arrive(&ring_empty[slot]);   // the slot's bits have been used (not only asked for)
                }
            }
            // ---- the unit's counts: warp w reads TMEM quadrant w % 4, every sixth chunk of 16 columns
            if (ok) ok = mbar_wait_limit(&done_bar, unit_n & 1, limit, err);
            // one decision for all expansion warps: they meet at barriers from here on
            uint32_t bad;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t"
                "setp.eq.u32 p, %1, 0;\n\t"
                "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
                "selp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(bad)
                : "r"((uint32_t)ok), "n"(32 * kF4ExpWarps)
                : "memory");
            ok = bad == 0;
            if (!ok) {
                failed = 1;
                break;
            }
            tc_fence_after();
            const uint32_t q = warp & 3, d = work.d;
            const uint32_t row0 = bi * kF4RowsA + q * 32;
            uint32_t *mine = turn + warp * kF4Turn;
            for (uint32_t cb = (warp >> 2) * 16; cb < kF4RowsB; cb += kF4ExpWarps * 4) {
                const uint32_t col0 = bj * kF4RowsB + cb;
                if (col0 >= d || row0 >= d || col0 + 15 < row0) continue;   // nothing on or above the diagonal
                uint32_t v[16];
                tmem_ld16(tmem + ((q * 32u) << 16) + cb, v);
                tmem_wait_ld(v);
                const uint32_t row = row0 + lane;
                __syncwarp();
#pragma unroll
                for (uint32_t c = 0; c < 16; ++c) {
                    const uint32_t col = col0 + c, cnt = (uint32_t)__uint_as_float(v[c]);
                    mine[lane * 17 + c] = cnt;
                    if (cnt && row < d && col < d && col > row) atomicAdd(&out[(uint64_t)col * d + row], cnt);
                }
                __syncwarp();
#pragma unroll 4
                for (uint32_t r2 = 0; r2 < 32; r2 += 2) {   // two rows of 16 columns per instruction
                    const uint32_t rr = row0 + r2 + (lane >> 4), col = col0 + (lane & 15);
                    const uint32_t cnt = mine[(r2 + (lane >> 4)) * 17 + (lane & 15)];
                    if (cnt && rr < d && col < d && col >= rr) atomicAdd(&out[(uint64_t)rr * d + col], cnt);
                }
            }
            tc_fence_before();
            // the stages hold transposes until every warp is through
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kF4ExpWarps) : "memory");
            if (lane == 0) mbar_arrive(&free_bar);
        } else if (warp == kF4ExpWarps) {
            // ---- MMA issue (one thread; its serial chain is on the path of every step, so stage,
            // phase and descriptors are carried along instead of computed)
            if (lane == 0) {
                if (unit_n > 0) ok = mbar_wait_limit(&free_bar, (unit_n - 1) & 1, limit, err);
                uint32_t acc = 0;
                for (uint32_t k = 2 * ns; k > 0; --k) {
                    if (!ok || !mbar_wait_limit(&stage_full[mma_st], mma_par, limit, err)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t bd = desc0 + mma_st * (uint32_t)(kF4StageBytes >> 4);
                    const uint32_t a0 = tmem + kF4ColA + mma_st * 32, sc = tmem + kF4ScaleCol;
                    // K steps of 64: pieces 0 and 1, then 2 and 3, of either 128 bits
                    tc_mma_f4(tmem, a0, bd, sc, sc + 16, acc);
                    acc = 1;
                    tc_mma_f4(tmem, a0 + 8, bd + 2, sc + 32, sc + 48, 1u);
                    tc_mma_f4(tmem, a0 + 16, bd + 4, sc, sc + 16, 1u);
                    tc_mma_f4(tmem, a0 + 24, bd + 6, sc + 32, sc + 48, 1u);
                    tc_commit(&stage_empty[mma_st]);
                    if (++mma_st == kF4Stages) {
                        mma_st = 0;
                        mma_par ^= 1;
                    }
                }
                if (!ok) failed = 1;
                tc_commit(&done_bar);   // also after a failed wait: the MMAs issued still read the stages
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        } else {
            // ---- TMA producer (one thread)
            if (lane == 0) {
                const uint32_t bytes = diag ? kF4RowsB * kF4RowBytes : kF4RingBytes;
                for (uint32_t k = 0; k < ns; ++k) {
                    const uint32_t slot = (t + k) % kF4Ring, use = (t + k) / kF4Ring;
                    if (failed || (use && !mbar_wait_limit(&ring_empty[slot], (use - 1) & 1, limit, err))) {
                        ok = false;
                        break;
                    }
                    uint8_t *dst = ring + (size_t)slot * kF4RingBytes;
                    mbar_arrive_expect_tx(&ring_full[slot], bytes);
                    const int32_t x = (int32_t)((step0 + k) * kF4Words);
                    for (int h = 0; h < 2; ++h)
                        tma_load_2d(dst + h * 128 * kF4RowBytes, &bm_map, x, (int32_t)(bj * kF4RowsB + h * 128),
                                    &ring_full[slot]);
                    if (!diag)
                        tma_load_2d(dst + kF4RowsB * kF4RowBytes, &bm_map, x, (int32_t)(bi * kF4RowsA), &ring_full[slot]);
                    issued_n = issued_n + 1;
                }
                if (!ok) failed = 1;
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        }
        g += ns;
        t += ns;
    }
    __syncthreads();
    if (failed) {
        // let what is in flight land before the CTA's memory goes away: the MMAs issued (the
        // last commit of done_bar has this CTA's last phase), and the last box of every ring slot
        mbar_wait_limit(&done_bar, unit_n ? (unit_n - 1) & 1 : 0, limit, err);
        const uint64_t n1 = issued_n;
        for (uint64_t k = n1 > (uint64_t)kF4Ring ? n1 - kF4Ring : 0; k < n1; ++k)
            mbar_wait_limit(&ring_full[k % kF4Ring], (uint32_t)((k / kF4Ring) & 1), limit, err);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

bool encode_bits_map_box(CUtensorMap *map, const uint64_t *bitmaps, uint32_t d, uint64_t n_words,
                         uint64_t row_stride, uint32_t box_words, uint32_t box_rows,
                         CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE);

bool encode_bits_map(CUtensorMap *map, const uint64_t *bitmaps, uint32_t d, uint64_t n_words, uint64_t row_stride) {
    return encode_bits_map_box(map, bitmaps, d, n_words, row_stride, 4, 128);
}

bool encode_bits_map_box(CUtensorMap *map, const uint64_t *bitmaps, uint32_t d, uint64_t n_words,
                         uint64_t row_stride, uint32_t box_words, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
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
    cuuint64_t dims[2] = {(cuuint64_t)n_words, (cuuint64_t)d};
    cuuint64_t strides[1] = {(cuuint64_t)row_stride * 8};
    cuuint32_t box[2] = {box_words, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<uint64_t *>(bitmaps), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

size_t tc_smem_bytes() { return (size_t)kTcStages * kTcStageBytes + (size_t)kTcRing * kTcBitSlot + 1024; }
size_t f4_smem_bytes() {
    static_assert(kF4ExpWarps * kF4Turn * 4 <= kF4Stages * kF4StageBytes, "transposes use the stages' memory");
    return (size_t)kF4Stages * kF4StageBytes + (size_t)kF4Ring * kF4RingBytes + 1024;
}
size_t tc256_smem_bytes() { return (size_t)kT2Stages * kT2StageBytes + (size_t)kT2Ring * kT2BitSlot + 1024; }

int cooc_f4_device(const uint64_t *bitmaps, uint32_t d, uint64_t n_words, uint64_t row_stride, uint32_t *out,
                   cudaStream_t st, int n_sm, uint32_t *dev_err, uint64_t *launches) {
    if (d == 0) return 0;
    if ((reinterpret_cast<uintptr_t>(bitmaps) & 15) || (row_stride & 1)) return -1;
    CUtensorMap map;
    if (n_words && !encode_bits_map_box(&map, bitmaps, d, n_words, row_stride, kF4Words, 128,
                                        CU_TENSOR_MAP_SWIZZLE_64B))
        return -1;
    SG_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)d * d * 4, st));
    if (n_words == 0) return 0;
    const F4Work w = f4_plan(d, n_words, (uint64_t)n_sm);
    const size_t smem = f4_smem_bytes();
    SG_CUDA_TRY(cudaFuncSetAttribute(cooc_f4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cooc_f4_kernel<<<(unsigned)w.ctas, kF4Threads, smem, st>>>(map, w, out, dev_err);
    SG_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += 1;
    return 0;
}

int cooc_tc256_device(const uint64_t *bitmaps, uint32_t d, uint64_t n_words, uint64_t row_stride, uint32_t *out,
                      cudaStream_t st, int n_sm, uint32_t *dev_err, uint64_t *launches) {
    if (d == 0) return 0;
    if ((reinterpret_cast<uintptr_t>(bitmaps) & 15) || (row_stride & 1)) return -1;
    SG_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)d * d * 4, st));
    const uint32_t n_blocks = (d + kT2Rows - 1) / kT2Rows;
    const uint32_t pairs = n_blocks * (n_blocks + 1) / 2;
    // one wave: split the transactions so that pairs x splits <= SMs; each split
    // covers at most 2^20 transactions (fp32 exactness of the partial counts);
    // splits start on an even word (TMA boxes of two words)
    uint64_t splits = std::max<uint64_t>(1, (uint64_t)n_sm / pairs);
    uint64_t wps = (n_words + splits - 1) / splits;
    wps = std::min<uint64_t>(wps, (1ull << 20) / 64);
    wps = (wps + 1) / 2 * 2;
    splits = (n_words + wps - 1) / wps;
    CUtensorMap map;
    if (!encode_bits_map_box(&map, bitmaps, d, n_words, row_stride, 2, kT2Rows)) return -1;
    const size_t smem = tc256_smem_bytes();
    SG_CUDA_TRY(cudaFuncSetAttribute(cooc_tc256_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid(pairs, (unsigned)splits);
    cooc_tc256_kernel<<<grid, kT2Threads, smem, st>>>(map, n_words, d, n_blocks, wps, out, dev_err);
    SG_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += 1;
    return 0;
}

int cooc_tc_device(const uint64_t *bitmaps, uint32_t d, uint64_t n_words, uint64_t row_stride, uint32_t *out,
                   cudaStream_t st, int n_sm, uint32_t *dev_err, uint64_t *launches) {
    if (d == 0) return 0;
    if ((reinterpret_cast<uintptr_t>(bitmaps) & 15) || (row_stride & 1)) return -1;
    SG_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)d * d * 4, st));
    const uint32_t n_tiles = (d + 127) / 128;
    const uint32_t pairs = n_tiles * (n_tiles + 1) / 2;
    // one wave: split the transactions so that pairs x splits <= SMs; each split
    // covers at most 2^20 transactions (fp32 exactness of the partial counts)
    uint64_t splits = std::max<uint64_t>(1, (uint64_t)n_sm / pairs);
    uint64_t wps = (n_words + splits - 1) / splits;
    wps = std::min<uint64_t>(wps, (1ull << 20) / 64);
    wps = (wps + 3) / 4 * 4;
    splits = (n_words + wps - 1) / wps;
    CUtensorMap map;
    if (!encode_bits_map(&map, bitmaps, d, n_words, row_stride)) return -1;
    const size_t smem = tc_smem_bytes();
    SG_CUDA_TRY(cudaFuncSetAttribute(cooc_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid(pairs, (unsigned)splits);
    cooc_tc_kernel<<<grid, kTcThreads, smem, st>>>(map, n_words, d, n_tiles, wps, out, dev_err);
    SG_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += 1;
    return 0;
}

}  // namespace sg
