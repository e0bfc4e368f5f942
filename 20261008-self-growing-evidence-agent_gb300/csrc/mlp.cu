// mlp.cu -- the frontier-scoring MLP: fused forward, backward and Adam kernels.
//
// No reference counterpart (the reference orders its search by singleton
// support only, kernel_bitmap.cu:276-283).  Network: in_dim -> H -> H -> 1,
// ReLU, sigmoid output; weights are bf16 (row-major [out][in]), biases,
// activations and accumulation fp32.  Training keeps fp32 master weights
// and refreshes the bf16 copy after every Adam step.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdio>

#include "common.cuh"
#include "engine.h"
#include "tcgen05.cuh"

namespace sg {

constexpr int kMlpMaxIn = 64;

__device__ __forceinline__ float bf2f(uint16_t b) { return __uint_as_float(((uint32_t)b) << 16); }

// ---------------------------------------------------------------- forward
// A CTA owns tiles of 128 rows.  Layer 1 (in_dim multiply-adds per hidden unit)
// runs on the CUDA cores; layer 2 is the contraction and runs on the tensor
// cores: h1 is fp32, so each value is cut into three bf16 parts (its top 8
// significant bits, the next 8, the last 8: the cut is exact) that are
// multiplied with the bf16 weights by tcgen05.mma and accumulated in fp32 in
// tensor memory, the top parts in one accumulator and the two small parts in
// another.  Layer 3 and the sigmoid read both back.
//
// Per 64 hidden units (one 128-byte swizzle atom of K): 256 threads compute
// two rows x 16 units each, write the three parts as K-major atoms, and one
// thread issues the 12 MMAs (4 K steps x 3 parts, N = H).  Two CTAs share an SM
// when the weights and tensor memory allow (H <= 128), so one computes while
// the other's MMAs run.
//
// Bound: the chain of dependent steps of a tile, about 15,000 clocks of a CTA (2,000 of
// them waiting for MMAs) with 16 warps an SM; its shared memory traffic alone would take
// 3,800.  Layer 1 on the tensor cores too took a fifth of the instructions out and gave
// 66 us, 32 warps an SM 72 us.
// Measured (300,000 rows, H = 128, whole call): 64 us against 1,560 us for one
// thread per hidden unit with scalar multiply-adds (a shared-memory load for each).  Of
// that, 6 us came from two-float multiply-adds and the next tile's inputs fetched ahead, 4
// from reading W2 once, its loads in flight together.  Probabilities are off float64 by
// 2.4e-8 (root mean square; 2.5e-8 before), without a bias above 3e-9 (1.5e-9 before).
constexpr uint32_t kFwdRows = 128;
constexpr uint32_t kFwdThreads = 256;
constexpr uint32_t kFwdPart = kFwdRows * 128;   // one part's atom: 128 rows x 64 bf16
constexpr uint32_t kFwdXs = kFwdRows + 4;       // row pitch of the transposed inputs (conflict-free stores)

// Shared-memory layout (bytes from a 1,024-byte boundary).
struct FwdLayout {
    uint32_t a, w1, x, b1, b2, w3, red, bytes, w2_resident;
};
__host__ __device__ inline uint32_t mlp_chunks(uint32_t H) { return (H + 63) / 64; }
inline FwdLayout mlp_fwd_layout(uint32_t F, uint32_t H, bool w2_resident) {
    FwdLayout l;
    l.w2_resident = w2_resident;
    uint32_t at = (w2_resident ? mlp_chunks(H) : 1u) * H * 128;
    l.a = at;
    at += 3 * kFwdPart;
    l.w1 = at;
    at += F * H * 4;
    l.x = at;
    at += F * kFwdXs * 4;
    l.b1 = at;
    at += H * 4;
    l.b2 = at;
    at += H * 4;
    l.w3 = at;
    at += H * 4;
    l.red = at;
    at += 2 * kFwdRows * 4;
    l.bytes = at + 1024;
    return l;
}

// Two floats in one 64-bit register: Blackwell adds and multiplies them in one instruction.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Eight consecutive non-negative values of row r -> their three bf16 parts, as
// 16-byte piece c of the row in the three atoms.
__device__ __forceinline__ void store_parts(uint8_t *a, uint32_t r, uint32_t c, const float (&h)[8]) {
    uint32_t p[3][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t v[2] = {__float_as_uint(h[2 * q]), __float_as_uint(h[2 * q + 1])};
        p[0][q] = __byte_perm(v[0], v[1], 0x7632);
        // what the top part leaves (a value minus its top part: an add of the negated part); an
        // infinite value keeps its top part alone (inf - inf is NaN, whose maximum with 0 is 0)
        auto rest = [](uint32_t (&x)[2]) {
            float lo, hi;
            unpack2(add2(pack2(__uint_as_float(x[0]), __uint_as_float(x[1])),
                         pack2(__uint_as_float((x[0] & 0xffff0000u) | 0x80000000u),
                               __uint_as_float((x[1] & 0xffff0000u) | 0x80000000u))),
                    lo, hi);
            x[0] = __float_as_uint(lo);
            x[1] = __float_as_uint(hi);
        };
        rest(v);
#pragma unroll
        for (int e = 0; e < 2; ++e) v[e] = __float_as_uint(fmaxf(__uint_as_float(v[e]), 0.f));
        p[1][q] = __byte_perm(v[0], v[1], 0x7632);
        rest(v);
        p[2][q] = __byte_perm(v[0], v[1], 0x7632);
    }
    uint8_t *dst = a + r * 128 + ((c ^ (r & 7)) << 4);
#pragma unroll
    for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint4 *>(dst + k * kFwdPart) = make_uint4(p[k][0], p[k][1], p[k][2], p[k][3]);
}

// Eight bf16 weights W2[j][i .. i+7] (16-byte loads when the matrix is aligned).
__device__ __forceinline__ uint4 load_w8(const uint16_t *p, bool aligned) {
    if (aligned) return __ldg(reinterpret_cast<const uint4 *>(p));
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = (uint32_t)p[2 * q] | ((uint32_t)p[2 * q + 1] << 16);
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// an infinite or NaN bf16 in either half
__device__ __forceinline__ bool bf2_nonfinite(uint32_t w) {
    return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u;
}

// K chunk kc of W2 as a swizzled K-major atom of H rows x 64 columns; true when
// this thread met an infinite or NaN weight.
__device__ __forceinline__ bool load_w2_chunk(uint8_t *dst, const uint16_t *W2, uint32_t H, uint32_t kc, bool aligned) {
    const uint32_t shift = H - kc * 64 >= 64 ? 3 : 2, pieces = 1u << shift;   // H is a multiple of 32
    bool odd = false;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < H * pieces; i += kFwdThreads) {
        const uint32_t j = i >> shift, c = i & (pieces - 1);
        const uint4 w = load_w8(W2 + (size_t)j * H + kc * 64 + c * 8, aligned);
        odd |= bf2_nonfinite(w.x) || bf2_nonfinite(w.y) || bf2_nonfinite(w.z) || bf2_nonfinite(w.w);
        *reinterpret_cast<uint4 *>(dst + j * 128 + ((c ^ (j & 7)) << 4)) = w;
    }
    return odd;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

// Z1/Z2 (pre-activations) are written when non-null (training); vec: both
// allow 16-byte stores.  tm_cols: allocated TMEM columns (the two accumulators
// are its halves).
__global__ void __launch_bounds__(kFwdThreads, 2) mlp_fwd_kernel(
    const float *__restrict__ X, uint32_t n, uint32_t F, uint32_t H, const uint16_t *__restrict__ W1,
    const float *__restrict__ b1, const uint16_t *__restrict__ W2, const float *__restrict__ b2,
    const uint16_t *__restrict__ w3, const float *__restrict__ b3, float *__restrict__ Z1, float *__restrict__ Z2,
    float *__restrict__ P, FwdLayout lay, uint32_t tm_cols, uint32_t vec, uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t mma_bar;
    __shared__ uint32_t tmem_slot;
    uint8_t *sm = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    uint8_t *a = sm + lay.a;
    float *w1s = reinterpret_cast<float *>(sm + lay.w1);   // [F][H]
    float *xs = reinterpret_cast<float *>(sm + lay.x);     // [F][kFwdXs]
    float *b1s = reinterpret_cast<float *>(sm + lay.b1);
    float *b2s = reinterpret_cast<float *>(sm + lay.b2);
    float *w3s = reinterpret_cast<float *>(sm + lay.w3);
    float *red = reinterpret_cast<float *>(sm + lay.red);  // [2][128]
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t chunks = mlp_chunks(H);
    const bool w2_aligned = (reinterpret_cast<uintptr_t>(W2) & 15) == 0;

    if (warp == 0) tmem_alloc(&tmem_slot, tm_cols);
    if (tid == 0) {
        mbar_init(&mma_bar, 1);
        fence_mbar_init();
    }
    for (uint32_t i = tid; i < H * F; i += kFwdThreads) w1s[(i % F) * H + i / F] = bf2f(W1[i]);
    for (uint32_t i = tid; i < H; i += kFwdThreads) {
        b1s[i] = b1[i];
        b2s[i] = b2[i];
        w3s[i] = bf2f(w3[i]);
    }
    bool odd = false;   // an infinite or NaN weight: 0 parts times it would be NaN
    if (lay.w2_resident) {
        for (uint32_t kc = 0; kc < chunks; ++kc) odd |= load_w2_chunk(sm + kc * H * 128, W2, H, kc, w2_aligned);
    } else {
#pragma unroll 8
        for (uint32_t i = tid; i < H * H / 8; i += kFwdThreads) {
            const uint4 w = load_w8(W2 + (size_t)i * 8, w2_aligned);
            odd |= bf2_nonfinite(w.x) || bf2_nonfinite(w.y) || bf2_nonfinite(w.z) || bf2_nonfinite(w.w);
        }
    }
    tc_fence_before();
    const bool scalar = __syncthreads_or(odd);
    tc_fence_after();
    const uint32_t d_top = tmem_slot, d_low = d_top + tm_cols / 2;
    // D f32, A and B bf16, both K-major, N = H, M = 128
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((H >> 3) << 17) | ((128u >> 4) << 24);
    const float bias3 = b3[0];
    const uint32_t tiles = n / kFwdRows + (n % kFwdRows != 0);
    uint32_t parity = 0;
    bool ok = true;
    // eight aligned inputs a row (the search's features): a 16-byte load per thread and tile, one
    // tile ahead
    const bool quad = F == 8 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    float4 xq = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch_quad = [&](uint64_t tile) {
        const uint64_t row = tile * kFwdRows + (tid >> 1);
        xq = row < n ? __ldg(reinterpret_cast<const float4 *>(X + row * 8) + (tid & 1)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    if (quad) fetch_quad(blockIdx.x);
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t r0 = (uint64_t)tile * kFwdRows;
        if (quad) {
            const uint32_t r = tid >> 1, f = (tid & 1) * 4;
            xs[f * kFwdXs + r] = xq.x;
            xs[(f + 1) * kFwdXs + r] = xq.y;
            xs[(f + 2) * kFwdXs + r] = xq.z;
            xs[(f + 3) * kFwdXs + r] = xq.w;
            fetch_quad(tile + gridDim.x);
        } else {
            for (uint32_t i = tid; i < kFwdRows * F; i += kFwdThreads) {
                const uint32_t r = i / F, f = i - r * F;
                xs[f * kFwdXs + r] = r0 + r < n ? X[r0 * F + i] : 0.f;
            }
        }
        __syncthreads();
        const uint32_t p = tid & 63, cq = tid >> 6;
        for (uint32_t kc = 0; kc < chunks; ++kc) {
            const uint32_t cw = min(64u, H - kc * 64);
            if (kc > 0 && !scalar) {   // the chunk's buffers: free once the last chunk's MMAs have read them
                ok = mbar_wait_bounded(&mma_bar, parity, err);
                parity ^= 1;
                if (__syncthreads_or(!ok)) {
                    ok = false;
                    break;
                }
            }
#pragma unroll
            for (uint32_t g = 0; g < 2; ++g) {
                const uint32_t jc = cq * 16 + g * 8;   // column of the chunk
                if (jc >= cw) break;
                const uint32_t j0 = kc * 64 + jc;
                uint64_t zz[2][4];   // rows p and p + 64, two units each
                {
                    const ulonglong2 ba = *reinterpret_cast<const ulonglong2 *>(b1s + j0);
                    const ulonglong2 bb = *reinterpret_cast<const ulonglong2 *>(b1s + j0 + 4);
                    zz[0][0] = zz[1][0] = ba.x;
                    zz[0][1] = zz[1][1] = ba.y;
                    zz[0][2] = zz[1][2] = bb.x;
                    zz[0][3] = zz[1][3] = bb.y;
                }
#pragma unroll 4
                for (uint32_t f = 0; f < F; ++f) {
                    const ulonglong2 wa = *reinterpret_cast<const ulonglong2 *>(w1s + f * H + j0);
                    const ulonglong2 wb = *reinterpret_cast<const ulonglong2 *>(w1s + f * H + j0 + 4);
                    const uint64_t w[4] = {wa.x, wa.y, wb.x, wb.y};
                    const float x0 = xs[f * kFwdXs + p], x1 = xs[f * kFwdXs + p + 64];
                    const uint64_t xx0 = pack2(x0, x0), xx1 = pack2(x1, x1);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        zz[0][q] = fma2(w[q], xx0, zz[0][q]);
                        zz[1][q] = fma2(w[q], xx1, zz[1][q]);
                    }
                }
                float z[2][8];
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int q = 0; q < 4; ++q) unpack2(zz[e][q], z[e][2 * q], z[e][2 * q + 1]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint64_t row = r0 + p + 64 * e;
                    if (Z1 && row < n) {
                        float *dst = Z1 + row * H + j0;
                        if (vec) {
                            *reinterpret_cast<float4 *>(dst) = make_float4(z[e][0], z[e][1], z[e][2], z[e][3]);
                            *reinterpret_cast<float4 *>(dst + 4) = make_float4(z[e][4], z[e][5], z[e][6], z[e][7]);
                        } else {
#pragma unroll
                            for (int q = 0; q < 8; ++q) dst[q] = z[e][q];
                        }
                    }
                    float h[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) h[q] = fmaxf(z[e][q], 0.f);
                    store_parts(a, p + 64 * e, jc >> 3, h);
                }
            }
            if (scalar) continue;
            if (!lay.w2_resident) load_w2_chunk(sm, W2, H, kc, w2_aligned);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
                const uint32_t a0 = smem_addr(a), w0 = smem_addr(sm) + (lay.w2_resident ? kc * H * 128 : 0u);
                for (uint32_t k = 0; k < cw / 16; ++k) {
                    const uint64_t bd = smem_desc_sw128(w0 + k * 32);
                    const uint32_t acc = (kc | k) ? 1u : 0u;
                    mma_bf16(d_top, smem_desc_sw128(a0 + k * 32), bd, idesc, acc);
                    mma_bf16(d_low, smem_desc_sw128(a0 + kFwdPart + k * 32), bd, idesc, acc);
                    mma_bf16(d_low, smem_desc_sw128(a0 + 2 * kFwdPart + k * 32), bd, idesc, 1u);
                }
                tc_commit(&mma_bar);
            }
        }
        if (!ok) break;
        if (!scalar) {
            ok = mbar_wait_bounded(&mma_bar, parity, err);
            parity ^= 1;
        }
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        tc_fence_after();
        // layer 3: warp w reads the 32 rows of TMEM quadrant w % 4, columns half w / 4
        const uint32_t row_l = (warp & 3) * 32 + lane, half = warp >> 2, c0 = half * (H / 2);
        const uint64_t row = r0 + row_l;
        uint64_t s[2] = {0, 0};   // four sums
        for (uint32_t c = c0; c < c0 + H / 2; c += 16) {
            float z[16];
            if (!scalar) {
                uint32_t t[16], l[16];
                const uint32_t lanes = ((warp & 3) * 32) << 16;
                tmem_ld16(d_top + lanes + c, t);
                tmem_ld16(d_low + lanes + c, l);
                tmem_wait_ld(t, l);
#pragma unroll
                for (int q = 0; q < 16; q += 2)
                    unpack2(add2(pack2(__uint_as_float(t[q]), __uint_as_float(t[q + 1])),
                                 pack2(__uint_as_float(l[q]), __uint_as_float(l[q + 1]))),
                            z[q], z[q + 1]);
            } else {
                // non-finite weights: the plain sum, so that they meet the whole activation
#pragma unroll 1
                for (int q = 0; q < 16; ++q) {
                    float acc = 0.f;
                    for (uint32_t i = 0; i < H; ++i) {
                        float z1 = b1s[i];
                        for (uint32_t f = 0; f < F; ++f) z1 = fmaf(w1s[f * H + i], xs[f * kFwdXs + row_l], z1);
                        acc = fmaf(bf2f(W2[(size_t)(c + q) * H + i]), fmaxf(z1, 0.f), acc);
                    }
                    z[q] = acc;
                }
            }
#pragma unroll
            for (int q = 0; q < 16; q += 4) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(b2s + c + q);
                const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(w3s + c + q);
                unpack2(add2(pack2(z[q], z[q + 1]), b.x), z[q], z[q + 1]);
                unpack2(add2(pack2(z[q + 2], z[q + 3]), b.y), z[q + 2], z[q + 3]);
                s[0] = fma2(w.x, pack2(fmaxf(z[q], 0.f), fmaxf(z[q + 1], 0.f)), s[0]);
                s[1] = fma2(w.y, pack2(fmaxf(z[q + 2], 0.f), fmaxf(z[q + 3], 0.f)), s[1]);
            }
            if (Z2 && row < n) {
                float *dst = Z2 + row * H + c;
                if (vec) {
#pragma unroll
                    for (int q = 0; q < 16; q += 4)
                        *reinterpret_cast<float4 *>(dst + q) = make_float4(z[q], z[q + 1], z[q + 2], z[q + 3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 16; ++q) dst[q] = z[q];
                }
            }
        }
        float s0, s1, s2, s3;
        unpack2(s[0], s0, s1);
        unpack2(s[1], s2, s3);
        red[half * kFwdRows + row_l] = (s0 + s1) + (s2 + s3);
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid < kFwdRows && r0 + tid < n) {
            const float v = bias3 + (red[tid] + red[kFwdRows + tid]);
            P[r0 + tid] = 1.f / (1.f + expf(-v));
        }
    }
    if (!ok) mbar_wait_bounded(&mma_bar, parity ^ 1, err);   // MMAs in flight still read shared memory
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(d_top, tm_cols);
    }
}

// ---------------------------------------------------------------- backward
// Gradients of the (weighted) binary cross-entropy, added into the given
// buffers with fp32 atomics; loss gets the summed weighted BCE.
//
// blockIdx.x owns a run of row batches (32 rows each) and sums its gradients in
// registers, so each gradient gets one atomic per CTA; blockIdx.y is a role:
//   y < nb * nb    dW2 block (y / nb, y % nb) of T x T: sum over rows of
//                  dz2[r][j] h1[r][i], (T / 16)^2 sums per thread; the blocks of
//                  the first column also sum dw3 and db2, the first also db3 and
//                  the loss
//   y >= nb * nb   hidden block y - nb * nb of layer 1: dh1 = dz2 W2 for 32
//                  rows, then dW1 and db1
// (T = 64 for H <= 64, else 128; nb = ceil(H / T).)  The dW2 atomics are
// 16-byte vectors of consecutive columns, so a warp's instruction covers whole
// sectors.
// Bound: latency (one batch of rows a CTA), so every load of a batch is in flight at
// once; loads in loops of four and weights two bytes at a time took 35 us at 4,096
// rows and H = 128, now 23.
// Measured (4,096 rows, H = 128, forward, backward and their fills): 68 to 77 us a
// call, of which 46 on the device, against 145 us with 256 CTAs whose threads each
// added single dW2 columns 512 bytes apart.  Error against float64, 24 draws each of 500 to
// 20,000 rows and H = 64 to 256: weight gradients 2e-7 to 6e-7 of their norm, before 2e-7 to
// 7e-7; the loss 6e-8 to 1.3e-7, before 3e-7 to 1.8e-6.
constexpr int kBwdRows = 32;
constexpr int kBwdThreads = 256;

struct BwdArgs {
    const float *X;
    uint32_t n, F, H, batches;
    const uint16_t *W2, *w3;
    const float *Z1, *Z2, *P, *Y, *WT;
    float scale;
    float *dW1, *db1, *dW2, *db2, *dw3, *db3, *loss;
    uint32_t vec;   // dW2 allows 16-byte accesses
};

__device__ __forceinline__ void red_add4(float *p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// dz3 of 32 rows (threads 0..31); returns this row's loss term.
__device__ __forceinline__ float bwd_dz3(const BwdArgs &g, uint64_t r, float *dz3) {
    float d = 0.f, l = 0.f;
    if (r < g.n) {
        const float wt = g.WT ? g.WT[r] : 1.f;
        const float p = g.P[r], y = g.Y[r];
        d = g.scale * wt * (p - y);
        const float pc = fminf(fmaxf(p, 1e-7f), 1.f - 1e-7f);
        l = -g.scale * wt * (y * logf(pc) + (1.f - y) * logf(1.f - pc));
    }
    dz3[threadIdx.x] = d;
    return l;
}

// KF: dW1 sums per thread in the layer-1 role (F <= KF * kBwdThreads / T)
template <int T, int KF> __global__ void __launch_bounds__(kBwdThreads) mlp_bwd_kernel(BwdArgs g) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float dz3[kBwdRows];
    const uint32_t tid = threadIdx.x, H = g.H, nb = (H + T - 1) / T;
    constexpr uint32_t kCols = kBwdThreads / T;   // threads sharing a column
    constexpr uint32_t kMine = kBwdRows / kCols;  // rows of a batch per thread
    const uint32_t col = tid % T, part = tid / T;
    float *dz2 = sm;   // [32][T]
    if (blockIdx.y < nb * nb) {
        const uint32_t bj = blockIdx.y / nb, bi = blockIdx.y - bj * nb;
        float *h1 = sm + kBwdRows * T;   // [32][T]
        const uint32_t j = bj * T + col, i = bi * T + col;
        const float wj3 = j < H ? bf2f(g.w3[j]) : 0.f;
        const uint32_t ty = tid >> 4, tx = tid & 15;
        constexpr int M = T / 64;   // 4 x 4 sub-blocks per direction
        float acc[4 * M][4 * M];
#pragma unroll
        for (int x = 0; x < 4 * M; ++x)
#pragma unroll
            for (int y = 0; y < 4 * M; ++y) acc[x][y] = 0.f;
        float gw3 = 0.f, gb2 = 0.f, gb3 = 0.f, loss = 0.f;
        for (uint32_t b = blockIdx.x; b < g.batches; b += gridDim.x) {
            const uint64_t r0 = (uint64_t)b * kBwdRows;
            float z1s[kMine], z2s[kMine];   // this thread's rows of its column, all on their way at once
#pragma unroll
            for (uint32_t m = 0; m < kMine; ++m) {
                const uint64_t row = r0 + part + m * kCols;
                z2s[m] = row < g.n && j < H ? g.Z2[row * H + j] : 0.f;
                z1s[m] = row < g.n && i < H ? g.Z1[row * H + i] : 0.f;
            }
            __syncthreads();
            if (tid < kBwdRows) {
                loss += bwd_dz3(g, r0 + tid, dz3);
                gb3 += dz3[tid];
            }
            __syncthreads();
#pragma unroll
            for (uint32_t m = 0; m < kMine; ++m) {
                const uint32_t r = part + m * kCols;
                const float z1 = z1s[m], z2 = z2s[m];
                const float d = dz3[r];
                const float g2 = z2 > 0.f ? d * wj3 : 0.f;
                gw3 = fmaf(d, fmaxf(z2, 0.f), gw3);
                gb2 += g2;
                dz2[r * T + col] = g2;
                h1[r * T + col] = fmaxf(z1, 0.f);
            }
            __syncthreads();
#pragma unroll 4
            for (int r = 0; r < kBwdRows; ++r) {
                float u[4 * M], v[4 * M];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float4 p = *reinterpret_cast<const float4 *>(dz2 + r * T + m * 64 + ty * 4);
                    const float4 q = *reinterpret_cast<const float4 *>(h1 + r * T + m * 64 + tx * 4);
                    u[4 * m] = p.x, u[4 * m + 1] = p.y, u[4 * m + 2] = p.z, u[4 * m + 3] = p.w;
                    v[4 * m] = q.x, v[4 * m + 1] = q.y, v[4 * m + 2] = q.z, v[4 * m + 3] = q.w;
                }
#pragma unroll
                for (int x = 0; x < 4 * M; ++x)
#pragma unroll
                    for (int y = 0; y < 4 * M; ++y) acc[x][y] = fmaf(u[x], v[y], acc[x][y]);
            }
        }
#pragma unroll
        for (int x = 0; x < 4 * M; ++x) {
            const uint32_t jj = bj * T + (x >> 2) * 64 + ty * 4 + (x & 3);
            if (jj >= H) continue;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const uint32_t ii = bi * T + m * 64 + tx * 4;
                if (ii >= H) continue;   // H is a multiple of 32: whole groups of four
                float *dst = g.dW2 + (size_t)jj * H + ii;
                if (g.vec) {
                    red_add4(dst, acc[x][4 * m], acc[x][4 * m + 1], acc[x][4 * m + 2], acc[x][4 * m + 3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) atomicAdd(dst + q, acc[x][4 * m + q]);
                }
            }
        }
        if (bi == 0 && j < H) {
            atomicAdd(&g.dw3[j], gw3);
            atomicAdd(&g.db2[j], gb2);
        }
        if (blockIdx.y == 0 && tid < 32) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
                loss += __shfl_xor_sync(0xffffffffu, loss, o);
            }
            if (tid == 0) {
                atomicAdd(g.db3, gb3);
                atomicAdd(g.loss, loss);
            }
        }
        return;
    }
    // ---- layer 1
    const uint32_t bi = blockIdx.y - nb * nb;
    float *w2 = sm + kBwdRows * T;          // [T (out)][T (in)] of the current output block
    float *xs = w2 + T * T;                 // [32][F]
    float *g1 = dz2;                        // [32][T], once dz2 has been read
    const bool w2_aligned = (reinterpret_cast<uintptr_t>(g.W2) & 15) == 0;
    constexpr int R = kBwdRows * T / kBwdThreads / 4;   // rows per thread, four columns each
    constexpr uint32_t kQuads = T / 4;
    const uint32_t iq = (tid % kQuads) * 4, rg = (tid / kQuads) * R;
    float gw[KF], gb1 = 0.f;
#pragma unroll
    for (int k = 0; k < KF; ++k) gw[k] = 0.f;
    for (uint32_t b = blockIdx.x; b < g.batches; b += gridDim.x) {
        const uint64_t r0 = (uint64_t)b * kBwdRows;
        float z1s[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t row = r0 + rg + r;
                const uint32_t i = bi * T + iq + q;
                z1s[r][q] = row < g.n && i < H ? g.Z1[row * H + i] : 0.f;
            }
        __syncthreads();
        if (tid < kBwdRows) bwd_dz3(g, r0 + tid, dz3);
        for (uint32_t k = tid; k < kBwdRows * g.F; k += kBwdThreads)
            xs[k] = r0 + k / g.F < g.n ? g.X[r0 * g.F + k] : 0.f;
        float acc[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[r][q] = 0.f;
        for (uint32_t bj = 0; bj < nb; ++bj) {
            const uint32_t j = bj * T + col;
            const float wj3 = j < H ? bf2f(g.w3[j]) : 0.f;
            float z2s[kMine];
#pragma unroll
            for (uint32_t m = 0; m < kMine; ++m) {
                const uint64_t row = r0 + part + m * kCols;
                z2s[m] = row < g.n && j < H ? g.Z2[row * H + j] : 0.f;
            }
            __syncthreads();
            if (nb > 1 || b == blockIdx.x) {
                constexpr uint32_t kPieces = T * T / 8 / kBwdThreads, kRow = T / 8;   // eight weights a piece
                uint4 w[kPieces];
#pragma unroll
                for (uint32_t x = 0; x < kPieces; ++x) {
                    const uint32_t at = tid + x * kBwdThreads, o = bj * T + at / kRow, i = bi * T + at % kRow * 8;
                    w[x] = o < H && i < H ? load_w8(g.W2 + (size_t)o * H + i, w2_aligned) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (uint32_t x = 0; x < kPieces; ++x) {
                    const uint32_t v[4] = {w[x].x, w[x].y, w[x].z, w[x].w};
                    float *dst = w2 + (size_t)(tid + x * kBwdThreads) * 8;
#pragma unroll
                    for (int q = 0; q < 4; q += 2)
                        *reinterpret_cast<float4 *>(dst + 2 * q) =
                            make_float4(__uint_as_float(v[q] << 16), __uint_as_float(v[q] & 0xffff0000u),
                                        __uint_as_float(v[q + 1] << 16), __uint_as_float(v[q + 1] & 0xffff0000u));
                }
            }
#pragma unroll
            for (uint32_t m = 0; m < kMine; ++m) {
                const uint32_t r = part + m * kCols;
                dz2[r * T + col] = z2s[m] > 0.f ? dz3[r] * wj3 : 0.f;
            }
            __syncthreads();
            // every column of a padded block is zero on the dz2 side
#pragma unroll 2
            for (int k = 0; k < T; k += 4) {
                float4 w[4], d[R];
#pragma unroll
                for (int e = 0; e < 4; ++e) w[e] = *reinterpret_cast<const float4 *>(w2 + (k + e) * T + iq);
#pragma unroll
                for (int r = 0; r < R; ++r) d[r] = *reinterpret_cast<const float4 *>(dz2 + (rg + r) * T + k);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float dv[4] = {d[r].x, d[r].y, d[r].z, d[r].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        acc[r][0] = fmaf(dv[e], w[e].x, acc[r][0]);
                        acc[r][1] = fmaf(dv[e], w[e].y, acc[r][1]);
                        acc[r][2] = fmaf(dv[e], w[e].z, acc[r][2]);
                        acc[r][3] = fmaf(dv[e], w[e].w, acc[r][3]);
                    }
                }
            }
        }
        __syncthreads();
        // the ReLU of layer 1
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < 4; ++q) g1[(rg + r) * T + iq + q] = z1s[r][q] > 0.f ? acc[r][q] : 0.f;
        __syncthreads();
#pragma unroll 4
        for (int r = 0; r < kBwdRows; ++r) {
            const float v = g1[r * T + col];
            if (part == 0) gb1 += v;
#pragma unroll
            for (int k = 0; k < KF; ++k) {
                const uint32_t f = part + k * kCols;
                if (f < g.F) gw[k] = fmaf(v, xs[r * g.F + f], gw[k]);
            }
        }
    }
    const uint32_t i = bi * T + col;
    if (i >= H) return;
    if (part == 0) atomicAdd(&g.db1[i], gb1);
#pragma unroll
    for (int k = 0; k < KF; ++k) {
        const uint32_t f = part + k * kCols;
        if (f < g.F) atomicAdd(&g.dW1[(size_t)i * g.F + f], gw[k]);
    }
}

// Adam on fp32 master weights; refreshes the bf16 copy (round to nearest even).
__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, uint16_t *__restrict__ p16, uint32_t n, float lr, float beta1,
                            float beta2, float eps, float bc1, float bc2, float wd) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i] + wd * p[i];
        const float mi = beta1 * m[i] + (1.f - beta1) * gi;
        const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
        p[i] = pi;
        if (p16) p16[i] = __bfloat16_as_ushort(__float2bfloat16_rn(pi));
    }
}

void launch_mlp_forward(const float *X, uint32_t n, uint32_t F, uint32_t H, const uint16_t *W1, const float *b1,
                        const uint16_t *W2, const float *b2, const uint16_t *w3, const float *b3, float *Z1,
                        float *Z2, float *P, uint32_t *dev_err, cudaStream_t st, int n_sm) {
    if (n == 0) return;
    // the whole W2 in shared memory when it fits beside the rest, else one K chunk at a time
    FwdLayout lay = mlp_fwd_layout(F, H, true);
    if (lay.bytes > 226 * 1024) lay = mlp_fwd_layout(F, H, false);
    uint32_t cols = 32;
    while (cols < 2 * H) cols *= 2;
    const uint32_t per_sm = cols <= 256 && lay.bytes <= 112 * 1024 ? 2u : 1u;
    const uint32_t tiles = n / kFwdRows + (n % kFwdRows != 0);
    const uint32_t vec = ((reinterpret_cast<uintptr_t>(Z1) | reinterpret_cast<uintptr_t>(Z2)) & 15) == 0;
    SG_CUDA_TRY(cudaFuncSetAttribute(mlp_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.bytes));
    mlp_fwd_kernel<<<std::min(tiles, (uint32_t)n_sm * per_sm), kFwdThreads, lay.bytes, st>>>(
        X, n, F, H, W1, b1, W2, b2, w3, b3, Z1, Z2, P, lay, cols, vec, dev_err);
    SG_CUDA_TRY(cudaGetLastError());
}

template <int T, int KF> static void launch_bwd(const BwdArgs &g, int n_sm, cudaStream_t st) {
    const uint32_t nb = (g.H + T - 1) / T, roles = nb * nb + nb;
    const size_t smem = (size_t)std::max(2 * kBwdRows * T, kBwdRows * T + T * T + kBwdRows * (int)g.F) * 4;
    SG_CUDA_TRY(cudaFuncSetAttribute(mlp_bwd_kernel<T, KF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint32_t x = std::max(1u, std::min(g.batches, 2u * (uint32_t)n_sm / roles));
    mlp_bwd_kernel<T, KF><<<dim3(x, roles), kBwdThreads, smem, st>>>(g);
    SG_CUDA_TRY(cudaGetLastError());
}

}  // namespace sg

using namespace sg;

namespace {
bool mlp_shape_ok(uint32_t F, uint32_t H) { return F >= 1 && F <= kMlpMaxIn && H >= 32 && H <= 256 && H % 32 == 0; }
}  // namespace

extern "C" {

int sgfim_mlp_forward(sgfim_handle *h, const float *X, uint32_t n, uint32_t in_dim, uint32_t hidden,
                      const uint16_t *W1, const float *b1, const uint16_t *W2, const float *b2, const uint16_t *w3,
                      const float *b3, float *Z1, float *Z2, float *P, void *stream) {
    if (!h || (n && (!X || !P)) || !W1 || !b1 || !W2 || !b2 || !w3 || !b3)
        return fail(h, SGFIM_EINVAL, "null argument");
    if (!mlp_shape_ok(in_dim, hidden)) return fail(h, SGFIM_EINVAL, "mlp shape: in_dim 1..64, hidden 32..256 step 32");
    try {
        cudaSetDevice(h->device);
        launch_mlp_forward(X, n, in_dim, hidden, W1, b1, W2, b2, w3, b3, Z1, Z2, P,
                           h->dev_err.as<uint32_t>(), stream ? (cudaStream_t)stream : (cudaStream_t)0, h->n_sm);
        h->launches++;
        return SGFIM_OK;
    } catch (const CudaError &e) {
        return fail(h, SGFIM_EDEVICE, e.what);
    }
}

int sgfim_mlp_backward(sgfim_handle *h, const float *X, uint32_t n, uint32_t in_dim, uint32_t hidden,
                       const uint16_t *W2, const uint16_t *w3, const float *Z1, const float *Z2, const float *P,
                       const float *Y, const float *WT, float scale, float *dW1, float *db1, float *dW2, float *db2,
                       float *dw3, float *db3, float *loss, void *stream) {
    if (!h || (n && (!X || !Z1 || !Z2 || !P || !Y)) || !W2 || !w3 || !dW1 || !db1 || !dW2 || !db2 || !dw3 || !db3 ||
        !loss)
        return fail(h, SGFIM_EINVAL, "null argument");
    if (!mlp_shape_ok(in_dim, hidden)) return fail(h, SGFIM_EINVAL, "mlp shape: in_dim 1..64, hidden 32..256 step 32");
    try {
        cudaSetDevice(h->device);
        if (n == 0) return SGFIM_OK;
        cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)0;
        const BwdArgs g{X, n, in_dim, hidden, n / kBwdRows + (n % kBwdRows != 0), W2, w3, Z1, Z2, P, Y, WT, scale,
                        dW1, db1, dW2, db2, dw3, db3, loss, (reinterpret_cast<uintptr_t>(dW2) & 15) == 0};
        if (hidden <= 64) {
            if (in_dim <= 8) launch_bwd<64, 2>(g, h->n_sm, st);
            else launch_bwd<64, 16>(g, h->n_sm, st);
        } else {
            if (in_dim <= 8) launch_bwd<128, 4>(g, h->n_sm, st);
            else launch_bwd<128, 32>(g, h->n_sm, st);
        }
        h->launches++;
        return SGFIM_OK;
    } catch (const CudaError &e) {
        return fail(h, SGFIM_EDEVICE, e.what);
    }
}

int sgfim_adam_step(sgfim_handle *h, float *param, const float *grad, float *m, float *v, uint16_t *param_bf16,
                    uint32_t n, float lr, float beta1, float beta2, float eps, uint32_t step, float weight_decay,
                    void *stream) {
    if (!h || !param || !grad || !m || !v || step == 0) return fail(h, SGFIM_EINVAL, "bad argument");
    try {
        cudaSetDevice(h->device);
        const float bc1 = 1.f - powf(beta1, (float)step), bc2 = 1.f - powf(beta2, (float)step);
        const unsigned blocks = std::min<unsigned>((n + 255) / 256, 1024);
        adam_kernel<<<blocks ? blocks : 1, 256, 0, stream ? (cudaStream_t)stream : (cudaStream_t)0>>>(
            param, grad, m, v, param_bf16, n, lr, beta1, beta2, eps, bc1, bc2, weight_decay);
        SG_CUDA_TRY(cudaGetLastError());
        h->launches++;
        return SGFIM_OK;
    } catch (const CudaError &e) {
        return fail(h, SGFIM_EDEVICE, e.what);
    }
}

}  // extern "C"
