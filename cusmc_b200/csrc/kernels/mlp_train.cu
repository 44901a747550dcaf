// Tensor-core (tcgen05) kernels of the proposal network: the forward pass
// over a row set, and the gradient of the CE objective
//     J = sum over rows of (b * theta - a * e^theta)
// with respect to every parameter, both with BF16 operands and FP32
// accumulation in tensor memory.
//
// One CTA of 512 threads (four warpgroups) walks row tiles of 128 rows.
// Thread (g, r), g = warpgroup, r = thread index within it, owns row r of
// the tile (TMEM lane r; warp w reads TMEM lanes 32 (w mod 4) ..) and columns
// 16 g .. 16 g + 15 of each 64-wide layer, so the CUDA-core epilogues (GELU,
// GELU', the BF16 repacking) are spread over 16 warps.  Per tile:
//   D1 = X  . W1^T          (M=128, N=64,  K=16)   first layer
//   D2 = H1 . W2^T          (M=128, N=64,  K=64)   second layer
//   D1 = dZ2 . W2           (M=128, N=64,  K=64)   back-propagation into layer 1
//   D4 += [dZ2 | dZ1]^T . [H1 | X | 1]   (M=128, N=96, K=128 rows)
// so D4 accumulates dW2^T, dW1^T and the bias gradients over every tile the
// CTA processes.  A row's theta is the sum of its four groups' partial dot
// products (exchanged through shared memory, added in group order); the
// GELU derivatives stay in the registers of the thread that computed them,
// and the output layer's gradient is accumulated per thread in registers
// and reduced once at the end in a fixed order (the gradient is
// deterministic).
//
// Operands live in shared memory without swizzle, in core matrices of 8 rows
// x 16 bytes: tile F = [H1 | X | 1] and tile Z = [dZ2 | dZ1], 128 rows each,
// core matrix (row group g, column chunk c) at (16 c + g) * 128 bytes.  The
// layer MMAs read them K-major (columns are the contraction); the weight-
// gradient MMA contracts over the rows and reads the same bytes MN-major, so
// no transposed copy exists: a thread stores its sixteen columns of a layer as
// two 16-byte words, rows next to each other.  F is double-buffered: the
// weight-gradient MMA of a tile overlaps the next tile's first layer.
//
// One thread issues the MMAs, completion is signalled through an mbarrier
// (the weight-gradient MMA's with the next tile's first), and every wait is
// bounded: on a timeout the kernel records an error, skips its further waits,
// waits (bounded) for its MMAs, frees its tensor memory and returns.
//
// What bounds it: the CUDA-core epilogues (two GELUs with their derivatives
// per hidden unit and row); the tensor pipe is nearly idle.  Measured (B200):
// 1e6 rows 613 us with transposed operand copies stored 2 bytes at a time
// (2,830 instructions per warp and tile), 269 us in this form (1,515; issue
// slots 69 % busy).
#include "../include/csmc_mlp.h"
#include "sim.cuh"

#include <cuda_runtime.h>

namespace csmc {
namespace {

constexpr int kRows = 128;                      // rows per tile
constexpr int kGroups = 4;                      // warpgroups per CTA
constexpr int kThreads = 128 * kGroups;
constexpr int kCols = CSMC_MLP_HID / kGroups;   // layer columns per thread (16)
constexpr uint32_t kTmemCols = 256;             // D1/D3 [0,64), D2 [64,128), D4 [128,224)
constexpr uint32_t kColD1 = 0, kColD2 = 64, kColD4 = 128;
constexpr int kN4 = 96;                         // [H1 (64) | X (16) | 1 | 0 x 15]

constexpr int kPartial = 128 * kN4 + 68;        // floats of a CTA's partials: D4, dw3, db3, padded to 16 bytes

// shared-memory carve-up (bytes)
constexpr uint32_t kChunk = 128 * 16;           // one column chunk: 8 columns of 128 rows
constexpr uint32_t kFBytes = (kN4 / 8) * kChunk;
constexpr uint32_t kF = 0;                      // F tiles, two buffers: chunks 0..7 H1, 8..9 X, 10..11 [1 | 0]
constexpr uint32_t kX = 8 * kChunk;             // X within F
constexpr uint32_t kZ = kF + 2 * kFBytes;       // Z tile: chunks 0..7 dZ2, 8..15 dZ1
constexpr uint32_t kB1 = kZ + 16 * kChunk;      // W1          64 x 16
constexpr uint32_t kB2 = kB1 + 64 * 16 * 2;     // W2          64 x 64 (out x in)
constexpr uint32_t kTh = kB2 + 64 * 64 * 2;     // theta partials [group][row] (floats)
constexpr uint32_t kMisc = kTh + kGroups * 128 * 4;  // mbarrier, tmem address, biases, reductions
constexpr uint32_t kMiscBytes = 4096;
constexpr uint32_t kRedStride = 17;             // per-warp output-layer sums: 16 columns, db3
constexpr uint32_t kSmemBytes = 160 * 1024;     // the carve-up takes 102 KB; more than half an SM's: one CTA per SM
static_assert(kMisc + kMiscBytes <= kSmemBytes, "shared-memory carve-up");
static_assert(1536 + 16 * kRedStride * 4 <= kMiscBytes, "reduction slots");

constexpr uint32_t kWaitLimit = 1u << 20;       // bounded mbarrier polls

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// byte offset of element (r, k) in a K-major no-swizzle tile of R rows
__device__ __forceinline__ uint32_t kmaj(uint32_t r, uint32_t k, uint32_t R) {
    return (((k >> 3) * (R >> 3) + (r >> 3)) << 7) + ((r & 7u) << 4) + ((k & 7u) << 1);
}

// shared-memory matrix descriptor: start, leading (K) and stride (row
// group) byte offsets, version 1, no swizzle
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | (static_cast<uint64_t>((lbo >> 4) & 0x3fffu) << 16) |
           (static_cast<uint64_t>((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// instruction descriptor: FP32 accumulator, BF16 A and B, M=128; each operand
// K-major or MN-major
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t N, bool a_mn = false, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) | ((N >> 3) << 17) |
           ((128u >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    const uint32_t z = 0;  // no output lane disabled
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(z));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Two floats rounded to BF16 (to nearest even), the first in the low half.
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Stores this thread's sixteen columns (chunks c and c + 1) of row r.
__device__ __forceinline__ void st_cols(uint8_t *tile, uint32_t c, uint32_t r, const float *v) {
    uint4 *o = reinterpret_cast<uint4 *>(tile + c * kChunk + r * 16u);
    o[0] = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
    o[kChunk / 16] = make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]), pack2(v[14], v[15]));
}

// mode 0: forward only (clipped theta per row into theta_out); mode 1:
// gradient partials per CTA: D4 (128 x 96 floats: row m = output neuron of
// [layer 2 | layer 1], column n = input [h1 | x | 1 | 0]), dw3 (64), db3, 0.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
    mlp_tc_kernel(const MlpRow *rows, uint64_t n_rows, const MlpParams *P, float *theta_out, float *partials,
                  double *objective, int *error) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t grp = tid >> 7, r = tid & 127u;  // warpgroup, row within the tile
    const uint32_t c0 = grp * kCols;                // this thread's first layer column
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sm + kMisc);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(sm + kMisc + 8);
    float *b1s = reinterpret_cast<float *>(sm + kMisc + 512);
    float *b2s = reinterpret_cast<float *>(sm + kMisc + 768);
    float *w3s = reinterpret_cast<float *>(sm + kMisc + 1024);
    float *red = reinterpret_cast<float *>(sm + kMisc + 1536);  // [warp][kRedStride]
    float *thp = reinterpret_cast<float *>(sm + kTh);           // [group][row]
    const uint32_t mbar_a = smem_u32(mbar);

    // ---- constant operands: W1 (B1), W2 (B2; read MN-major as W2^T in the
    // back-propagation), eight inputs of a unit at a time, the ones columns
    if (tid < 128) {
        const uint32_t o = tid >> 1, c = tid & 1u;
        *reinterpret_cast<uint4 *>(sm + kB1 + kmaj(o, 8u * c, 64)) = reinterpret_cast<const uint4 *>(&P->w1[0][0])[tid];
    }
    *reinterpret_cast<uint4 *>(sm + kB2 + kmaj(tid >> 3, 8u * (tid & 7u), 64)) =
        reinterpret_cast<const uint4 *>(&P->w2[0][0])[tid];
    static_assert(kThreads == CSMC_MLP_HID * CSMC_MLP_HID / 8, "one 16-byte word of W2 per thread");
    {  // chunks 10 and 11 of both F buffers: the ones column, then zeros
        uint8_t *f = sm + kF + (grp >> 1) * kFBytes + (10u + (grp & 1u)) * kChunk + r * 16u;
        *reinterpret_cast<uint4 *>(f) = make_uint4((grp & 1u) ? 0u : 0x3f80u, 0u, 0u, 0u);
    }
    if (tid < 64) {
        b1s[tid] = P->b1[tid];
        b2s[tid] = P->b2[tid];
        w3s[tid] = P->w3[tid];
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_a));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tmem_holder;
    const uint32_t lane_base = ((warp & 3u) * 32u) << 16;  // this warp's TMEM lanes (rows)
    const float b3 = P->b3;
    double J = 0.0;
    float dw3[kCols];  // this thread's rows' g * h2 for its columns, over all tiles
#pragma unroll
    for (int i = 0; i < kCols; ++i) dw3[i] = 0.0f;
    float db3 = 0.0f;
    uint32_t phase = 0, buf = 0;
    bool ok = true, first = true;
    // a wait that gave up leaves ok false: no further waits
    auto wait_mma = [&]() {
        if (ok) ok = mbar_wait(mbar_a, phase);
        phase ^= 1u;
        tc_after_sync();
    };

    // the row's four features of this group and its a, b, one tile ahead
    const uint64_t tiles = (n_rows + kRows - 1) / kRows;
    uint32_t xf[2] = {0u, 0u};
    float ra = 0.0f, rb = 0.0f;
    auto load_row = [&](uint64_t tile) {
        const uint64_t i = tile * kRows + r;
        xf[0] = xf[1] = 0u;
        ra = rb = 0.0f;
        if (tile < tiles && i < n_rows) {
            const uint32_t *w = reinterpret_cast<const uint32_t *>(rows + i);
            xf[0] = w[2 * grp];
            xf[1] = w[2 * grp + 1];
            ra = __uint_as_float(w[8]);
            rb = __uint_as_float(w[9]);
        }
    };
    load_row(blockIdx.x);
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t row_i = tile * kRows + r;
        const bool valid = row_i < n_rows;
        uint8_t *const F = sm + kF + buf * kFBytes;
        buf ^= 1u;
        const float row_a = ra, row_b = rb;
        // each group stores four of the row's sixteen features
        *reinterpret_cast<uint2 *>(F + kX + (grp >> 1) * kChunk + r * 16u + (grp & 1u) * 8u) = make_uint2(xf[0], xf[1]);
        load_row(tile + gridDim.x);
        fence_async_smem();
        tc_before_sync();
        __syncthreads();
        // ---- layer 1
        if (tid == 0) {
            tc_after_sync();
            mma_bf16(tmem + kColD1, sdesc(smem_u32(F + kX), kChunk, 128), sdesc(smem_u32(sm + kB1), 1024, 128),
                     idesc_bf16(64), 0);
            mma_commit(mbar_a);  // and the previous tile's weight-gradient MMAs
        }
        wait_mma();
        float dg1[kCols];  // GELU'(z1) of this thread's columns
        {
            float z[16];
            tmem_ld16(tmem + lane_base + kColD1 + c0, z);
#pragma unroll
            for (int i = 0; i < kCols; ++i) {
                float gv;
                gelu_both(f_add(z[i], b1s[c0 + i]), gv, dg1[i]);
                z[i] = gv;
            }
            st_cols(F, 2u * grp, r, z);
        }
        fence_async_smem();
        tc_before_sync();
        __syncthreads();
        // ---- layer 2
        if (tid == 0) {
            tc_after_sync();
#pragma unroll
            for (uint32_t kk = 0; kk < 4; ++kk)
                mma_bf16(tmem + kColD2, sdesc(smem_u32(F + kk * 2 * kChunk), kChunk, 128),
                         sdesc(smem_u32(sm + kB2 + kk * 2048), 1024, 128), idesc_bf16(64), kk > 0);
            mma_commit(mbar_a);
        }
        wait_mma();
        float h2[kCols], dg2[kCols];
        {
            float z2[16];
            tmem_ld16(tmem + lane_base + kColD2 + c0, z2);
            float part = 0.0f;
#pragma unroll
            for (int i = 0; i < kCols; ++i) {
                gelu_both(f_add(z2[i], b2s[c0 + i]), h2[i], dg2[i]);
                part = f_fma(h2[i], w3s[c0 + i], part);
            }
            thp[grp * 128 + r] = part;
        }
        tc_before_sync();
        __syncthreads();
        const float th = f_add(f_add(f_add(f_add(b3, thp[r]), thp[128 + r]), thp[256 + r]), thp[384 + r]);
        const bool inside = th >= -CSMC_MLP_THETA_MAX && th <= CSMC_MLP_THETA_MAX;
        const float thc = inside ? th : (th < 0.0f ? -CSMC_MLP_THETA_MAX : CSMC_MLP_THETA_MAX);
        if (MODE == 0) {
            if (valid && grp == 0) theta_out[row_i] = thc;
            continue;
        }
        const float e = exp2_f(f_mul(thc, 1.44269502f));
        if (valid && grp == 0) J += static_cast<double>(row_b) * thc - static_cast<double>(row_a) * e;
        const float g = (valid && inside) ? f_add(row_b, -f_mul(row_a, e)) : 0.0f;
        if (grp == 0) db3 = f_add(db3, g);
        {
            float dz[kCols];
#pragma unroll
            for (int i = 0; i < kCols; ++i) {
                dw3[i] = f_fma(g, h2[i], dw3[i]);
                dz[i] = f_mul(f_mul(g, w3s[c0 + i]), dg2[i]);
            }
            st_cols(sm + kZ, 2u * grp, r, dz);
        }
        fence_async_smem();
        tc_before_sync();
        __syncthreads();
        // ---- back-propagation into the first layer: dH1 = dZ2 . W2
        if (tid == 0) {
            tc_after_sync();
#pragma unroll
            for (uint32_t kk = 0; kk < 4; ++kk)
                mma_bf16(tmem + kColD1, sdesc(smem_u32(sm + kZ + kk * 2 * kChunk), kChunk, 128),
                         sdesc(smem_u32(sm + kB2 + kk * 256), 128, 1024), idesc_bf16(64, false, true), kk > 0);
            mma_commit(mbar_a);
        }
        wait_mma();
        {
            float dh[16];
            tmem_ld16(tmem + lane_base + kColD1 + c0, dh);
#pragma unroll
            for (int i = 0; i < kCols; ++i) dh[i] = f_mul(dh[i], dg1[i]);
            st_cols(sm + kZ, 8u + 2u * grp, r, dh);
        }
        fence_async_smem();
        tc_before_sync();
        __syncthreads();
        // ---- weight gradients: D4 += Z^T . F, sixteen rows at a time
        if (tid == 0) {
            tc_after_sync();
#pragma unroll
            for (uint32_t kk = 0; kk < 8; ++kk)
                mma_bf16(tmem + kColD4, sdesc(smem_u32(sm + kZ + kk * 256), 128, kChunk),
                         sdesc(smem_u32(F + kk * 256), 128, kChunk), idesc_bf16(kN4, true, true), (!first || kk > 0));
        }
        first = false;
    }
    if (MODE == 1 && !first) {  // the last tile's weight gradients
        if (tid == 0) mma_commit(mbar_a);
        wait_mma();
    }
    if (__syncthreads_or(ok ? 0 : 1)) {
        if (!ok && error) atomicExch(error, 1);
        // one more bounded wait for the MMAs still in flight before freeing
        (void)mbar_wait(mbar_a, phase ^ 1u);
        ok = false;
    }
    tc_after_sync();

    if (MODE == 1) {
        float *out = partials + static_cast<size_t>(blockIdx.x) * kPartial;
        if (grp < 3) {  // groups 0..2 read 32 of D4's 96 columns each
            if (ok && !first) {  // block-uniform
                float v[16];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t col = grp * 32u + 16u * c;
                    tmem_ld16(tmem + lane_base + kColD4 + col, v);
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        *reinterpret_cast<float4 *>(out + r * kN4 + col + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
            } else {
                for (int i = 0; i < 32; ++i) out[r * kN4 + grp * 32 + i] = 0.0f;
            }
        }
        // output layer: per warp, the sum over its 32 rows (butterfly), then
        // the four warps of a group in warp order
#pragma unroll
        for (int i = 0; i < kCols; ++i) {
            float v = dw3[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp * kRedStride + i] = v;
        }
        float vb = db3;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vb += __shfl_xor_sync(0xffffffffu, vb, o);
        if (lane == 0) red[warp * kRedStride + kCols] = vb;
        __syncthreads();
        if (tid < 64) {  // dw3[k]: group k / 16, its warps 4g .. 4g + 3
            const uint32_t gk = tid / kCols, i = tid % kCols;
            const float *rw = red + (4 * gk) * kRedStride + i;
            out[128 * kN4 + tid] =
                f_add(f_add(f_add(rw[0], rw[kRedStride]), rw[2 * kRedStride]), rw[3 * kRedStride]);
        }
        if (tid == 64)
            out[128 * kN4 + 64] = f_add(f_add(f_add(red[kCols], red[kRedStride + kCols]), red[2 * kRedStride + kCols]),
                                        red[3 * kRedStride + kCols]);
        if (tid == 65) out[128 * kN4 + 65] = 0.0f;
        __shared__ double jred[128];
        if (grp == 0) jred[r] = J;
        __syncthreads();
        if (tid == 0) {
            double sum = 0.0;
#pragma unroll 32
            for (int i = 0; i < 128; ++i) sum += jred[i];
            objective[blockIdx.x] = sum;
        }
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

}  // namespace

size_t mlp_tc_smem_bytes() { return kSmemBytes; }
int mlp_tc_partial_floats() { return kPartial; }

int mlp_tc_launch(int mode, const MlpRow *rows, uint64_t n_rows, const MlpParams *P, float *theta_out,
                  float *partials, double *objective, int *error, int grid, void *stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (mode == 0) {
        auto fn = mlp_tc_kernel<0>;
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return static_cast<int>(e);
        fn<<<grid, kThreads, kSmemBytes, st>>>(rows, n_rows, P, theta_out, partials, objective, error);
    } else {
        auto fn = mlp_tc_kernel<1>;
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return static_cast<int>(e);
        fn<<<grid, kThreads, kSmemBytes, st>>>(rows, n_rows, P, theta_out, partials, objective, error);
    }
    return static_cast<int>(cudaGetLastError());
}

}  // namespace csmc
