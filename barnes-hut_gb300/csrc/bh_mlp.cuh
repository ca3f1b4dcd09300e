// bh_mlp.cuh -- layout constants and tile helpers of the learned-correction MLP, shared by the
// standalone MLP kernels (bh_mlp.cu) and the fused correction kernels (bh_learned.cu).
#pragma once
#include <cuda_bf16.h>

#include "bh_internal.cuh"
#include "bh_pairs.cuh"
#include "bh_tc.cuh"

namespace bh {

constexpr int MLP_IN = 6, MLP_K0 = 16, MLP_H = 64, MLP_NO = 16, MLP_OUT = 2;
constexpr int P_W1 = 0, P_B1 = 1024, P_W2 = 1088, P_B2 = 5184, P_W3 = 5248, P_B3 = 9344,
              P_W4 = 9408, P_B4 = 10432, P_TOTAL = 10448;
// image byte offsets
constexpr int I_B1 = 0, I_B2 = 2048, I_B3 = 10240, I_B4 = 18432, I_FWD = 20480;
constexpr int I_B2T = 20480, I_B3T = 28672, I_B4T = 36864, I_TOTAL = 38912;
static_assert(P_TOTAL == MLP_PARAMS && I_TOTAL == MLP_IMAGE_BYTES, "MLP layout");

__device__ __forceinline__ uint16_t bf16_bits(float v) {
    __nv_bfloat16 b = __float2bfloat16_rn(v);
    return *reinterpret_cast<uint16_t *>(&b);
}

// Two values in one packed conversion, v0 in the low half: the same roundings as bf16_bits.  Single
// conversions run on the MUFU pipe, beside the tanh that bound the network's kernels: 1,000,003 rows
// forward 101 us with them, 70 with packed ones.
__device__ __forceinline__ uint32_t bf16x2_bits(float v0, float v1) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v1), "f"(v0));
    return r;
}

__device__ __forceinline__ void copy_bytes(uint8_t *dst, const uint8_t *src, int bytes) {
    for (int i = threadIdx.x * 16; i < bytes; i += blockDim.x * 16)
        *reinterpret_cast<uint4 *>(dst + i) = *reinterpret_cast<const uint4 *>(src + i);
}

// write the 16 BF16 values of row r of a K-major 128 x 16 tile (2 core columns)
__device__ __forceinline__ void store_row16(uint8_t *tile, int r, const float *v) {
#pragma unroll
    for (int c = 0; c < 2; c++) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            w[q] = bf16x2_bits(v[8 * c + 2 * q], v[8 * c + 2 * q + 1]);
        *reinterpret_cast<uint4 *>(tile + tc::kmajor_off(r, 8 * c, 2)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// write the 16 BF16 values v[0..15] to columns c0 .. c0 + 15 (c0 a multiple of 8) of row r of a
// K-major tile with kc core columns
__device__ __forceinline__ void store_cols16(uint8_t *tile, int r, int c0, int kc, const float *v) {
#pragma unroll
    for (int c = 0; c < 2; c++) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            w[q] = bf16x2_bits(v[8 * c + 2 * q], v[8 * c + 2 * q + 1]);
        *reinterpret_cast<uint4 *>(tile + tc::kmajor_off(r, c0 + 8 * c, kc)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// barrier over the n threads that use barrier `id`, and the same with the conjunction of p
__device__ __forceinline__ void group_sync(int id, int n) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ bool group_and(int id, int n, bool p) {
    uint32_t r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"(p ? 1u : 0u), "r"(id), "r"(n)
        : "memory");
    return r != 0;
}

// GELU (tanh form) of two values at once: tc::gelu_and_grad's arithmetic on the packed FP32 instructions,
// rounding by rounding (x fma(t, 1/2, 1/2) equals (x / 2)(1 + t): the halves are exact scalings),
// so an activation has the same bits whichever of the two computed it.  Seven FP32 operations and
// one MUFU operation per value; packing them halves the issue slots, which bound the scalar form.
__device__ __forceinline__ f2_t gelu2(f2_t x) {
    const f2_t c1 = f2_pack(tc::GELU_C1, tc::GELU_C1), c0 = f2_pack(tc::GELU_C0, tc::GELU_C0);
    const f2_t half = f2_pack(0.5f, 0.5f);
    const f2_t u = f2_mul(c0, f2_fma(f2_mul(f2_mul(c1, x), x), x, x));
    float u0, u1;
    f2_unpack(u, u0, u1);
    const f2_t t = f2_pack(tc::tanh_approx(u0), tc::tanh_approx(u1));
    return f2_mul(x, f2_fma(t, half, half));
}

__device__ __forceinline__ uint32_t bf16x2_bits(f2_t v) {
    float a, b;
    f2_unpack(v, a, b);
    return bf16x2_bits(a, b);
}

// Forward of one 128-row tile by a group of 128 threads (four consecutive warps, the first a
// multiple of four) that share barrier `bar`, one mbarrier, the tile buffer ACT (128 x 64 BF16) and
// 64 TMEM columns.  The caller has written the input rows to the first 4 KB of ACT (K-major
// 128 x 16); thread r of the group owns row r and receives its two outputs.  sW = forward images,
// bias = b1, b2, b3, b4 (208 floats, 16-byte aligned) in shared memory.  `ok` becomes false where a
// bounded tensor-core wait gave up (the outputs are then void); the group leaves together, before
// the next tile's first MMA, with the return value false.
//
// Bound: 192 tanh per row on the MUFU pipe (39 us for 1,000,003 rows), 1,344 FP32 operations and the
// issue slots, close to each other (a polynomial in the tanh's place for 3 of 8 columns: 70 -> 77 us);
// several groups per SM overlap one group's MMA round trips with the others' epilogues.
// The accumulator is read 32 columns at a time, which keeps a thread within 64 registers.
__device__ __forceinline__ bool mlp_group_forward(uint32_t sW, uint8_t *ACT, const float *bias, uint32_t tmem,
                                                  uint64_t *mbar, uint32_t &phase, int bar, bool &ok, float *y) {
    const int r = threadIdx.x & 127;
    const uint32_t sACT = tc::smem_u32(ACT), lane = (uint32_t)(threadIdx.x & 96) << 16;
    tc::fence_async_smem();
    tc::fence_before();
    if (!group_and(bar, 128, ok)) return false;
    if (r == 0) {
        tc::fence_after();
        tc::mma(tmem, tc::kdesc(sACT, 2, 0), tc::kdesc(sW + I_B1, 2, 0), tc::idesc_bf16(128, 64), 0);
        tc::commit(mbar);
    }
#pragma unroll 1
    for (int layer = 0; layer < 3; layer++) {
        ok = ok && tc::mbar_wait(mbar, phase);
        phase ^= 1u;
        tc::fence_after();
        const ulonglong2 *b2 = reinterpret_cast<const ulonglong2 *>(bias + 64 * layer);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float v[32];
            tc::ld16(tmem + lane + 32 * h, v);
            tc::ld16(tmem + lane + 32 * h + 16, v + 16);
            tc::ld_wait();
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const ulonglong2 b = b2[8 * h + 2 * c + q];
                    const float *x = v + 8 * c + 4 * q;
                    w[2 * q] = bf16x2_bits(gelu2(f2_add(f2_pack(x[0], x[1]), b.x)));
                    w[2 * q + 1] = bf16x2_bits(gelu2(f2_add(f2_pack(x[2], x[3]), b.y)));
                }
                *reinterpret_cast<uint4 *>(ACT + tc::kmajor_off(r, 32 * h + 8 * c, 8)) =
                    make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        const uint32_t wimg = sW + (layer == 0 ? I_B2 : layer == 1 ? I_B3 : I_B4);
        tc::fence_async_smem();
        tc::fence_before();
        group_sync(bar, 128);
        if (r == 0) {
            tc::fence_after();
            const uint32_t idesc = layer < 2 ? tc::idesc_bf16(128, 64) : tc::idesc_bf16(128, 16);
#pragma unroll
            for (int j = 0; j < 4; j++) tc::mma(tmem, tc::kdesc(sACT, 8, j), tc::kdesc(wimg, 8, j), idesc, j);
            tc::commit(mbar);
        }
    }
    ok = ok && tc::mbar_wait(mbar, phase);
    phase ^= 1u;
    tc::fence_after();
    float v[2];
    tc::ld2(tmem + lane, v);
    tc::ld_wait();
    y[0] = v[0] + bias[192];
    y[1] = v[1] + bias[193];
    tc::fence_before();  // the next tile's MMA overwrites the columns just read
    return true;
}

// write the 64 BF16 values of row r of a K-major 128 x 64 tile (8 core columns)
__device__ __forceinline__ void store_row64(uint8_t *tile, int r, const float *v) {
#pragma unroll
    for (int c = 0; c < 8; c++) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            w[q] = bf16x2_bits(v[8 * c + 2 * q], v[8 * c + 2 * q + 1]);
        *reinterpret_cast<uint4 *>(tile + tc::kmajor_off(r, 8 * c, 8)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
// load 64 accumulator columns of this thread's lane starting at column col
__device__ __forceinline__ void ld64(uint32_t tbase, int col, float *v) {
    const uint32_t lane = (uint32_t)(threadIdx.x & 96) << 16;
#pragma unroll
    for (int c = 0; c < 4; c++) tc::ld16(tbase + lane + col + 16 * c, v + 16 * c);
    tc::ld_wait();
}

// one MMA round: issue (thread 0), commit, wait (all threads).  Returns false on timeout.
template <typename F>
__device__ __forceinline__ bool mma_round(uint64_t *mbar, uint32_t &phase, F issue) {
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (threadIdx.x == 0) {
        issue();
        tc::commit(mbar);
    }
    bool ok = tc::mbar_wait(mbar, phase);
    phase ^= 1u;
    tc::fence_after();
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

// Forward of one 128-row tile by a CTA of 128 threads, whose input rows are already in A0 (K-major
// 128 x 16): the tile-at-a-time form for a few items (k_learned_correct_few).  Thread t owns row t and
// receives the two outputs in y[0..1].  W = forward images in shared memory, bias = 208 floats (b1, b2,
// b3, b4) in shared memory, ACT = 128 x 64 scratch tile, tmem = 64 allocated columns.  Returns false if a tensor-core wait timed out.
__device__ __forceinline__ bool mlp_tile_forward(uint32_t sW, uint32_t sA0, uint8_t *ACT,
                                                 const float *bias, uint32_t tmem, uint64_t *mbar,
                                                 uint32_t &phase, float *y) {
    const int tid = threadIdx.x;
    const uint32_t sACT = tc::smem_u32(ACT);
    float v[64];
    bool ok = mma_round(mbar, phase, [&] {
        tc::mma(tmem, tc::kdesc(sA0, 2, 0), tc::kdesc(sW + I_B1, 2, 0), tc::idesc_bf16(128, 64), 0);
    });
    if (!ok) return false;
    for (int layer = 0; layer < 3; layer++) {
        ld64(tmem, 0, v);
#pragma unroll
        for (int j = 0; j < 64; j++) v[j] = tc::gelu(v[j] + bias[64 * layer + j]);
        store_row64(ACT, tid, v);
        const uint32_t wimg = sW + (layer == 0 ? I_B2 : layer == 1 ? I_B3 : I_B4);
        const uint32_t idesc = layer < 2 ? tc::idesc_bf16(128, 64) : tc::idesc_bf16(128, 16);
        ok = mma_round(mbar, phase, [&] {
            for (int j = 0; j < 4; j++) tc::mma(tmem, tc::kdesc(sACT, 8, j), tc::kdesc(wimg, 8, j), idesc, j);
        });
        if (!ok) return false;
    }
    const uint32_t lane = (uint32_t)(tid & 96) << 16;
    tc::ld16(tmem + lane, v);
    tc::ld_wait();
    y[0] = v[0] + bias[192];
    y[1] = v[1] + bias[193];
    tc::fence_before();  // the next tile's MMA overwrites the columns just read
    return true;
}

}  // namespace bh
