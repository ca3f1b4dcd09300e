// bh_mlp.cu -- learned far-field correction: a 6 -> 64 -> 64 -> 64 -> 2 GELU MLP on tcgen05.
//
// No reference counterpart (python-bh has no learned component).  BF16 weights and activations,
// FP32 accumulation in tensor memory, FP32 master weights and Adam moments in global memory.
//
// Master parameter layout (float, offsets below): W1[16][64] (rows >= 6 zero), b1[64],
// W2[64][64], b2[64], W3[64][64], b3[64], W4[64][16] (columns >= 2 zero), b4[16]; W_l[in][out].
// Packed images (BF16, K-major core-matrix tiles, see bh_tc.cuh):
//   forward  B1[64 out][16 in], B2[64][64], B3[64][64], B4[16 out][64 in]  (GEMM y = x W)
//   backward B2T[64 in][64 out], B3T[64][64], B4T[64 in][16 out]            (GEMM dx = dy W^T)
//
// Training tile = 128 (input, target) rows; per tile 4 forward GEMMs, 3 backward dA GEMMs and
// 2 weight-gradient GEMMs.  The weight gradients dW = A^T dH reduce over the rows of the tile,
// so the rows are the MMA's K dimension and the layer widths (16 or 64) its M and N dimensions.
// The activations and the dH are stored once, row by row: the forward and dA GEMMs read a tile as
// a K-major operand, the weight-gradient GEMMs read the same bytes as the MN-major transpose
// (tc::tdesc).  Two layers share one M = 128 MMA by lying side by side in one tile: [a1 | a2]^T
// [dh2 | dh3] holds dW2 and dW3 as diagonal blocks, [a0 | a3]^T [dh1 | dh4] holds dW1 and dW4.
#include "bh_mlp.cuh"

namespace bh {

constexpr int MT = 128;  // rows per tile

// ------------------------------------------------------------------ packing
__global__ void k_mlp_pack(const float *p, uint8_t *img) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    // forward images
    if (t < 64 * 16) {  // B1[n][k] = W1[k][n]
        int n = t / 16, k = t % 16;
        float v = k < MLP_IN ? p[P_W1 + k * 64 + n] : 0.f;
        *reinterpret_cast<uint16_t *>(img + I_B1 + tc::kmajor_off(n, k, 2)) = bf16_bits(v);
    }
    if (t < 64 * 64) {
        int n = t / 64, k = t % 64;
        *reinterpret_cast<uint16_t *>(img + I_B2 + tc::kmajor_off(n, k, 8)) =
            bf16_bits(p[P_W2 + k * 64 + n]);
        *reinterpret_cast<uint16_t *>(img + I_B3 + tc::kmajor_off(n, k, 8)) =
            bf16_bits(p[P_W3 + k * 64 + n]);
        // backward: B2T[n = in][k = out] = W2[in][out]
        *reinterpret_cast<uint16_t *>(img + I_B2T + tc::kmajor_off(n, k, 8)) =
            bf16_bits(p[P_W2 + n * 64 + k]);
        *reinterpret_cast<uint16_t *>(img + I_B3T + tc::kmajor_off(n, k, 8)) =
            bf16_bits(p[P_W3 + n * 64 + k]);
    }
    if (t < 16 * 64) {  // B4[n][k] = W4[k][n] (n < 16 outputs)
        int n = t / 64, k = t % 64;
        float v = n < MLP_OUT ? p[P_W4 + k * 16 + n] : 0.f;
        *reinterpret_cast<uint16_t *>(img + I_B4 + tc::kmajor_off(n, k, 8)) = bf16_bits(v);
        // B4T[n = in (64)][k = out (16)] = W4[in][out]
        int n2 = t / 16, k2 = t % 16;
        float v2 = k2 < MLP_OUT ? p[P_W4 + n2 * 16 + k2] : 0.f;
        *reinterpret_cast<uint16_t *>(img + I_B4T + tc::kmajor_off(n2, k2, 2)) = bf16_bits(v2);
    }
}

// ---------------------------------------------------------------- inference
constexpr int INFER_GROUPS = 8;  // 128-row tiles in flight per CTA, one per group of 128 threads
constexpr int INFER_CTAS = 1;    // CTAs per SM (64 registers a thread, 151 KB, all of the TMEM columns)
struct MlpSmemInfer {
    // byte offsets in dynamic shared memory
    static constexpr int W = 0;                              // forward images, I_FWD bytes
    static constexpr int ACT = I_FWD;                        // per group: 128 x 64 BF16
    static constexpr int BIAS = ACT + INFER_GROUPS * 16384;  // 208 floats
    static constexpr int TOTAL = BIAS + 208 * 4;
    static_assert(INFER_CTAS * (TOTAL + 1024) <= 227 * 1024, "INFER_CTAS must fit in the SM's shared memory");
    static_assert(INFER_CTAS * INFER_GROUPS * 64 <= 512, "and in its tensor memory");
};

// biases b1, b2, b3, b4 side by side
__device__ __forceinline__ void load_bias(float *bias, const float *params) {
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        bias[i] = params[P_B1 + i];
        bias[64 + i] = params[P_B2 + i];
        bias[128 + i] = params[P_B3 + i];
    }
    if (threadIdx.x < 16) bias[192 + threadIdx.x] = params[P_B4 + threadIdx.x];
}

// out[r] = MLP(feats[r][0..5]) for r < P; feats row stride fs floats, out row stride 2.
// 1,000,003 rows, stride 8: 119 us -> 70 us (one 128-thread tile per CTA, scalar epilogue, single
// conversions and the whole accumulator row in registers before; 101 us with single conversions, when
// two CTAs of four groups took 107 and four of two 111: each stages the weights).
__global__ void __launch_bounds__(128 * INFER_GROUPS, INFER_CTAS)
k_mlp_infer(const float *feats, int fs, long long P, const uint8_t *img, const float *params, float *out,
            unsigned *err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ uint64_t mbars[INFER_GROUPS];
    __shared__ uint32_t tslot;
    float *bias = reinterpret_cast<float *>(sm + MlpSmemInfer::BIAS);
    const int tid = threadIdx.x, grp = tid >> 7, r = tid & 127;
    uint8_t *ACT = sm + MlpSmemInfer::ACT + 16384 * grp;
    copy_bytes(sm + MlpSmemInfer::W, img, I_FWD);
    load_bias(bias, params);
    if (tid < 32) {
        tc::tmem_alloc(&tslot, 64 * INFER_GROUPS);
        tc::tmem_relinquish();
    }
    if (tid < INFER_GROUPS) {
        tc::mbar_init(&mbars[tid], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tslot + 64 * grp, sW = tc::smem_u32(sm + MlpSmemInfer::W);
    uint32_t phase = 0;
    bool ok = true;
    // rows start on 16 bytes: two vector loads a row (a row's last floats may not exist)
    const bool vin = (fs & 3) == 0 && (reinterpret_cast<uintptr_t>(feats) & 15) == 0;
    const bool vout = (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    const long long ntiles = (P + MT - 1) / MT, stride = (long long)gridDim.x * INFER_GROUPS;
    auto load = [&](long long t, float *f) {
        const long long row = t * MT + r;
        if (row >= P) {
#pragma unroll
            for (int k = 0; k < MLP_IN; k++) f[k] = 0.f;
        } else if (vin) {
            const float4 a = *reinterpret_cast<const float4 *>(feats + row * fs);
            const float2 b = *reinterpret_cast<const float2 *>(feats + row * fs + 4);
            f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y;
        } else {
#pragma unroll
            for (int k = 0; k < MLP_IN; k++) f[k] = feats[row * fs + k];
        }
    };
    float f[16];
#pragma unroll
    for (int k = MLP_IN; k < 16; k++) f[k] = 0.f;
    long long t = blockIdx.x + (long long)gridDim.x * grp;
    if (t < ntiles) load(t, f);
    for (; t < ntiles; t += stride) {
        const long long row = t * MT + r;
        store_row16(ACT, r, f);
        if (t + stride < ntiles) load(t + stride, f);  // in flight while this tile runs
        float y[2];
        if (!mlp_group_forward(sW, ACT, bias, tmem, &mbars[grp], phase, 1 + grp, ok, y)) break;
        if (row < P && ok) {
            if (vout) {
                *reinterpret_cast<float2 *>(out + row * 2) = make_float2(y[0], y[1]);
            } else {
                out[row * 2 + 0] = y[0];
                out[row * 2 + 1] = y[1];
            }
        }
    }
    if (!ok) {  // flagged; a second bounded wait for the MMAs in flight
        atomicOr(err, 8u /*BH_DEV_WAIT_TIMEOUT*/);
        tc::mbar_wait(&mbars[grp], phase ^ 1u);
    }
    tc::fence_before();
    __syncthreads();
    if (tid < 32) tc::tmem_dealloc(tslot, 64 * INFER_GROUPS);
}

// ----------------------------------------------------------------- training
constexpr int TT = 512;  // training threads: 128 rows x 4 groups of 16 columns
struct MlpSmemTrain {
    static constexpr int W = 0;              // all images, I_TOTAL bytes
    static constexpr int T12 = I_TOTAL;      // 128 x 128: [a1 | a2]
    static constexpr int T03 = T12 + 32768;  // 128 x 80: [a0 (16) | a3]
    static constexpr int D23 = T03 + 20480;  // 128 x 128: [dh2 | dh3]
    static constexpr int D14 = D23 + 32768;  // 128 x 80: [dh1 | dh4 (16)]
    static constexpr int BIAS = D14 + 20480;  // 208 floats
    static constexpr int TOTAL = BIAS + 832;
};
constexpr int KC12 = 16, KC03 = 10;  // core columns of the 128- and 80-column tiles
// TMEM columns
constexpr uint32_t T_H1 = 0, T_H2 = 64, T_H3 = 128, T_Y = 192, T_DA = 208, T_G23 = 288, T_G14 = 416;

// Column sums over the warp's 32 rows: lanes 2 c and 2 c + 1 return the sum of v[c] (FP32, a
// butterfly that halves the columns a lane still carries at each exchange: 16 shuffles).
__device__ __forceinline__ float colsum16(const float *v) {
    const int lane = threadIdx.x & 31;
    float a[8], b[4], c[2];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const bool hi = lane & 16;
        a[i] = (hi ? v[i + 8] : v[i]) + __shfl_xor_sync(0xffffffffu, hi ? v[i] : v[i + 8], 16);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const bool hi = lane & 8;
        b[i] = (hi ? a[i + 4] : a[i]) + __shfl_xor_sync(0xffffffffu, hi ? a[i] : a[i + 4], 8);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const bool hi = lane & 4;
        c[i] = (hi ? b[i + 2] : b[i]) + __shfl_xor_sync(0xffffffffu, hi ? b[i] : b[i + 2], 4);
    }
    const bool hi = lane & 2;
    float s = (hi ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, hi ? c[0] : c[1], 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// grad[0..15] += g, four at a time where the address allows
__device__ __forceinline__ void add16(float *grad, const float *g, bool vec) {
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
        if (vec)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(grad + k), "f"(g[k]),
                         "f"(g[k + 1]), "f"(g[k + 2]), "f"(g[k + 3])
                         : "memory");
        else
#pragma unroll
            for (int q = 0; q < 4; q++) atomicAdd(grad + k + q, g[k + q]);
    }
}

// One pass over rows [0, P) of (feats, targets): accumulates d(loss)/d(params) into grad (FP32,
// atomics) and the sum of squared errors into *loss.  loss = mean over rows and outputs of
// (y - target)^2, gradient scaled by 2 / (P * 2).
//
// Bound: the chain of nine MMA round trips per tile (one tile per SM at a time: the two layers'
// operands take 143 KB) and the epilogues' FP32 work.  16 warps share a tile, a thread 16 columns
// of one row, so an epilogue is a sixteenth of the row's work a thread; gelu' is formed with gelu
// (one tanh) and kept in registers until the way back; the biases' gradients are FP32 column sums
// by shuffles.  65,536 rows, the training step: 3,790 us -> 35 us (39 with single bf16 conversions;
// before: shared-memory FP32 atomics, 32 lanes to one address, and scattered 2-byte stores of
// transposed copies of every operand).
__global__ void __launch_bounds__(TT, 1) k_mlp_train(const float *feats, int fs, const float *targets,
                                                     long long P, const uint8_t *img,
                                                     const float *params, float *grad, float *loss,
                                                     unsigned *err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tslot;
    using L = MlpSmemTrain;
    float *bias = reinterpret_cast<float *>(sm + L::BIAS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = (warp & 3) * 32 + lane, cg = warp >> 2;  // row, column group (a warp reads TMEM lanes 32 (warp % 4) ..)
    copy_bytes(sm + L::W, img, I_TOTAL);
    load_bias(bias, params);
    // the padding columns of a0 (6..15) and dh4 (2..15) are zero throughout
    if (tid < MT) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(sm + L::T03 + tc::kmajor_off(tid, 8, KC03)) = z;
        *reinterpret_cast<uint4 *>(sm + L::D14 + tc::kmajor_off(tid, 64, KC03)) = z;
        *reinterpret_cast<uint4 *>(sm + L::D14 + tc::kmajor_off(tid, 72, KC03)) = z;
    }
    if (tid < 32) {
        tc::tmem_alloc(&tslot, 512);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(&mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tm = tslot, tl = tm + ((uint32_t)(warp & 3) << 21);  // this warp's TMEM lanes
    const uint32_t sW = tc::smem_u32(sm + L::W), s12 = tc::smem_u32(sm + L::T12), s03 = tc::smem_u32(sm + L::T03);
    const uint32_t d23 = tc::smem_u32(sm + L::D23), d14 = tc::smem_u32(sm + L::D14);
    uint32_t phase = 0;
    bool ok = true;  // per thread; the CTA leaves together before the next tile's first MMA
    const float gscale = 2.f / (float)(P * MLP_OUT);
    const long long ntiles = (P + MT - 1) / MT;
    float gb1 = 0.f, gb2 = 0.f, gb3 = 0.f;  // bias gradients of column 16 cg + lane / 2
    float gb4[2] = {0.f, 0.f}, lsum = 0.f;  // (column group 0)
    // thread 0 issues; everybody waits for the MMAs issued so far
    auto round = [&](auto issue) {
        tc::fence_async_smem();
        tc::fence_before();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            issue();
        }
    };
    auto wait = [&]() {
        ok = ok && tc::mbar_wait(&mbar, phase);
        phase ^= 1u;
        tc::fence_after();
    };
    auto gemm64 = [&](uint32_t dcol, uint32_t a, int kc, uint32_t w) {  // 128 x 64 += A (64) x W
#pragma unroll
        for (int j = 0; j < 4; j++)
            tc::mma(tm + dcol, tc::kdesc(a, kc, j), tc::kdesc(w, 8, j), tc::idesc_bf16(128, 64), j);
        tc::commit(&mbar);
    };
    // activations of one layer: the thread's 16 columns of gelu(h + b) to the tile's columns c0 + 16 cg
    auto forward = [&](uint32_t hcol, int layer, uint8_t *tile, int c0, int kc, float *dg) {
        float v[16];
        tc::ld16(tl + hcol + 16 * cg, v);
        tc::ld_wait();
        const float4 *b4 = reinterpret_cast<const float4 *>(bias + 64 * layer + 16 * cg);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 b = b4[q];
            v[4 * q] = tc::gelu_and_grad(v[4 * q] + b.x, dg[4 * q]);
            v[4 * q + 1] = tc::gelu_and_grad(v[4 * q + 1] + b.y, dg[4 * q + 1]);
            v[4 * q + 2] = tc::gelu_and_grad(v[4 * q + 2] + b.z, dg[4 * q + 2]);
            v[4 * q + 3] = tc::gelu_and_grad(v[4 * q + 3] + b.w, dg[4 * q + 3]);
        }
        store_cols16(tile, r, c0 + 16 * cg, kc, v);
    };
    // dh = da * gelu'(h) of one layer; returns the thread's column sum (FP32 values, before rounding)
    auto backward = [&](const float *dg, uint8_t *tile, int c0, int kc) -> float {
        float v[16];
        tc::ld16(tl + T_DA + 16 * cg, v);
        tc::ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] *= dg[j];
        store_cols16(tile, r, c0 + 16 * cg, kc, v);
        return colsum16(v);
    };
    float f[MLP_IN], tg[2];
    auto load = [&](long long t) {
        const long long row = t * MT + r;
        const bool valid = row < P;
#pragma unroll
        for (int k = 0; k < MLP_IN; k++) f[k] = valid ? feats[row * fs + k] : 0.f;
        tg[0] = valid ? targets[row * 2] : 0.f;
        tg[1] = valid ? targets[row * 2 + 1] : 0.f;
    };
    bool pending = false;  // the previous tile's last MMAs have not been waited for
    uint32_t acc = 0u;     // the weight gradients of earlier tiles are in TMEM
    if (cg == 0 && blockIdx.x < ntiles) load(blockIdx.x);
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const bool valid = t * MT + r < P;
        if (pending) wait();  // the operand tiles are free again
        pending = false;
        float yt[2] = {tg[0], tg[1]};
        if (cg == 0) {
            uint4 w;
            w.x = bf16x2_bits(f[0], f[1]);
            w.y = bf16x2_bits(f[2], f[3]);
            w.z = bf16x2_bits(f[4], f[5]);
            w.w = 0u;
            *reinterpret_cast<uint4 *>(sm + L::T03 + tc::kmajor_off(r, 0, KC03)) = w;
            if (t + gridDim.x < ntiles) load(t + gridDim.x);  // in flight while this tile runs
        }
        if (!__syncthreads_and(ok ? 1 : 0)) break;
        float dg1[16], dg2[16], dg3[16];
        round([&] {
            tc::mma(tm + T_H1, tc::kdesc(s03, KC03, 0), tc::kdesc(sW + I_B1, 2, 0), tc::idesc_bf16(128, 64), 0);
            tc::commit(&mbar);
        });
        wait();
        forward(T_H1, 0, sm + L::T12, 0, KC12, dg1);
        round([&] { gemm64(T_H2, s12, KC12, sW + I_B2); });
        wait();
        forward(T_H2, 1, sm + L::T12, 64, KC12, dg2);
        round([&] { gemm64(T_H3, s12 + 8 * 128, KC12, sW + I_B3); });
        wait();
        forward(T_H3, 2, sm + L::T03, 16, KC03, dg3);
        round([&] {
#pragma unroll
            for (int j = 0; j < 4; j++)
                tc::mma(tm + T_Y, tc::kdesc(s03 + 2 * 128, KC03, j), tc::kdesc(sW + I_B4, 8, j), tc::idesc_bf16(128, 16), j);
            tc::commit(&mbar);
        });
        wait();
        if (cg == 0) {  // loss and output gradient (rows past the end: zero, and so is all that follows)
            float y[2], dy[2];
            tc::ld2(tl + T_Y, y);
            tc::ld_wait();
#pragma unroll
            for (int k = 0; k < MLP_OUT; k++) {
                const float e = valid ? y[k] + bias[192 + k] - yt[k] : 0.f;
                lsum += e * e;
                dy[k] = gscale * e;
                gb4[k] += dy[k];
            }
            *reinterpret_cast<uint32_t *>(sm + L::D14 + tc::kmajor_off(r, 64, KC03)) =
                bf16x2_bits(dy[0], dy[1]);
        }
        round([&] {  // da3 = dh4 W4^T
            tc::mma(tm + T_DA, tc::kdesc(d14 + 8 * 128, KC03, 0), tc::kdesc(sW + I_B4T, 2, 0), tc::idesc_bf16(128, 64), 0);
            tc::commit(&mbar);
        });
        wait();
        gb3 += backward(dg3, sm + L::D23, 64, KC12);
        round([&] { gemm64(T_DA, d23 + 8 * 128, KC12, sW + I_B3T); });
        wait();
        gb2 += backward(dg2, sm + L::D23, 0, KC12);
        round([&] {
            gemm64(T_DA, d23, KC12, sW + I_B2T);
#pragma unroll
            for (int j = 0; j < 8; j++)  // [a1 | a2]^T [dh2 | dh3] over the tile's 128 rows
                tc::mma(tm + T_G23, tc::tdesc(s12, KC12, j), tc::tdesc(d23, KC12, j), tc::idesc_bf16_t(128, 128),
                        acc | (j > 0 ? 1u : 0u));
        });
        wait();
        gb1 += backward(dg1, sm + L::D14, 0, KC03);
        round([&] {
            // [a0 | a3]^T [dh1 | dh4]: rows 80..127 of the product read past the tile's 80
            // columns (the bytes that follow in shared memory) and are not used
#pragma unroll
            for (int j = 0; j < 8; j++)
                tc::mma(tm + T_G14, tc::tdesc(s03, KC03, j), tc::tdesc(d14, KC03, j), tc::idesc_bf16_t(128, 80),
                        acc | (j > 0 ? 1u : 0u));
            tc::commit(&mbar);
        });
        pending = true;
        acc = 1u;
    }
    if (pending) wait();
    if (__syncthreads_and(ok ? 1 : 0)) {
        // ---- this CTA's share of the gradients to global memory (nothing without a tile)
        if (acc) {
            const bool vec = (reinterpret_cast<uintptr_t>(grad) & 15) == 0;
            float g[16];
            // G23: row r; dW2 = rows 0..63 columns 0..63, dW3 = rows 64..127 columns 64..127
            tc::ld16(tl + T_G23 + (r < 64 ? 0 : 64) + 16 * cg, g);
            tc::ld_wait();
            add16(grad + (r < 64 ? P_W2 + r * 64 : P_W3 + (r - 64) * 64) + 16 * cg, g, vec);
            // G14: dW1 = rows 0..5 columns 0..63, dW4 = rows 16..79 columns 64, 65
            // (tcgen05.ld is warp-collective: every lane loads)
            tc::ld16(tl + T_G14 + 16 * cg, g);
            tc::ld_wait();
            if (r < MLP_IN) add16(grad + P_W1 + r * 64 + 16 * cg, g, vec);
            if (cg == 0) {
                tc::ld2(tl + T_G14 + 64, g);
                tc::ld_wait();
                if (r >= 16 && r < 80)
                    for (int k = 0; k < MLP_OUT; k++) atomicAdd(&grad[P_W4 + (r - 16) * 16 + k], g[k]);
            }
            if ((lane & 1) == 0) {
                const int c = 16 * cg + (lane >> 1);
                atomicAdd(&grad[P_B1 + c], gb1);
                atomicAdd(&grad[P_B2 + c], gb2);
                atomicAdd(&grad[P_B3 + c], gb3);
            }
            if (cg == 0) {
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
                    gb4[0] += __shfl_xor_sync(0xffffffffu, gb4[0], o);
                    gb4[1] += __shfl_xor_sync(0xffffffffu, gb4[1], o);
                }
                if (lane < MLP_OUT) atomicAdd(&grad[P_B4 + lane], lane ? gb4[1] : gb4[0]);
                if (lane == 0) atomicAdd(loss, lsum);
            }
        }
    } else {  // flagged; a second bounded wait for the MMAs in flight
        if (tid == 0) {
            atomicOr(err, 8u /*BH_DEV_WAIT_TIMEOUT*/);
            tc::mbar_wait(&mbar, phase ^ 1u);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (tid < 32) tc::tmem_dealloc(tm, 512);
}

// the operand images' copies of parameter i (k_mlp_pack's layout)
__device__ __forceinline__ void pack_param(uint8_t *img, int i, float v) {
    auto put = [&](int off) { *reinterpret_cast<uint16_t *>(img + off) = bf16_bits(v); };
    if (i < P_B1) {  // W1[k][n]
        const int k = (i - P_W1) / 64, n = (i - P_W1) % 64;
        put(I_B1 + tc::kmajor_off(n, k, 2));
    } else if (i >= P_W2 && i < P_B2) {
        const int k = (i - P_W2) / 64, n = (i - P_W2) % 64;
        put(I_B2 + tc::kmajor_off(n, k, 8));
        put(I_B2T + tc::kmajor_off(k, n, 8));
    } else if (i >= P_W3 && i < P_B3) {
        const int k = (i - P_W3) / 64, n = (i - P_W3) % 64;
        put(I_B3 + tc::kmajor_off(n, k, 8));
        put(I_B3T + tc::kmajor_off(k, n, 8));
    } else if (i >= P_W4 && i < P_B4) {  // W4[k][n]
        const int k = (i - P_W4) / 16, n = (i - P_W4) % 16;
        put(I_B4 + tc::kmajor_off(n, k, 8));
        put(I_B4T + tc::kmajor_off(k, n, 2));
    }
}

// Adam (Kingma & Ba) on the master parameters; zeroes the gradient.  img (or NULL): the operand
// images follow the parameters (a launch less per training step).
__global__ void k_mlp_adam(float *p, float *m, float *v, float *g, int step, float lr, float b1,
                           float b2, float eps, uint8_t *img) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P_TOTAL) return;
    // structurally zero entries stay zero
    bool fixed = (i >= P_W1 && i < P_B1 && (i - P_W1) / 64 >= MLP_IN) ||
                 (i >= P_W4 && i < P_B4 && (i - P_W4) % 16 >= MLP_OUT) || (i >= P_B4 + MLP_OUT);
    float gi = fixed ? 0.f : g[i];
    g[i] = 0.f;
    if (fixed) {
        p[i] = 0.f;
        if (img) pack_param(img, i, 0.f);
        return;
    }
    float mi = b1 * m[i] + (1.f - b1) * gi;
    float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float mh = mi / (1.f - powf(b1, (float)step));
    float vh = vi / (1.f - powf(b2, (float)step));
    const float pi = p[i] - lr * mh / (sqrtf(vh) + eps);
    p[i] = pi;
    if (img) pack_param(img, i, pi);
}

// -------------------------------------------------------------------- launches
cudaError_t mlp_init() {
    cudaError_t e = cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         MlpSmemInfer::TOTAL);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                MlpSmemTrain::TOTAL);
}

cudaError_t mlp_pack(const float *params, uint8_t *img, cudaStream_t st) {
    k_mlp_pack<<<16, 256, 0, st>>>(params, img);
    return cudaGetLastError();
}

cudaError_t mlp_infer(const float *feats, int fs, long long P, const uint8_t *img,
                      const float *params, float *out, unsigned *err, cudaStream_t st) {
    if (P <= 0) return cudaSuccess;
    long long tiles = (P + MT - 1) / MT;
    const long long cap = device_sm_count() * (long long)INFER_CTAS;
    int grid = (int)(tiles < cap ? tiles : cap);
    k_mlp_infer<<<grid, 128 * INFER_GROUPS, MlpSmemInfer::TOTAL, st>>>(feats, fs, P, img, params, out, err);
    return cudaGetLastError();
}

cudaError_t mlp_train(const float *feats, int fs, const float *targets, long long P,
                      const uint8_t *img, const float *params, float *grad, float *loss,
                      unsigned *err, cudaStream_t st) {
    if (P <= 0) return cudaSuccess;
    long long tiles = (P + MT - 1) / MT;
    const long long cap = device_sm_count();
    int grid = (int)(tiles < cap ? tiles : cap);
    k_mlp_train<<<grid, TT, MlpSmemTrain::TOTAL, st>>>(feats, fs, targets, P, img, params,
                                                            grad, loss, err);
    return cudaGetLastError();
}

cudaError_t mlp_adam(float *p, float *m, float *v, float *g, int step, float lr, uint8_t *img, cudaStream_t st) {
    k_mlp_adam<<<(P_TOTAL + 127) / 128, 128, 0, st>>>(p, m, v, g, step, lr, 0.9f, 0.999f, 1e-8f, img);
    return cudaGetLastError();
}

}  // namespace bh
