// bh_tree.cu -- create_tree and summarize kernels.
//
// create_tree = prologue -> bbox (its last block squares the box) -> place -> scan (one pass)
//   -> scatter (permutation, per-quadrant sort, gather) -> work items (one pass).
//   Replaces set_particles_bounding_box (python-bh/barneshut/implementations/base.py:211-239),
//   g_place_particles, g_calculate_box_cumm, g_sort_particles
//   (python-bh/barneshut/kernels/grid_decomposition/gpu/grid.py:15-76).
// summarize = one kernel over tiles of leaf boxes: leaf moments, pyramid, records.
//   Replaces g_summarize (gpu/grid.py:78-114) and calc_COM (internals/cloud.py:9-17).
#include <cstring>

#include "bh_internal.cuh"

namespace bh {

constexpr int TPB = 256;

static inline unsigned grid_for(long long n, int tpb, long long cap) {
    long long b = (n + tpb - 1) / tpb;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (unsigned)b;
}

// ----------------------------------------------------------------- prologue
// Zero the box and quadrant histograms, reset the bounding-box accumulators and
// pair counters, advance the state epoch.
__global__ void k_prologue(DevPlan d) {
    step_enter();
    long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long stride = (long long)gridDim.x * blockDim.x;
    if (tid == 0) {
        d.glob->epoch += 1;
        d.glob->near_pairs = 0;
        d.glob->far_pairs = 0;
        d.glob->corr_pairs = 0;
        d.glob->far_pids = 0;
        d.glob->nbig = 0;
        d.glob->nhuge = 0;
    }
    if (tid < d.nsys) {
        d.dyn[tid].bbmin[0] = d.dyn[tid].bbmin[1] = ~0ull;
        d.dyn[tid].bbmax[0] = d.dyn[tid].bbmax[1] = 0ull;
    }
    for (long long b = tid; b < d.B_total; b += stride) {
        reinterpret_cast<int4 *>(d.qcounts)[b] = make_int4(0, 0, 0, 0);
    }
}

// One thread per system: the square bounding box (helpers/grid.py:10-26), its
// box edge step = edge / G (base.py:233) and 1 / step, once per step.
__device__ void bbox_finalize_sys(const DevPlan &d, int s, SysDyn &dy) {
    double mnx = unord_bits(dy.bbmin[0]), mny = unord_bits(dy.bbmin[1]);
    double mxx = unord_bits(dy.bbmax[0]), mxy = unord_bits(dy.bbmax[1]);
    if (d.sys[s].fixed_grid) {  // part of a larger system: the whole system's extents
        mnx = d.sys[s].fg_ext[0];
        mny = d.sys[s].fg_ext[1];
        mxx = d.sys[s].fg_ext[2];
        mxy = d.sys[s].fg_ext[3];
    }
    double step;
    square_bbox(mnx, mny, mxx, mxy, d.sys[s].G, &step);
    dy.minx = mnx;
    dy.miny = mny;
    dy.step = step;
    dy.inv_step = step > 0.0 ? 1.0 / step : 0.0;
    // float key estimate: p and mn rounded to float (relative error 2^-24 each), their
    // difference and the product with float(1 / step) rounded (2^-24 each); in box edges the
    // error is at most ((|p| + |mn|) / step + 2 q) 2^-24 <= ((2 |mn| + |edge|) / step + 2 G) 2^-24;
    // a factor 4 covers the remaining roundings
    dy.minx_f = __double2float_rn(mnx);
    dy.miny_f = __double2float_rn(mny);
    dy.inv_step_f = __double2float_rn(dy.inv_step);
    if (step > 0.0 && isfinite(step)) {
        const double am = fmax(fabs(mnx), fabs(mny)), G = (double)d.sys[s].G;
        const double tol = 4.0 * ((2.0 * am + G * step) * dy.inv_step + 2.0 * G) * 5.9604644775390625e-8;
        dy.key_tol = tol < 0.25 ? (float)tol : 1.f;
    } else {
        dy.key_tol = 1.f;  // the FP64 key for every particle
    }
}

// --------------------------------------------------------------------- bbox
// Min / max of x and y per system on the ordered-integer image of the doubles
// (integer min/max, no FP64 pipe work).  Each block reduces a contiguous tile.
__device__ __forceinline__ void minmax_ord(unsigned long long u, unsigned long long &mn, unsigned long long &mx) {
    mn = u < mn ? u : mn;
    mx = u > mx ? u : mx;
}

__device__ __forceinline__ void bbox_block_commit(const DevPlan &d, int s, unsigned long long mn0,
                                                  unsigned long long mn1, unsigned long long mx0,
                                                  unsigned long long mx1, unsigned long long (*red)[TPB / 32]) {
    for (int o = 16; o; o >>= 1) {
        unsigned long long a = __shfl_xor_sync(0xffffffffu, mn0, o); mn0 = a < mn0 ? a : mn0;
        a = __shfl_xor_sync(0xffffffffu, mn1, o); mn1 = a < mn1 ? a : mn1;
        a = __shfl_xor_sync(0xffffffffu, mx0, o); mx0 = a > mx0 ? a : mx0;
        a = __shfl_xor_sync(0xffffffffu, mx1, o); mx1 = a > mx1 ? a : mx1;
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { red[0][w] = mn0; red[1][w] = mn1; red[2][w] = mx0; red[3][w] = mx1; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < TPB / 32; k++) {
            mn0 = red[0][k] < mn0 ? red[0][k] : mn0; mn1 = red[1][k] < mn1 ? red[1][k] : mn1;
            mx0 = red[2][k] > mx0 ? red[2][k] : mx0; mx1 = red[3][k] > mx1 ? red[3][k] : mx1;
        }
        if (mx0 | mx1) {
            atomicMin(&d.dyn[s].bbmin[0], mn0); atomicMin(&d.dyn[s].bbmin[1], mn1);
            atomicMax(&d.dyn[s].bbmax[0], mx0); atomicMax(&d.dyn[s].bbmax[1], mx1);
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(TPB) k_bbox(DevPlan d) {
    step_enter();
    const int cur = d.glob->epoch & 1;
    const double *X = d.X[cur], *Y = d.Y[cur];
    __shared__ unsigned long long red[4][TPB / 32];
    __shared__ int sys0;
    if (d.nsys == 1) {
        // one system: a grid-stride sweep over 16-byte pairs, four pairs of each array in flight
        // per thread (the state arrays are 256-byte aligned)
        const long long n2 = d.n_total >> 1, stride = (long long)gridDim.x * TPB;
        const double2 *X2 = reinterpret_cast<const double2 *>(X), *Y2 = reinterpret_cast<const double2 *>(Y);
        unsigned long long mn0 = ~0ull, mn1 = ~0ull, mx0 = 0, mx1 = 0;
        long long i = (long long)blockIdx.x * TPB + threadIdx.x;
        for (; i + 3 * stride < n2; i += 4 * stride) {
            double2 a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                a[u] = X2[i + u * stride];
                b[u] = Y2[i + u * stride];
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                minmax_ord(ord_bits(a[u].x), mn0, mx0);
                minmax_ord(ord_bits(a[u].y), mn0, mx0);
                minmax_ord(ord_bits(b[u].x), mn1, mx1);
                minmax_ord(ord_bits(b[u].y), mn1, mx1);
            }
        }
        for (; i < n2; i += stride) {
            const double2 a = X2[i], b = Y2[i];
            minmax_ord(ord_bits(a.x), mn0, mx0);
            minmax_ord(ord_bits(a.y), mn0, mx0);
            minmax_ord(ord_bits(b.x), mn1, mx1);
            minmax_ord(ord_bits(b.y), mn1, mx1);
        }
        if ((d.n_total & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
            minmax_ord(ord_bits(X[d.n_total - 1]), mn0, mx0);
            minmax_ord(ord_bits(Y[d.n_total - 1]), mn1, mx1);
        }
        bbox_block_commit(d, 0, mn0, mn1, mx0, mx1, red);
    }
    const long long tile = (long long)TPB * 16;
    for (long long t0 = (long long)blockIdx.x * tile; d.nsys > 1 && t0 < d.n_total; t0 += (long long)gridDim.x * tile) {
        long long t1 = t0 + tile < d.n_total ? t0 + tile : d.n_total;
        if (threadIdx.x == 0) sys0 = find_seg(d.poff_tab, d.nsys, t0);
        __syncthreads();
        int s_first = sys0;
        bool one_sys = d.poff_tab[s_first + 1] >= t1;
        unsigned long long mn0 = ~0ull, mn1 = ~0ull, mx0 = 0, mx1 = 0;
        int cs = s_first;
        if (one_sys && t1 - t0 == tile) {  // a whole tile of one system: 16-byte pairs, all in flight
            const double2 *X2 = reinterpret_cast<const double2 *>(X + t0), *Y2 = reinterpret_cast<const double2 *>(Y + t0);
            double2 a[8], b[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                a[u] = X2[threadIdx.x + u * TPB];
                b[u] = Y2[threadIdx.x + u * TPB];
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                minmax_ord(ord_bits(a[u].x), mn0, mx0);
                minmax_ord(ord_bits(a[u].y), mn0, mx0);
                minmax_ord(ord_bits(b[u].x), mn1, mx1);
                minmax_ord(ord_bits(b[u].y), mn1, mx1);
            }
        } else for (long long i = t0 + threadIdx.x; i < t1; i += TPB) {
            if (!one_sys) {
                int s = find_seg(d.poff_tab, d.nsys, i);
                if (s != cs) {
                    if (mx0 | mx1) {
                        atomicMin(&d.dyn[cs].bbmin[0], mn0); atomicMin(&d.dyn[cs].bbmin[1], mn1);
                        atomicMax(&d.dyn[cs].bbmax[0], mx0); atomicMax(&d.dyn[cs].bbmax[1], mx1);
                    }
                    mn0 = mn1 = ~0ull; mx0 = mx1 = 0; cs = s;
                }
            }
            unsigned long long ux = ord_bits(X[i]), uy = ord_bits(Y[i]);
            mn0 = ux < mn0 ? ux : mn0; mx0 = ux > mx0 ? ux : mx0;
            mn1 = uy < mn1 ? uy : mn1; mx1 = uy > mx1 ? uy : mx1;
        }
        if (!one_sys) {
            if (mx0 | mx1) {
                atomicMin(&d.dyn[cs].bbmin[0], mn0); atomicMin(&d.dyn[cs].bbmin[1], mn1);
                atomicMax(&d.dyn[cs].bbmax[0], mx0); atomicMax(&d.dyn[cs].bbmax[1], mx1);
            }
        } else {
            bbox_block_commit(d, s_first, mn0, mn1, mx0, mx1, red);
        }
        __syncthreads();
    }
    // the last block to finish squares every system's box, a thread per system (512 systems one after
    // another took 1.4 ms)
    __shared__ unsigned ticket;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) ticket = atomicAdd(&d.glob->bbox_done, 1u);
    __syncthreads();
    if (ticket != gridDim.x - 1) return;
    __threadfence();
    for (int s = threadIdx.x; s < d.nsys; s += TPB)
        if (d.sys[s].n > 0) bbox_finalize_sys(d, s, d.dyn[s]);
    if (threadIdx.x == 0) d.glob->bbox_done = 0u;
}

// The box-origin tables of the systems (read by k_gather): the blocks share a single system's table,
// or take whole systems.
__device__ __forceinline__ void fill_origins(const DevPlan &d) {
    for (int s = d.nsys == 1 ? 0 : blockIdx.x; s < d.nsys; s += d.nsys == 1 ? 1 : gridDim.x) {
        if (d.sys[s].n == 0) continue;
        const SysDyn &dy = d.dyn[s];
        const int G = d.sys[s].G;
        double *org = d.org + d.sys[s].ooff;
        const int k0 = d.nsys == 1 ? blockIdx.x * TPB : 0, dk = d.nsys == 1 ? gridDim.x * TPB : TPB;
        for (int k = k0 + threadIdx.x; k < G; k += dk) {
            org[k] = box_origin(dy.minx, k, dy.step);
            org[G + k] = box_origin(dy.miny, k, dy.step);
        }
    }
}

// -------------------------------------------------------------------- place
// Box keys bit-exact with the reference's FP64 keys (computed at twice the box resolution, so
// each particle also gets its quadrant within the box), and a histogram of (box, quadrant)
// pairs aggregated over runs of equal keys in the block (a box's count is the sum of its
// four); a particle's slot is its rank within its quadrant.
constexpr int PLACE_PP = 4;  // consecutive particles per thread

// (64 registers: 4 CTAs per SM)
__global__ void __launch_bounds__(TPB, 4) k_place(DevPlan d) {
    step_enter();
    constexpr int PT = TPB * PLACE_PP;  // particles per block round
    __shared__ int skeys[PT + 1], runold[PT], wmax[TPB / 32];
    const int cur = d.glob->epoch & 1;
    const double *X = d.X[cur], *Y = d.Y[cur];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e0 = (int)threadIdx.x * PLACE_PP;  // the thread's first particle in the round
    fill_origins(d);
    for (long long base = (long long)blockIdx.x * PT; base < d.n_total; base += (long long)gridDim.x * PT) {
        const long long i0 = base + e0;
        double x[PLACE_PP], y[PLACE_PP];
        if (i0 + PLACE_PP <= d.n_total && (i0 & 1) == 0) {  // (always, but for a ragged end)
            const double2 *X2 = reinterpret_cast<const double2 *>(X + i0);
            const double2 *Y2 = reinterpret_cast<const double2 *>(Y + i0);
#pragma unroll
            for (int j = 0; j < PLACE_PP / 2; j++) {
                const double2 a = X2[j], b = Y2[j];
                x[2 * j] = a.x; x[2 * j + 1] = a.y;
                y[2 * j] = b.x; y[2 * j + 1] = b.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < PLACE_PP; j++) {
                x[j] = i0 + j < d.n_total ? X[i0 + j] : 0.0;
                y[j] = i0 + j < d.n_total ? Y[i0 + j] : 0.0;
            }
        }
        int key[PLACE_PP];
        // the thread's particles usually lie in one system: its constants are loaded once
        const int s_first = find_seg(d.poff_tab, d.nsys, i0 < d.n_total ? i0 : d.n_total - 1);
        const bool one_sys = d.poff_tab[s_first + 1] >= i0 + PLACE_PP;
        if (one_sys) {
            const SysDesc &sd = d.sys[s_first];
            const SysDyn &dy = d.dyn[s_first];
            const double mnx = dy.minx, mny = dy.miny, st = dy.step, inv = dy.inv_step;
            const float mnxf = dy.minx_f, mnyf = dy.miny_f, invf = dy.inv_step_f, tol = dy.key_tol;
            const int G = sd.G;
            const long long boff = sd.boff;
#pragma unroll
            for (int j = 0; j < PLACE_PP; j++) {
                const unsigned hx = (unsigned)(__double_as_longlong(x[j]) >> 52) & 0x7FFu;
                const unsigned hy = (unsigned)(__double_as_longlong(y[j]) >> 52) & 0x7FFu;
                if (hx == 0x7FFu || hy == 0x7FFu) raise_err(d.glob, 1u /*BH_DEV_NAN_POSITION*/);
                const int k2x = half_key1_f32(x[j], mnx, st, inv, mnxf, invf, tol, G);
                const int k2y = half_key1_f32(y[j], mny, st, inv, mnyf, invf, tol, G);
                const int box = (int)(boff + (long long)(k2x >> 1) * G + (k2y >> 1));
                key[j] = 4 * box + (k2x & 1) * 2 + (k2y & 1);
                skeys[e0 + j] = key[j];
            }
        } else
#pragma unroll
        for (int j = 0; j < PLACE_PP; j++) {
            const long long i = i0 + j;
            key[j] = -1;
            if (i < d.n_total) {
                const int s = find_seg(d.poff_tab, d.nsys, i);
                const SysDesc &sd = d.sys[s];
                const SysDyn &dy = d.dyn[s];
                // finite test on the exponent bits (no FP64 operation)
                const unsigned hx = (unsigned)(__double_as_longlong(x[j]) >> 52) & 0x7FFu;
                const unsigned hy = (unsigned)(__double_as_longlong(y[j]) >> 52) & 0x7FFu;
                if (hx == 0x7FFu || hy == 0x7FFu) raise_err(d.glob, 1u /*BH_DEV_NAN_POSITION*/);
                // keys at twice the box resolution: box key and quadrant within the box
                const int k2x = half_key1_f32(x[j], dy.minx, dy.step, dy.inv_step, dy.minx_f, dy.inv_step_f, dy.key_tol, sd.G);
                const int k2y = half_key1_f32(y[j], dy.miny, dy.step, dy.inv_step, dy.miny_f, dy.inv_step_f, dy.key_tol, sd.G);
                const int box = (int)(sd.boff + (long long)(k2x >> 1) * sd.G + (k2y >> 1));
                key[j] = 4 * box + (k2x & 1) * 2 + (k2y & 1);
            }
            skeys[e0 + j] = key[j];
        }
        if (threadIdx.x == 0) skeys[PT] = INT_MIN;
        // runs of consecutive particles of the round with the same (box, quadrant): the run's
        // last particle adds the run's length to the quadrant count, whose old value is the run's
        // first slot, so a quadrant whose particles lie in one round gets its slots in input
        // order (the common case when the input is the previous step's order); k_segsort puts
        // the runs of different blocks in order
        __syncthreads();
        int h[PLACE_PP];  // the first particle of each particle's run: a max-scan of run heads
        int hm = 0;
#pragma unroll
        for (int j = 0; j < PLACE_PP; j++) {
            const int e = e0 + j;
            const int kp = e > 0 ? skeys[e - 1] : INT_MIN;
            if (key[j] != kp) hm = e;
            h[j] = hm;
        }
        int hx = hm;  // inclusive max over the threads before and including this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) hx = max(hx, __shfl_up_sync(0xffffffffu, hx, o) * (lane >= o));
        if (lane == 31) wmax[warp] = hx;
        int hb = __shfl_up_sync(0xffffffffu, hx, 1) * (lane >= 1);  // exclusive, within the warp
        __syncthreads();
        for (int w = 0; w < warp; w++) hb = max(hb, wmax[w]);
#pragma unroll
        for (int j = 0; j < PLACE_PP; j++) {
            h[j] = max(h[j], hb);
            const int e = e0 + j;
            if (key[j] >= 0 && key[j] != skeys[e + 1]) runold[h[j]] = atomicAdd(&d.qcounts[key[j]], e - h[j] + 1);
        }
        __syncthreads();
        int kv[PLACE_PP], sv[PLACE_PP];
#pragma unroll
        for (int j = 0; j < PLACE_PP; j++) {
            kv[j] = key[j];  // 4 * box + quadrant
            sv[j] = key[j] >= 0 ? runold[h[j]] + (e0 + j - h[j]) : 0;
        }
        if (i0 + PLACE_PP <= d.n_total && (i0 & 3) == 0) {
            *reinterpret_cast<int4 *>(d.key + i0) = make_int4(kv[0], kv[1], kv[2], kv[3]);
            *reinterpret_cast<int4 *>(d.slot + i0) = make_int4(sv[0], sv[1], sv[2], sv[3]);
        } else {
#pragma unroll
            for (int j = 0; j < PLACE_PP; j++)
                if (i0 + j < d.n_total) {
                    d.key[i0 + j] = kv[j];
                    d.slot[i0 + j] = sv[j];
                }
        }
        __syncthreads();  // the block's shared arrays are reused in the next round
    }
}

// --------------------------------------------------------------------- scan
// Exclusive scans in one pass (decoupled look-back): tiles are numbered in the order their CTAs
// start (a ticket), so every tile's predecessors are already running; a tile publishes its sum,
// then its inclusive prefix once it has read its predecessors' (a predecessor's inclusive prefix
// ends the look-back).  A tile state is gen << 34 | flag << 32 | value (flag 1 = the tile's sum,
// 2 = inclusive prefix); a state of another generation is not yet written, and the scan's last
// tile bumps the generation, so the states need no clearing between scans.  Waits are bounded:
// on timeout the tile raises BH_DEV_WAIT_TIMEOUT and carries on (the result is then invalid).
constexpr unsigned long long SST_AGG = 1ull << 32, SST_PRE = 2ull << 32;
constexpr long long LOOKBACK_SPIN = 1ll << 22;

__device__ __forceinline__ int block_excl_scan(int v, int *sh, int *total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = lane < nw ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) sh[lane] = t;
    }
    __syncthreads();
    int pre = (w ? sh[w - 1] : 0) + x - v;
    if (total) *total = sh[nw - 1];
    __syncthreads();
    return pre;
}

// Generations run 1 .. 2^30 - 1 (30 bits in a state); 0 never tags a state, so the zeroed
// states of a freshly bound plan read as not yet written.
__device__ __forceinline__ unsigned next_gen(unsigned g) { return g >= 0x3FFFFFFFu ? 1u : g + 1u; }

// Warp 0 of the CTA: publish the tile's sum `agg`, look back, publish the inclusive prefix and
// return the tile's exclusive prefix (to lane 0; the caller broadcasts through shared memory).
__device__ int lookback(unsigned long long *state, int tile, unsigned gen, int agg, Globals *glob) {
    const int lane = threadIdx.x & 31;
    volatile unsigned long long *vs = state;
    const unsigned long long tag = (unsigned long long)(gen & 0x3FFFFFFFu) << 34;
    if (tile == 0) {
        if (lane == 0) {
            __threadfence();
            vs[0] = tag | SST_PRE | (unsigned)agg;
        }
        return 0;
    }
    if (lane == 0) {
        __threadfence();
        vs[tile] = tag | SST_AGG | (unsigned)agg;
    }
    int excl = 0;
    int k = tile - 1;  // the nearest predecessor not yet read
    bool timed_out = false;
    while (k >= 0) {
        const int idx = k - lane;
        unsigned long long st = idx >= 0 ? 0ull : (tag | SST_PRE);  // before tile 0: prefix 0
        long long it = 0;
        for (;;) {
            if (idx >= 0) st = vs[idx];
            const bool ready = (st >> 34) == (tag >> 34) && (st & (3ull << 32)) != 0;
            if (__all_sync(0xffffffffu, ready)) break;
            if (++it > LOOKBACK_SPIN) {
                timed_out = true;
                break;
            }
        }
        if (timed_out) break;
        const unsigned pre_mask = __ballot_sync(0xffffffffu, (st & SST_PRE) == SST_PRE);
        const int stop = pre_mask ? __ffs(pre_mask) - 1 : 31;  // nearest inclusive prefix
        int v = lane <= stop ? (int)(unsigned)(st & 0xFFFFFFFFull) : 0;
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        excl += v;
        if (pre_mask) break;
        k -= 32;
    }
    if (lane == 0) {
        if (timed_out) raise_err(glob, 8u /*BH_DEV_WAIT_TIMEOUT*/);
        __threadfence();
        vs[tile] = tag | SST_PRE | (unsigned)(excl + agg);
    }
    return excl;
}

// out[i] = sum(in[0..i)) for i < n, out[n] = sum(in[0..n)); scan k of the plan's three.  QSUM:
// element i is the sum of the four quadrant counts in[4 i .. 4 i + 3] (a box's particles).
template <bool QSUM>
__global__ void __launch_bounds__(TPB) k_scan_lookback(const int *in, long long n, int *out,
                                                      unsigned long long *state, Globals *glob, int k) {
    step_enter();
    __shared__ int sh[32];
    __shared__ int s_tile, s_excl;
    __shared__ unsigned s_gen;
    const long long ntiles = (n + SCAN_TILE - 1) / SCAN_TILE > 0 ? (n + SCAN_TILE - 1) / SCAN_TILE : 1;
    if (threadIdx.x == 0) {
        s_tile = (int)atomicAdd(&glob->scan_ticket[k], 1u);
        s_gen = *(volatile unsigned *)&glob->scan_gen[k];
    }
    __syncthreads();
    const int tile = s_tile;
    const long long b0 = (long long)tile * SCAN_TILE + (long long)threadIdx.x * 16;
    int v[16], sum = 0;
#pragma unroll
    for (int q = 0; q < 16; q++) {
        v[q] = 0;
        if (b0 + q < n) {
            if (QSUM) {
                const int4 c = reinterpret_cast<const int4 *>(in)[b0 + q];
                v[q] = c.x + c.y + c.z + c.w;
            } else {
                v[q] = in[b0 + q];
            }
        }
        sum += v[q];
    }
    int tot;
    int pre = block_excl_scan(sum, sh, &tot);
    if (threadIdx.x < 32) {
        const int e = lookback(state, tile, s_gen, tot, glob);
        if (threadIdx.x == 0) s_excl = e;
    }
    __syncthreads();
    pre += s_excl;
#pragma unroll
    for (int q = 0; q < 16; q++) {
        if (b0 + q < n) out[b0 + q] = pre;
        pre += v[q];
    }
    if (tile == ntiles - 1 && threadIdx.x == 0) {
        out[n] = s_excl + tot;
        glob->scan_ticket[k] = 0u;  // every tile has its ticket: ready for the next scan
        glob->scan_gen[k] = next_gen(s_gen);
    }
}

static cudaError_t scan_excl(const int *in, int *out, long long n, unsigned long long *state,
                             Globals *glob, int k, cudaStream_t st, bool qsum = false) {
    long long ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (ntiles < 1) ntiles = 1;
    if (qsum)
        launch_step(k_scan_lookback<true>, (unsigned)ntiles, TPB, 0, st, in, n, out, state, glob, k);
    else
        launch_step(k_scan_lookback<false>, (unsigned)ntiles, TPB, 0, st, in, n, out, state, glob, k);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- work items
// Force work items: a target group with nt targets is split into
// ceil(nt / chunk) items so that dense groups spread over many CTAs.
__global__ void __launch_bounds__(TPB) k_group_items(DevPlan d) {
    step_enter();
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < d.NG_total; g += stride) {
        int s = find_seg(d.goff_tab, d.nsys, g);
        const SysDesc &sd = d.sys[s];
        long long lg = g - sd.goff;
        int gi = (int)(lg / sd.NGs), gj = (int)(lg - (long long)gi * sd.NGs);
        int gx0 = gi * sd.TG, gy0 = gj * sd.TG;
        int gx1 = min(sd.G, gx0 + sd.TG), gy1 = min(sd.G, gy0 + sd.TG);
        int nt = 0;
        for (int c = gx0; c < gx1; c++) {
            long long b0 = sd.boff + (long long)c * sd.G + gy0;
            nt += d.box_start[b0 + (gy1 - gy0)] - d.box_start[b0];
        }
        d.item_cnt[g] = (nt + d.chunk - 1) / d.chunk;
    }
}

__global__ void __launch_bounds__(TPB) k_fill_items(DevPlan d) {
    step_enter();
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < d.NG_total; g += stride) {
        int o = d.item_off[g], c = d.item_cnt[g];
        for (int k = 0; k < c; k++) d.item_group[o + k] = (int)g;
    }
}

// List-streaming work items.  Per group: the boxes holding fewer than dense_min particles share
// ceil(n_sparse / chunk) items (sub = -1); every denser box gets ceil(n_box / chunk) items of its
// own (sub = cx * TG + cy), which use per-box refined near lists, and a box holding at least
// quad_min particles gets items per quadrant instead (sub = TG^2 + 4 (cx * TG + cy) + quadrant),
// which use per-quadrant refined near lists.  A set of nt targets splits into sitem_count(nt)
// items: full chunks of STREAM_CHUNK and the remainder's pieces (sitem_range).  A group's items
// are the sparse ones, then the boxes' in (cx, cy) order, quadrant by quadrant.  One kernel: a
// warp per group (a lane per box) counts the group's items, the CTA scans its SITEM_TILE groups,
// a look-back over the preceding tiles gives their offset, and the lanes write their boxes'
// items.
constexpr int SITEM_WARPS = SITEM_TILE;  // one group per warp
static_assert(MAX_TG * MAX_TG <= 64, "a lane holds at most two boxes of a group");

// The items of one group, by a warp: the lane's boxes bi = lane, lane + 32 (bi = cx * TG + cy).
struct GroupItems {
    int kind[2], cnt[2], inc[2];  // the boxes' kinds, item counts and their inclusive prefixes in bi order
    int4 qc[2];
    int ns, nbox, tot0, total;    // sparse items, boxes, items of the first 32 boxes, all items
};

__device__ __forceinline__ void group_items(const DevPlan &d, long long g, GroupItems &r) {
    const int lane = threadIdx.x & 31;
    int nb[2] = {0, 0};
    r.kind[0] = r.kind[1] = r.cnt[0] = r.cnt[1] = 0;
    r.qc[0] = r.qc[1] = make_int4(0, 0, 0, 0);
    r.nbox = 0;
    int sparse = 0;
    if (g < d.NG_total) {
        const int s = find_seg(d.goff_tab, d.nsys, g);
        const SysDesc &sd = d.sys[s];
        const long long lg = g - sd.goff;
        const int gi = (int)(lg / sd.NGs), gj = (int)(lg - (long long)gi * sd.NGs);
        const int TG = sd.TG, tgs = __ffs(TG) - 1;
        r.nbox = TG * TG;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int bi = lane + 32 * u;
            const int cx = bi >> tgs, cy = bi & (TG - 1);
            if (bi < r.nbox && gi * TG + cx < sd.G && gj * TG + cy < sd.G) {
                const long long b = sd.boff + (long long)(gi * TG + cx) * sd.G + gj * TG + cy;
                nb[u] = d.box_start[b + 1] - d.box_start[b];
                r.kind[u] = box_item_kind(nb[u], d.dense_min, d.quad_min);
                if (r.kind[u] == 2) {
                    const int4 q = reinterpret_cast<const int4 *>(d.qcounts)[b];
                    r.qc[u] = q;
                    r.cnt[u] = sitem_count(q.x) + sitem_count(q.y) + sitem_count(q.z) + sitem_count(q.w);
                } else if (r.kind[u] == 1) {
                    r.cnt[u] = sitem_count(nb[u]);
                } else {
                    sparse += nb[u];
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sparse += __shfl_xor_sync(0xffffffffu, sparse, o);
    r.ns = sitem_count(sparse);
    // prefixes of the boxes' item counts in bi order (lane's first box, then second)
    r.inc[0] = r.cnt[0];
    r.inc[1] = r.cnt[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y0 = __shfl_up_sync(0xffffffffu, r.inc[0], o), y1 = __shfl_up_sync(0xffffffffu, r.inc[1], o);
        if (lane >= o) {
            r.inc[0] += y0;
            r.inc[1] += y1;
        }
    }
    r.tot0 = __shfl_sync(0xffffffffu, r.inc[0], 31);
    const int tot1 = __shfl_sync(0xffffffffu, r.inc[1], 31);
    r.total = g < d.NG_total ? r.ns + r.tot0 + tot1 : 0;
}

// ... written from item `off` on
__device__ __forceinline__ void group_items_write(const DevPlan &d, long long g, const GroupItems &r, int off) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) d.sitem_off[g] = off;
    for (int k = lane; k < r.ns; k += 32) {  // the sparse boxes' items
        d.sitem_group[off + k] = (int)g;
        d.sitem_sub[off + k] = -1;
        d.sitem_chunk[off + k] = make_int2(k, r.ns);
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int bi = lane + 32 * u;
        int o = off + r.ns + (u ? r.tot0 : 0) + r.inc[u] - r.cnt[u];
        if (r.kind[u] == 1) {
            const int nk = r.cnt[u];
            for (int k = 0; k < nk; k++, o++) {
                d.sitem_group[o] = (int)g;
                d.sitem_sub[o] = bi;
                d.sitem_chunk[o] = make_int2(k, nk);
            }
        } else if (r.kind[u] == 2) {
            const int qv[4] = {r.qc[u].x, r.qc[u].y, r.qc[u].z, r.qc[u].w};
            for (int q = 0; q < 4; q++) {
                const int nk = sitem_count(qv[q]);
                for (int k = 0; k < nk; k++, o++) {
                    d.sitem_group[o] = (int)g;
                    d.sitem_sub[o] = r.nbox + 4 * bi + q;
                    d.sitem_chunk[o] = make_int2(k, nk);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(SITEM_WARPS * 32) k_sitems(DevPlan d) {
    step_enter();
    __shared__ int wtot[SITEM_WARPS], wpre[SITEM_WARPS];
    __shared__ int s_tile, s_excl;
    __shared__ unsigned s_gen;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long ntiles = (d.NG_total + SITEM_TILE - 1) / SITEM_TILE;
    if (threadIdx.x == 0) {
        s_tile = (int)atomicAdd(&d.glob->scan_ticket[2], 1u);
        s_gen = *(volatile unsigned *)&d.glob->scan_gen[2];
    }
    __syncthreads();
    const int tile = s_tile;
    const long long g = (long long)tile * SITEM_TILE + warp;
    GroupItems gi;
    group_items(d, g, gi);
    if (lane == 0) wtot[warp] = gi.total;
    __syncthreads();
    if (threadIdx.x < 32) {
        int v = lane < SITEM_WARPS ? wtot[lane] : 0, x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane < SITEM_WARPS) wpre[lane] = x - v;
        const int tot = __shfl_sync(0xffffffffu, x, 31);
        const int e = lookback(d.sst_sitem, tile, s_gen, tot, d.glob);
        if (threadIdx.x == 0) {
            s_excl = e;
            if (tile == ntiles - 1) {
                d.sitem_off[d.NG_total] = e + tot;
                d.glob->scan_ticket[2] = 0u;
                d.glob->scan_gen[2] = next_gen(s_gen);
            }
        }
    }
    __syncthreads();
    if (g < d.NG_total) group_items_write(d, g, gi, s_excl + wpre[warp]);
}

// ------------------------------------------------------------------ scatter
// Counting sort into box order, each box's particles quadrant by quadrant, and within a quadrant
// in input order (the order the previous step left, or the caller's), so the step does not depend
// on the order in which k_place's atomics handed out slots:
//   k_perm     perm[box_start + earlier quadrants + slot] = input index (slots: k_place);
//   k_segsort  each quadrant's stretch of perm sorted ascending -- up to SEG_REG entries in a
//              thread's registers, longer ones listed for k_segsort_big (up to SEG_LANES entries
//              a warp each, a bitonic network in its registers; up to SEG_MERGE a CTA each, such runs
//              merged in shared memory; longer ones a CTA each, four stable 8-bit radix passes
//              through the dead slot array);
//   k_gather   output particle t takes input perm[t]: the FP64 state of the next buffer, the
//              32-byte packed record (offsets from the box origin computed in FP64, rounded
//              once to float) and the sorted key; and it sums the leaves (below).
constexpr int SEG_REG = 16;
constexpr int SEG_LANES = 256;  // longest stretch sorted by a warp
constexpr int SEG_CHECK = 128;  // stretches up to this long are checked for order by their thread

__device__ __forceinline__ int quad_first(const DevPlan &d, int key4) {
    const int box = key4 >> 2, quad = key4 & 3;
    const int4 qc = reinterpret_cast<const int4 *>(d.qcounts)[box];
    return d.box_start[box] + (quad > 0 ? qc.x : 0) + (quad > 1 ? qc.y : 0) + (quad > 2 ? qc.z : 0);
}

__global__ void __launch_bounds__(TPB) k_perm(DevPlan d) {
    step_enter();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < d.n_total; i += stride)
        d.perm[quad_first(d, d.key[i]) + d.slot[i]] = (int)i;
}

// a stretch of n <= SEG_REG entries in a thread's registers
__device__ __forceinline__ void seg_thread(int *p, int n) {
    int v[SEG_REG];
#pragma unroll
    for (int k = 0; k < SEG_REG; k++) v[k] = k < n ? p[k] : 0x7FFFFFFF;
    bool sorted = true;  // (padding sorts after every index)
#pragma unroll
    for (int k = 0; k + 1 < SEG_REG; k++) sorted &= v[k] <= v[k + 1];
    if (sorted) return;
    // odd-even transposition network: SEG_REG rounds sort SEG_REG entries
#pragma unroll
    for (int r = 0; r < SEG_REG; r++)
#pragma unroll
        for (int k = r & 1; k + 1 < SEG_REG; k += 2) {
            const int lo = min(v[k], v[k + 1]), hi = max(v[k], v[k + 1]);
            v[k] = lo;
            v[k + 1] = hi;
        }
#pragma unroll
    for (int k = 0; k < SEG_REG; k++)
        if (k < n) p[k] = v[k];
}

__global__ void __launch_bounds__(TPB) k_segsort(DevPlan d) {
    step_enter();
    const long long nq = 4 * d.B_total, stride = (long long)gridDim.x * blockDim.x;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += stride) {
        const int n = d.qcounts[q];
        if (n < 2) continue;
        const int s0 = quad_first(d, (int)q);
        if (n > SEG_REG && n <= SEG_CHECK) {  // listed only when out of order
            bool sorted = true;
            int prev = d.perm[s0];
            for (int k0 = 1; k0 < n && sorted; k0 += 8) {
                int v[8];
#pragma unroll
                for (int k = 0; k < 8; k++) v[k] = k0 + k < n ? d.perm[s0 + k0 + k] : 0x7FFFFFFF;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    sorted &= prev < v[k] || k0 + k >= n;
                    prev = v[k];
                }
            }
            if (sorted) continue;
        }
        if (n > SEG_LANES) {  // listed from the far end of the same array
            const unsigned k = atomicAdd(&d.glob->nhuge, 1u);
            d.bigseg[d.bigseg_cap - 1 - k] = make_int2(s0, n);
            continue;
        }
        if (n > SEG_REG) {
            const unsigned k = atomicAdd(&d.glob->nbig, 1u);
            d.bigseg[k] = make_int2(s0, n);
            continue;
        }
        seg_thread(d.perm + s0, n);
    }
}

// Ascending sort of the warp's 32 R values (element 32 r + lane in v[r]): a bitonic network, strides
// below 32 by shuffles, the others between a lane's registers.
template <int R>
__device__ __forceinline__ void warp_bitonic(int v[R]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32 * R; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1)
#pragma unroll
            for (int r = 0; r < R; r++) {
                const bool up = ((32 * r + lane) & size) == 0;
                if (stride >= 32) {
                    const int q = r ^ (stride >> 5);
                    if (q > r) {
                        const int lo = min(v[r], v[q]), hi = max(v[r], v[q]);
                        v[r] = up ? lo : hi;
                        v[q] = up ? hi : lo;
                    }
                } else {
                    const int o = __shfl_xor_sync(0xffffffffu, v[r], stride);
                    v[r] = up == ((lane & stride) == 0) ? min(v[r], o) : max(v[r], o);
                }
            }
}

// a stretch of n <= 32 R entries in registers; left alone when its slots were handed out in order
template <int R>
__device__ __forceinline__ void seg_regs(int *p, int n) {
    const int lane = threadIdx.x & 31;
    int v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = 32 * r + lane < n ? p[32 * r + lane] : 0x7FFFFFFF;
    bool sorted = true;  // (padding sorts after every index)
#pragma unroll
    for (int r = 0; r < R; r++) {
        int nx = __shfl_down_sync(0xffffffffu, v[r], 1);
        if (r + 1 < R) {
            const int first = __shfl_sync(0xffffffffu, v[r + 1], 0);
            if (lane == 31) nx = first;
        } else if (lane == 31) {
            nx = 0x7FFFFFFF;
        }
        sorted &= v[r] <= nx;
    }
    if (__all_sync(0xffffffffu, sorted)) return;
    warp_bitonic<R>(v);
#pragma unroll
    for (int r = 0; r < R; r++)
        if (32 * r + lane < n) p[32 * r + lane] = v[r];
}

// Ascending sort of src[0 .. n) by a CTA of NT threads: four stable 8-bit radix passes src -> dst ->
// src -> dst -> src.
template <int NT>
struct RadixScratch {
    int hist[256], base[256], run[256], wcnt[NT / 32][256];
};

template <int NT>
__device__ void cta_radix_sort(int *src, int *dst, int n, RadixScratch<NT> &rs) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int pass = 0; pass < 4; pass++) {
        const int sh = 8 * pass;
        for (int k = tid; k < 256; k += NT) {
            rs.hist[k] = 0;
            rs.run[k] = 0;
        }
        __syncthreads();
        for (int k = tid; k < n; k += NT) atomicAdd(&rs.hist[(src[k] >> sh) & 255], 1);
        __syncthreads();
        if (warp == 0) {
            int own[8], sum = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                own[k] = sum;
                sum += rs.hist[8 * lane + k];
            }
            int before = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += u;
            }
#pragma unroll
            for (int k = 0; k < 8; k++) rs.base[8 * lane + k] = before - sum + own[k];
        }
        __syncthreads();
        for (int c0 = 0; c0 < n; c0 += NT) {
            const int k = c0 + tid;
            const bool ok = k < n;
            const int v = ok ? src[k] : 0;
            const int dg = ok ? (v >> sh) & 255 : 256 + lane;  // invalid lanes match nobody
            for (int q = tid; q < (NT / 32) * 256; q += NT) (&rs.wcnt[0][0])[q] = 0;
            __syncthreads();
            const unsigned peers = __match_any_sync(0xffffffffu, dg);
            const int rank = __popc(peers & ((1u << lane) - 1u));
            if (ok && rank == 0) rs.wcnt[warp][dg] = __popc(peers);
            __syncthreads();
            if (ok) {
                int pos = rs.base[dg] + rs.run[dg] + rank;
                for (int q = 0; q < warp; q++) pos += rs.wcnt[q][dg];
                dst[pos] = v;
            }
            __syncthreads();
            for (int q = tid; q < 256; q += NT) {
                int t = 0;
                for (int ww = 0; ww < NT / 32; ww++) t += rs.wcnt[ww][q];
                rs.run[q] += t;
            }
            __syncthreads();
        }
        int *t = src;
        src = dst;
        dst = t;
        __threadfence_block();
        __syncthreads();
    }
}

// Long stretches.  Up to SEG_LANES entries a warp sorts in its registers (batches of small boxes in
// file order have most of theirs here: 27.3M particles 670 -> 344 us, against a shared-memory
// network).  Up to SEG_MERGE a CTA sorts runs of SEG_LANES that way and merges them pairwise in shared
// memory, each entry finding its place in the other run by binary search; longer ones take the radix
// passes.  (One warp on a shared-memory network took 45 us for a single stretch of 257 to 512
// entries, the longest chain of the tree build wherever boxes are dense: a whole step of 131,071
// Gaussian particles on 40 x 40 boxes 648 -> 605 us, of 500,000 on 79 x 79 1,889 -> 1,840.)
constexpr int SEG_MERGE = 4096;

__device__ __forceinline__ void seg_warp(int *p, int n) {  // n <= SEG_LANES
    if (n <= 32) seg_regs<1>(p, n);
    else if (n <= 64) seg_regs<2>(p, n);
    else if (n <= 128) seg_regs<4>(p, n);
    else seg_regs<8>(p, n);
}

template <int NT>
union LongScratch {
    RadixScratch<NT> rs;
    int run[2][SEG_MERGE];
};

// Ascending sort of the n distinct entries at p by a CTA of NT threads (tmp: n entries of scratch,
// used beyond SEG_MERGE).
template <int NT>
__device__ void cta_sort(int *p, int *tmp, int n, LongScratch<NT> &ls) {
    if (n > SEG_MERGE) {
        cta_radix_sort<NT>(p, tmp, n, ls.rs);
        return;
    }
    constexpr int R = SEG_LANES / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int m = SEG_LANES;
    while (m < n) m <<= 1;
    int *a = ls.run[0], *b = ls.run[1];
    // a stretch whose slots the atomics happened to hand out in input order is done already (the
    // common case when the input is the previous step's order)
    bool sorted = true;
    for (int k = tid; k < n; k += NT) {
        const int v = p[k];
        sorted &= k == 0 || p[k - 1] < v;
    }
    if (__syncthreads_and(sorted)) return;
    for (int c = warp; c < m / SEG_LANES; c += NT / 32) {
        int v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int k = SEG_LANES * c + 32 * r + lane;
            v[r] = k < n ? p[k] : 0x7FFFFFFF;
        }
        warp_bitonic<R>(v);
#pragma unroll
        for (int r = 0; r < R; r++) a[SEG_LANES * c + 32 * r + lane] = v[r];
    }
    __syncthreads();
    for (int w = SEG_LANES; w < m; w <<= 1) {
        for (int k = tid; k < m; k += NT) {
            // the entry's place: its own in its run, plus the entries of the other run before it
            // (equal ones, all padding, count for the right run only: every place is taken once)
            const int v = a[k], right = k & w;
            const int *o = a + ((k & ~(2 * w - 1)) | (right ^ w));
            int lo = 0;
            for (int h = w >> 1; h > 0; h >>= 1) lo += (right ? o[lo + h - 1] <= v : o[lo + h - 1] < v) ? h : 0;
            lo += (right ? o[lo] <= v : o[lo] < v) ? 1 : 0;
            b[(k & ~(2 * w - 1)) + (k & (w - 1)) + lo] = v;
        }
        __syncthreads();
        int *t = a;
        a = b;
        b = t;
    }
    for (int k = tid; k < n; k += NT) p[k] = a[k];
    __syncthreads();  // the runs are the next stretch's
}

__global__ void __launch_bounds__(TPB) k_segsort_big(DevPlan d) {
    step_enter();
    __shared__ LongScratch<TPB> ls;
    const int warp = threadIdx.x >> 5;
    const unsigned nhuge = d.glob->nhuge;
    for (unsigned b = blockIdx.x; b < nhuge; b += gridDim.x) {  // a CTA each
        const int2 sg = d.bigseg[d.bigseg_cap - 1 - b];
        cta_sort<TPB>(d.perm + sg.x, d.slot + sg.x, sg.y, ls);
    }
    const unsigned nbig = d.glob->nbig;
    for (unsigned e = (unsigned)(blockIdx.x * (TPB / 32) + warp); e < nbig; e += gridDim.x * (TPB / 32)) {  // a warp each
        const int2 sg = d.bigseg[e];
        seg_warp(d.perm + sg.x, sg.y);
    }
}

// The leaf-moment terms of one particle (offsets from its box origin, mass), the segmented scan
// of a warp's chunk of 32 box-sorted particles and the write of its sums: the box inside the
// chunk gets its FP64 moments in mom, a box that starts before the chunk leaves its part in the
// chunk's head partial, one that runs past it in the tail partial (k_summarize adds a multi-chunk
// box's partials in chunk order).  The products are rounded one by one (no contraction), so the
// fused pass in k_gather and the stand-alone k_leaf give the same sums.  The second moments
// (Sxx, Sxy, Syy) are summed only with SECOND (a plan with the learned correction, or training
// pairs on demand); otherwise they are zeros.
template <bool SECOND>
__device__ __forceinline__ void leaf_terms(float ox, float oy, float mf, float v[6]) {
    v[0] = mf;
    v[1] = __fmul_rn(mf, ox);
    v[2] = __fmul_rn(mf, oy);
    v[3] = SECOND ? __fmul_rn(v[1], ox) : 0.f;
    v[4] = SECOND ? __fmul_rn(v[1], oy) : 0.f;
    v[5] = SECOND ? __fmul_rn(v[2], oy) : 0.f;
}

// key: the lane's box (-1 past the end); c: the chunk (its first particle is 32 c)
template <bool SECOND>
__device__ __forceinline__ void leaf_chunk(const DevPlan &d, long long c, int key, float v[6]) {
    constexpr int NL = SECOND ? 6 : 3;  // moments summed
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int k2 = __shfl_up_sync(0xffffffffu, key, o);
#pragma unroll
        for (int q = 0; q < NL; q++) {
            const float y = __shfl_up_sync(0xffffffffu, v[q], o);
            if (lane >= o && k2 == key) v[q] = __fadd_rn(v[q], y);
        }
    }
    const int knext = __shfl_down_sync(0xffffffffu, key, 1);
    const int kfirst = __shfl_sync(0xffffffffu, key, 0);
    const bool last = key >= 0 && (lane == 31 || knext != key);  // the segment's last lane
    if (!last) return;
    const long long i0 = c << 5;
    const bool head = key == kfirst && d.box_start[key] < i0;              // began in an earlier chunk
    const bool tail = lane == 31 && d.box_start[key + 1] > i0 + 32;        // goes on in a later chunk
    if (head || tail) {
        float *pt = d.leafpart + 12 * c;
        if (head)
#pragma unroll
            for (int q = 0; q < NL; q++) pt[q] = v[q];
        if (tail)
#pragma unroll
            for (int q = 0; q < NL; q++) pt[6 + q] = v[q];
    } else {
        const int s = find_seg(d.boff_tab, d.nsys, key);
        double *m = d.mom + 6 * (d.sys[s].coff + (key - d.sys[s].boff));
#pragma unroll
        for (int q = 0; q < 6; q++) m[q] = q < NL ? f32_to_f64(v[q]) : 0.0;
    }
}

// Output particle t takes input perm[t]; each warp's 32 consecutive outputs form a leaf chunk,
// whose moments are summed on the spot (the stand-alone k_leaf repeats this from the packed
// records when the leaf moments were overwritten since).
template <bool SECOND>
__global__ void __launch_bounds__(TPB) k_gather(DevPlan d) {
    step_enter();
    const int cur = d.glob->epoch & 1, nxt = cur ^ 1;
    const int lane = threadIdx.x & 31;
    // SU particles per thread per round, each stage's loads issued for all of them before the
    // next stage uses them; the loop runs per warp (its first lane's index), for the scans.
    // Two per round keep the kernel at 64 registers, 4 CTAs per SM (four: 93, 2 CTAs, 9% slower)
    constexpr int SU = 2;
    const long long n = d.n_total, stride = (long long)gridDim.x * blockDim.x;
    // one system (the common case): its grid constants once, no search per particle
    const bool one = d.nsys == 1;
    const int G0 = d.sys[0].G;
    const long long boff0 = d.sys[0].boff, ooff0 = d.sys[0].ooff;
    const bool count_far = n >= STORE_GATHER_MIN;  // for k_store
    unsigned far_pids = 0;  // neighbours whose pids lie far apart (the lane's count)
    for (long long w0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); w0 < n; w0 += SU * stride) {
        const long long t0 = w0 + lane;
        int src[SU], key4[SU];
#pragma unroll
        for (int u = 0; u < SU; u++) {
            const long long t = t0 + u * stride;
            src[u] = t < n ? d.perm[t] : 0;
        }
#pragma unroll
        for (int u = 0; u < SU; u++) {
            const long long t = t0 + u * stride;
            key4[u] = t < n ? d.key[src[u]] : 0;
        }
        double x[SU], y[SU], m[SU], vx[SU], vy[SU];
        int pid[SU];
#pragma unroll
        for (int u = 0; u < SU; u++) {
            const long long t = t0 + u * stride;
            pid[u] = 0;
            if (t < n) {
                const int i = src[u];
                x[u] = d.X[cur][i];
                y[u] = d.Y[cur][i];
                m[u] = d.M[cur][i];
                vx[u] = d.VX[cur][i];
                vy[u] = d.VY[cur][i];
                pid[u] = d.PID[cur][i];
            }
        }
        float lx[SU], ly[SU], lm[SU];
#pragma unroll
        for (int u = 0; u < SU; u++) {
            const long long t = t0 + u * stride;
            lx[u] = ly[u] = lm[u] = 0.f;
            const int pn = count_far ? __shfl_down_sync(0xffffffffu, pid[u], 1) : pid[u];
            if (t >= n) continue;
            if (lane < 31 && t + 1 < n && (unsigned)(pn - pid[u] + STORE_NEAR) > 2u * STORE_NEAR) far_pids++;
            const int key = key4[u] >> 2;
            const int s = one ? 0 : find_seg(d.boff_tab, d.nsys, key);
            const int G = one ? G0 : d.sys[s].G;
            const long long boff = one ? boff0 : d.sys[s].boff, ooff = one ? ooff0 : d.sys[s].ooff;
            const int lb = (int)(key - boff);
            const int kx = lb / G, ky = lb - kx * G;
            d.X[nxt][t] = x[u];
            d.Y[nxt][t] = y[u];
            d.VX[nxt][t] = vx[u];
            d.VY[nxt][t] = vy[u];
            d.M[nxt][t] = m[u];
            d.PID[nxt][t] = pid[u];
            const double *org = d.org + ooff;  // box origins (tabulated by k_place)
            const float ox = f64_to_f32_rn(__dsub_rn(x[u], org[kx]));
            const float oy = f64_to_f32_rn(__dsub_rn(y[u], org[G + ky]));
            const float mf = f64_to_f32_rn(m[u]);
            d.PD[2 * t] = make_float4(ox, ox, oy, oy);
            d.PD[2 * t + 1] = make_float4(mf, mf, __int_as_float((int)t), __int_as_float((kx << 16) | ky));
            d.skey[t] = key;
            lx[u] = ox;
            ly[u] = oy;
            lm[u] = mf;
        }
#pragma unroll
        for (int u = 0; u < SU; u++) {
            const long long wu = w0 + u * stride;  // the chunk's first particle
            if (wu >= n) break;                    // (warp-uniform)
            const long long t = wu + lane;
            float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (t < n) leaf_terms<SECOND>(lx[u], ly[u], lm[u], v);
            leaf_chunk<SECOND>(d, wu >> 5, t < n ? key4[u] >> 2 : -1, v);
        }
    }
    if (count_far) {
        far_pids = __reduce_add_sync(0xffffffffu, far_pids);
        if (lane == 0 && far_pids) atomicAdd(&d.glob->far_pids, far_pids);
    }
}

// ---------------------------------------------------------------- summarize
// One CTA per tile of SUM_TILE x SUM_TILE leaf boxes: the boxes' moments (M, Sx, Sy, Sxx, Sxy,
// Syy about the box origin; k_gather summed them per chunk of 32 box-sorted particles), then
// pyramid levels 1..4 inside the tile, then the cell records of all of them.  Above the tiles
// (cells of 2^5 boxes and larger) a cell is built by the CTA that finishes its last child: each
// cell counts its children's arrivals, so the levels above rise along a reduction tree instead of
// waiting for one CTA.  Every sum runs in a fixed order, so the moments do not depend on
// scheduling.  Pyramid cells carry the second moments only for the learned correction (SECOND);
// the leaves always carry all six.
constexpr int SUM_THREADS = 128;  // 7 CTAs per SM: the 1,024 tiles of G = 512 in one wave
constexpr int SUM_CELLS = 256 + 64 + 16 + 4 + 1;  // a tile's cells at levels 0..4
constexpr int SUM_UP = 5;                         // the first level above the tiles (2^5 boxes)
static_assert(SUM_TILE == 1 << (SUM_UP - 1), "a tile is one cell of level SUM_UP - 1");

// The moments of child (a, b) of a level-l cell (q, FP64 about the child's origin) shifted to the
// cell origin, into o[6] (o[0..2] without SECOND); zeros when the child lies outside the grid.
template <bool SECOND>
__device__ __forceinline__ void child_terms(const double *q, bool has, int a, int b, int l, double step,
                                            double *o) {
    if (!has) {
#pragma unroll
        for (int k = 0; k < 6; k++) o[k] = 0.0;
        return;
    }
    const double dx = (double)(a << (l - 1)) * step, dy = (double)(b << (l - 1)) * step;
    const double M = q[0], Sx = q[1], Sy = q[2];
    o[0] = M;
    o[1] = Sx + M * dx;
    o[2] = Sy + M * dy;
    if (SECOND) {
        o[3] = q[3] + 2.0 * dx * Sx + M * dx * dx;
        o[4] = q[4] + dx * Sy + dy * Sx + M * dx * dy;
        o[5] = q[5] + 2.0 * dy * Sy + M * dy * dy;
    }
}

// a cell's four shifted children added in (0, 0), (0, 1), (1, 0), (1, 1) order
template <bool SECOND>
__device__ __forceinline__ void sum_children(const double *t, double *p) {
#pragma unroll
    for (int k = 0; k < (SECOND ? 6 : 3); k++) p[k] = ((t[k] + t[6 + k]) + t[12 + k]) + t[18 + k];
}

// Float records of cell c (level l): centre of mass relative to the cell origin and mass; with
// SECOND, the second moments about the centre of mass normalised by M s^2.
template <bool SECOND>
__device__ __forceinline__ void cell_record(const DevPlan &d, long long c, int l, double step,
                                            const double *q) {
    const double M = q[0];
    if (M > 0.0) {
        const double cx = q[1] / M, cy = q[2] / M;
        d.rec[c] = make_float4(f64_to_f32_rn(cx), f64_to_f32_rn(cy), f64_to_f32_rn(M), 0.f);
        if (SECOND) {
            const double sz = (double)(1 << l) * step;
            const double nrm = 1.0 / (M * sz * sz);
            const double ixx = q[3] - q[1] * cx, ixy = q[4] - q[1] * cy, iyy = q[5] - q[2] * cy;
            d.rec2[c] = make_float4(f64_to_f32_rn(ixx * nrm), f64_to_f32_rn(ixy * nrm),
                                    f64_to_f32_rn(iyy * nrm), 0.f);
        }
    } else {
        d.rec[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (SECOND) d.rec2[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Leaf moments from the packed records, balanced over the particles: a warp per chunk of 32
// box-sorted particles (k_gather does the same while it writes the records; this pass runs when
// the leaf moments have been overwritten since, bh_set_leaf_moments).  No atomics: fixed
// summation order.
template <bool SECOND>
__global__ void __launch_bounds__(TPB) k_leaf(DevPlan d) {
    const int lane = threadIdx.x & 31;
    const long long nch = (d.n_total + 31) >> 5;
    for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nch;
         c += ((long long)gridDim.x * blockDim.x) >> 5) {
        const long long i = (c << 5) + lane;
        int key = -1;
        float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (i < d.n_total) {
            key = d.skey[i];
            const float4 pxy = d.PD[2 * i], pm = d.PD[2 * i + 1];  // (x, x, y, y), (m, m, ., .)
            leaf_terms<SECOND>(pxy.x, pxy.z, pm.x, v);
        }
        leaf_chunk<SECOND>(d, c, key, v);
    }
}

// (s, c) += x, Kahan-compensated in FP32
__device__ __forceinline__ void kahan_add(float &s, float &c, float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}

// The moments of box lb of a system into m (6 values) and mom: a box inside one chunk has them from
// the chunk's sums; a box over several chunks adds its partials in chunk order.
template <bool SECOND>
__device__ __forceinline__ void leaf_sum(const DevPlan &d, const SysDesc &sd, long long lb, double *m) {
    constexpr int NM = SECOND ? 6 : 3;
    const int i0 = d.box_start[sd.boff + lb], i1 = d.box_start[sd.boff + lb + 1];
    double *mb = d.mom + 6 * (sd.coff + lb);
    if (i1 == i0) {  // empty: zeros
#pragma unroll
        for (int q = 0; q < 6; q++) m[q] = mb[q] = 0.0;
        return;
    }
    const long long c0 = i0 >> 5, c1 = (long long)(i1 - 1) >> 5;
    if (c0 == c1) {
#pragma unroll
        for (int q = 0; q < 6; q++) m[q] = mb[q];
        return;
    }
    float sm_[6], cc_[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        sm_[q] = q < NM ? d.leafpart[12 * c0 + 6 + q] : 0.f;
        cc_[q] = 0.f;
    }
    for (long long c = c0 + 1; c <= c1; c++)
#pragma unroll
        for (int q = 0; q < NM; q++) kahan_add(sm_[q], cc_[q], d.leafpart[12 * c + q]);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const double v = f32_to_f64(__fsub_rn(sm_[q], cc_[q]));
        m[q] = v;
        mb[q] = v;
    }
}

// One tile by a CTA of NT threads.  leaf_records: also the records of the boxes.  leaves_given: the leaf moments are already in d.mom
// (bh_set_leaf_moments); build the rest.  cm: the tile's cells, level by level (SUM_CELLS x 6); chm:
// shifted child moments, 64 cells x 4 children (x 6).
template <bool SECOND, int NT>
__device__ __forceinline__ void summarize_tile(const DevPlan &d, long long t, int leaves_given, bool leaf_records, double *cm,
                                               double *chm) {
    constexpr int NM = SECOND ? 6 : 3;  // moments a pyramid cell carries
    const int tid = threadIdx.x;
    const int loff[5] = {0, 256, 320, 336, 340};
    {
        const int s = find_seg(d.toff_tab, d.nsys, t);
        const SysDesc &sd = d.sys[s];
        const double step = d.dyn[s].step;
        const int G = sd.G, lt = (int)(t - sd.toff), ti = lt / sd.tps, tj = lt - ti * sd.tps;
        const int bx0 = ti * SUM_TILE, by0 = tj * SUM_TILE;
        const int nbx = min(SUM_TILE, G - bx0), nby = min(SUM_TILE, G - by0);
        const int lmax = min(SUM_UP - 1, sd.L - 1);  // the tile's top level
        // ---- level 0: the tile's boxes (zeros outside the grid)
        for (int k = tid; k < 6 * SUM_TILE * SUM_TILE; k += NT) {
            const int box = k / 6, cx = box / SUM_TILE, cy = box - cx * SUM_TILE;
            double v = 0.0;
            if (leaves_given && cx < nbx && cy < nby)
                v = d.mom[6 * (sd.coff + (long long)(bx0 + cx) * G + (by0 + cy)) + (k - 6 * box)];
            cm[k] = v;
        }
        __syncthreads();
        if (!leaves_given) {
            // a box inside one chunk has its moments from the chunk's sums; a box over several
            // chunks adds its partials in chunk order (the first chunk's tail, whole middle
            // chunks, the last chunk's head) and writes the sum to mom, as an empty box its zeros
            for (int k = tid; k < SUM_TILE * SUM_TILE; k += NT) {
                const int cx = k / SUM_TILE, cy = k - cx * SUM_TILE;
                if (cx >= nbx || cy >= nby) continue;
                leaf_sum<SECOND>(d, sd, (long long)(bx0 + cx) * G + (by0 + cy), cm + 6 * k);
            }
            __syncthreads();
        }
        // ---- levels 1..lmax inside the tile: a thread per (cell, child) shifts the child's
        // moments to the cell origin, then a thread per cell adds its four children in order
        for (int l = 1; l <= lmax; l++) {
            const int nl = SUM_TILE >> l, nc = nl << 1;  // cells per side at l and l - 1
            const int gl = sd.lvg[l], gc = sd.lvg[l - 1];
            const int I0 = bx0 >> l, J0 = by0 >> l;
            for (int t = tid; t < 4 * nl * nl; t += NT) {
                const int cell = t >> 2, a = (t >> 1) & 1, b = t & 1;
                const int ci = cell / nl, cj = cell - ci * nl;
                const bool has = 2 * (I0 + ci) + a < gc && 2 * (J0 + cj) + b < gc;
                child_terms<SECOND>(cm + 6 * (loff[l - 1] + (2 * ci + a) * nc + (2 * cj + b)), has, a, b,
                                    l, step, chm + 6 * t);
            }
            __syncthreads();
            for (int c = tid; c < nl * nl; c += NT) {
                const int ci = c / nl, cj = c - ci * nl;
                const bool inside = I0 + ci < gl && J0 + cj < gl;
                double p[6];
                sum_children<SECOND>(chm + 24 * c, p);
#pragma unroll
                for (int k = 0; k < NM; k++) cm[6 * (loff[l] + c) + k] = inside ? p[k] : 0.0;
                if (inside) {
                    const long long cc = sd.coff + sd.lvoff[l] + (long long)(I0 + ci) * gl + (J0 + cj);
#pragma unroll
                    for (int k = 0; k < NM; k++) d.mom[6 * cc + k] = p[k];
                }
            }
            __syncthreads();
        }
        // ---- records of the tile's cells, all levels at once (a record is a chain of FP64 operations)
        for (int k = leaf_records ? tid : 256 + tid; k < SUM_CELLS; k += NT) {
            const int l = k < 256 ? 0 : k < 320 ? 1 : k < 336 ? 2 : k < 340 ? 3 : 4;
            if (l > lmax) continue;
            const int nl = SUM_TILE >> l, c = k - loff[l], ci = c / nl, cj = c - ci * nl;
            const int gl = sd.lvg[l], I = (bx0 >> l) + ci, J = (by0 >> l) + cj;
            if (I < gl && J < gl)
                cell_record<SECOND>(d, sd.coff + sd.lvoff[l] + (long long)I * gl + J, l, step, cm + 6 * k);
        }
        // ---- above the tiles: the tile's top cell arrives at its parent; the CTA whose child
        // arrives last builds the parent (children in (0, 0), (0, 1), (1, 0), (1, 1) order, the
        // order of sum_children) and arrives at the next level
        if (sd.L > SUM_UP) {
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                int I = ti, J = tj;
                for (int l = SUM_UP; l < sd.L; l++) {
                    I >>= 1;
                    J >>= 1;
                    const int gl = sd.lvg[l], gc = sd.lvg[l - 1];
                    const int nch = (2 * I + 1 < gc ? 2 : 1) * (2 * J + 1 < gc ? 2 : 1);
                    const long long cl = sd.lvoff[l] + (long long)I * gl + J;  // relative to coff
                    unsigned *cnt = d.upcnt + sd.upoff + (cl - sd.lvoff[SUM_UP]);
                    if (atomicAdd(cnt, 1u) != (unsigned)nch - 1u) break;
                    __threadfence();
                    *cnt = 0u;  // ready for the next step
                    double p[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                    for (int a = 0; a < 2; a++)
                        for (int b = 0; b < 2; b++) {
                            const bool has = 2 * I + a < gc && 2 * J + b < gc;
                            double q[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, o[6];
                            if (has) {
                                const double *src =
                                    d.mom + 6 * (sd.coff + sd.lvoff[l - 1] + (long long)(2 * I + a) * gc + (2 * J + b));
#pragma unroll
                                for (int k = 0; k < NM; k++) q[k] = __ldcg(src + k);
                            }
                            child_terms<SECOND>(q, has, a, b, l, step, o);
#pragma unroll
                            for (int k = 0; k < NM; k++) p[k] = (a | b) ? p[k] + o[k] : o[k];
                        }
                    const long long cc = sd.coff + cl;
#pragma unroll
                    for (int k = 0; k < NM; k++) d.mom[6 * cc + k] = p[k];
                    cell_record<SECOND>(d, cc, l, step, p);
                    __threadfence();
                }
            }
        }
        __syncthreads();
    }
}

template <bool SECOND>
__global__ void __launch_bounds__(SUM_THREADS, 7) k_summarize(DevPlan d, int leaves_given) {
    step_enter();
    __shared__ double cm[SUM_CELLS * 6];
    __shared__ double chm[4 * 64 * 6];
    for (long long t = blockIdx.x; t < d.T_total; t += gridDim.x)
        summarize_tile<SECOND, SUM_THREADS>(d, t, leaves_given, true, cm, chm);
}

// ------------------------------------------------------------------ small systems
// create_tree (and, fused into a step, summarize) of one small system as one kernel: a cluster of
// 16 CTAs runs the phases of k_prologue, k_bbox, k_place, the box scan, k_perm, k_segsort and
// k_gather one after another with a cluster barrier between them, and makes the work items.  Bound:
// latency -- a phase is one or two dependent loads for every thread, and a kernel of its own costs three to five microseconds, its launch and its ramp, where a barrier costs
// half of one.  Every result is the same bits: the phases are the same arithmetic over the same chunks,
// and what depends on atomics (slots) is put in input order as in k_segsort.  10,000 particles on
// 16 x 16 boxes, load, step and store: 87 us with the general kernels, 77 with this one; 20,000 in box
// order 142 and 136, in file order 144 and 146; 60,000: 215 and 221 (16 SMs' share of the memory
// system then costs more than the launches), so the line is CL_MAX_N = 16,384 particles.
constexpr int CL_THREADS = 1024;
struct ClusterSmem {
    int start[CL_MAX_BOXES + 1];  // box_start
    SysDyn dyn;
    double org[2][CL_MAX_SIDE];  // box origins
    unsigned long long red[4][CL_THREADS / 32], ext[4];
    unsigned long long items;  // work items of the CTA's groups
    int scan[32], wtot[32], base;
    int nbig;
    union {
        struct {
            int2 big[2048];  // the CTA's long quadrants
            LongScratch<CL_THREADS> ls;
        } sort;
        struct {
            double cm[SUM_CELLS * 6], chm[4 * 64 * 6];
        } sum;
    } u;
};
static_assert(4 * CL_MAX_BOXES <= 2048 * 8 && CL_MAX_SIDE * CL_MAX_SIDE == CL_MAX_BOXES, "eight CTAs or more: 2,048 quadrants each at most");

// Work items of the groups [g0, g1) by one CTA, from item `base` on; returns their number.  WRITE:
// write them (the number alone needs no base).
// Walking plan: k_group_items, its scan and k_fill_items.
template <bool WRITE>
__device__ int cluster_walk_items(const DevPlan &d, ClusterSmem &sm, int g0, int g1, int base) {
    const SysDesc &sd = d.sys[0];
    int sum = 0;
    for (int k0 = g0; k0 < g1; k0 += CL_THREADS) {
        const int g = k0 + threadIdx.x;
        int cnt = 0;
        if (g < g1) {
            const int gi = g / sd.NGs, gj = g - gi * sd.NGs;
            const int gx0 = gi * sd.TG, gy0 = gj * sd.TG, gx1 = min(sd.G, gx0 + sd.TG), gy1 = min(sd.G, gy0 + sd.TG);
            int nt = 0;
            for (int c = gx0; c < gx1; c++) nt += sm.start[c * sd.G + gy1] - sm.start[c * sd.G + gy0];
            cnt = (nt + d.chunk - 1) / d.chunk;
        }
        int tot;
        const int off = base + sum + block_excl_scan(cnt, sm.scan, &tot);
        if (WRITE && g < g1) {
            d.item_cnt[g] = cnt;
            d.item_off[g] = off;
            for (int k = 0; k < cnt; k++) d.item_group[off + k] = g;
        }
        sum += tot;
    }
    return sum;
}

// List streaming: k_sitems, a warp per group, a round per 32 groups.
template <bool WRITE>
__device__ int cluster_stream_items(const DevPlan &d, ClusterSmem &sm, int g0, int g1, int base) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int sum = 0;
    for (int k0 = g0; k0 < g1; k0 += CL_THREADS / 32) {
        const int g = k0 + warp;
        GroupItems gi;
        group_items(d, g < g1 ? g : d.NG_total, gi);
        if (lane == 0) sm.wtot[warp] = gi.total;
        __syncthreads();
        if (warp == 0) {
            const int v = sm.wtot[lane];
            int x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            sm.wtot[lane] = x - v;
            if (lane == 31) sm.base = x;
        }
        __syncthreads();
        if (WRITE && g < g1) group_items_write(d, g, gi, base + sum + sm.wtot[warp]);
        sum += sm.base;
        __syncthreads();
    }
    return sum;
}

__global__ void __launch_bounds__(CL_THREADS, 1) k_tree_cluster(DevPlan d, int summary) {
    step_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem &sm = *reinterpret_cast<ClusterSmem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x, nct = gridDim.x;  // (the grid is one cluster)
    const int gt = rank * CL_THREADS + tid, GT = nct * CL_THREADS;
    const SysDesc &sd = d.sys[0];
    const int n = (int)d.n_total, G = sd.G, B = G * G;
    const unsigned epoch = d.glob->epoch + 1;  // (advanced below, once every CTA has read it)
    const int cur = epoch & 1, nxt = cur ^ 1;
    const double *X = d.X[cur], *Y = d.Y[cur];
    // ---- empty histograms; extents of the CTA's particles
    for (int b = gt; b < B; b += GT) reinterpret_cast<int4 *>(d.qcounts)[b] = make_int4(0, 0, 0, 0);
    unsigned long long e[4] = {~0ull, ~0ull, 0ull, 0ull};
    for (int i = gt; i < n; i += GT) {
        minmax_ord(ord_bits(X[i]), e[0], e[2]);
        minmax_ord(ord_bits(Y[i]), e[1], e[3]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, e[q], o);
            e[q] = q < 2 ? (v < e[q] ? v : e[q]) : (v > e[q] ? v : e[q]);
        }
        if (lane == 0) sm.red[q][warp] = e[q];
    }
    __syncthreads();
    if (warp < 4) {
        unsigned long long v = sm.red[warp][lane];
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
            v = warp < 2 ? (w < v ? w : v) : (w > v ? w : v);
        }
        if (lane == 0) sm.ext[warp] = v;
    }
    if (tid == 0) sm.nbig = 0;
    cluster_sync();
    // ---- the square box, by every CTA for itself; CTA 0 publishes it
    if (warp == 0) {
        unsigned long long v = ld_cluster(&sm.ext[lane >> 3], lane & 7);
        if (nct > 8) {  // 8 or 16 CTAs
            const unsigned long long w = ld_cluster(&sm.ext[lane >> 3], 8 + (lane & 7));
            v = lane < 16 ? (w < v ? w : v) : (w > v ? w : v);
        }
#pragma unroll
        for (int o = 4; o; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
            v = lane < 16 ? (w < v ? w : v) : (w > v ? w : v);
        }
        if ((lane & 7) == 0) (lane < 16 ? sm.dyn.bbmin : sm.dyn.bbmax)[(lane >> 3) & 1] = v;
        __syncwarp();
        if (lane == 0) {
            bbox_finalize_sys(d, 0, sm.dyn);
            if (rank == 0) {
                d.dyn[0] = sm.dyn;
                d.glob->epoch = epoch;
                d.glob->near_pairs = 0;
                d.glob->far_pairs = 0;
                d.glob->corr_pairs = 0;
                d.glob->far_pids = 0;
            }
        }
    }
    __syncthreads();
    const SysDyn &dy = sm.dyn;
    if (tid < 2 * G) sm.org[tid >= G][tid >= G ? tid - G : tid] = box_origin(tid >= G ? dy.miny : dy.minx, tid >= G ? tid - G : tid, dy.step);
    // ---- keys and slots (a run of equal keys in a warp shares an addition)
    for (int i0 = gt - lane; i0 < n; i0 += GT) {
        const int i = i0 + lane;
        int key = -1;
        if (i < n) {
            const double x = X[i], y = Y[i];
            const unsigned hx = (unsigned)(__double_as_longlong(x) >> 52) & 0x7FFu;
            const unsigned hy = (unsigned)(__double_as_longlong(y) >> 52) & 0x7FFu;
            if (hx == 0x7FFu || hy == 0x7FFu) raise_err(d.glob, 1u /*BH_DEV_NAN_POSITION*/);
            const int k2x = half_key1_f32(x, dy.minx, dy.step, dy.inv_step, dy.minx_f, dy.inv_step_f, dy.key_tol, G);
            const int k2y = half_key1_f32(y, dy.miny, dy.step, dy.inv_step, dy.miny_f, dy.inv_step_f, dy.key_tol, G);
            key = 4 * ((k2x >> 1) * G + (k2y >> 1)) + (k2x & 1) * 2 + (k2y & 1);
        }
        const int kp = __shfl_up_sync(0xffffffffu, key, 1);
        const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != kp);
        const int h = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));            // the run's first lane
        const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
        const int len = later ? __ffs(later) : 32 - lane;                          // (at its first lane)
        int s0 = 0;
        if (lane == h && key >= 0) s0 = atomicAdd(&d.qcounts[key], len);
        s0 = __shfl_sync(0xffffffffu, s0, h);
        if (i < n) {
            d.key[i] = key;
            d.slot[i] = s0 + lane - h;
        }
    }
    cluster_sync();
    // ---- box scan, by every CTA for itself; CTA 0 publishes it
    {
        constexpr int PER = (CL_MAX_BOXES + CL_THREADS - 1) / CL_THREADS;
        int v[PER], sum = 0;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int b = tid * PER + q;
            int4 c = make_int4(0, 0, 0, 0);
            if (b < B) c = reinterpret_cast<const int4 *>(d.qcounts)[b];
            v[q] = c.x + c.y + c.z + c.w;
            sum += v[q];
        }
        int pre = block_excl_scan(sum, sm.scan, nullptr);
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int b = tid * PER + q;
            if (b <= B) {  // (past the last box: the total)
                sm.start[b] = pre;
                if (rank == 0) d.box_start[b] = pre;
            }
            pre += v[q];
        }
        if (tid == CL_THREADS - 1 && PER * CL_THREADS == B) {
            sm.start[B] = pre;
            if (rank == 0) d.box_start[B] = pre;
        }
    }
    __syncthreads();
    // ---- permutation
    auto first = [&](int key4) {
        const int4 qc = reinterpret_cast<const int4 *>(d.qcounts)[key4 >> 2];
        const int quad = key4 & 3;
        return sm.start[key4 >> 2] + (quad > 0 ? qc.x : 0) + (quad > 1 ? qc.y : 0) + (quad > 2 ? qc.z : 0);
    };
    for (int i = gt; i < n; i += GT) d.perm[first(d.key[i]) + d.slot[i]] = i;
    cluster_sync();
    // ---- the CTA's groups (CTA 0, which has a pyramid to build, takes none) and their work items
    const int ng = (int)d.NG_total, per = (ng + nct - 2) / (nct - 1);
    const int ig0 = min(ng, max(0, rank - 1) * per), ig1 = rank == 0 ? ig0 : min(ng, rank * per);
    {
        const int c = d.stream ? cluster_stream_items<false>(d, sm, ig0, ig1, 0) : cluster_walk_items<false>(d, sm, ig0, ig1, 0);
        if (tid == 0) sm.items = (unsigned long long)c;
    }
    // ---- each quadrant's stretch in input order
    for (int q = tid * nct + rank; q < 4 * B; q += GT) {  // (every CTA takes its share of a few)
        const int cnt = d.qcounts[q];
        if (cnt < 2) continue;
        const int s0 = first(q);
        if (cnt > SEG_REG) {
            sm.u.sort.big[atomicAdd(&sm.nbig, 1)] = make_int2(s0, cnt);
            continue;
        }
        seg_thread(d.perm + s0, cnt);
    }
    __syncthreads();
    {
        const int nbig = sm.nbig;
        for (int k = warp; k < nbig; k += CL_THREADS / 32) {
            const int2 sg = sm.u.sort.big[k];
            if (sg.y > SEG_LANES) continue;
            seg_warp(d.perm + sg.x, sg.y);
        }
        for (int k = 0; k < nbig; k++) {
            const int2 sg = sm.u.sort.big[k];
            if (sg.y > SEG_LANES) cta_sort<CL_THREADS>(d.perm + sg.x, d.slot + sg.x, sg.y, sm.u.sort.ls);
        }
    }
    cluster_sync();
    int item_base = 0;  // (every thread)
    for (int r = 0; r < rank; r++) item_base += (int)ld_cluster(&sm.items, r);
    // ---- gather the state, sum the leaves
    {
        for (int w0 = gt - lane; w0 < n; w0 += GT) {
            const int t = w0 + lane;
            int key = -1;
            float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (t < n) {
                const int i = d.perm[t];
                key = d.key[i] >> 2;
                const double x = X[i], y = Y[i], m = d.M[cur][i];
                const int kx = key / G, ky = key - kx * G;
                d.X[nxt][t] = x;
                d.Y[nxt][t] = y;
                d.VX[nxt][t] = d.VX[cur][i];
                d.VY[nxt][t] = d.VY[cur][i];
                d.M[nxt][t] = m;
                d.PID[nxt][t] = d.PID[cur][i];
                const float ox = f64_to_f32_rn(__dsub_rn(x, sm.org[0][kx]));
                const float oy = f64_to_f32_rn(__dsub_rn(y, sm.org[1][ky]));
                const float mf = f64_to_f32_rn(m);
                d.PD[2 * t] = make_float4(ox, ox, oy, oy);
                d.PD[2 * t + 1] = make_float4(mf, mf, __int_as_float(t), __int_as_float((kx << 16) | ky));
                d.skey[t] = key;
                leaf_terms<false>(ox, oy, mf, v);
            }
            leaf_chunk<false>(d, w0 >> 5, key, v);
        }
    }
    cluster_sync();
    if (summary) {
        // ---- summarize: the boxes' moments and records over all CTAs, then the tiles' pyramids
        for (int b = tid * nct + rank; b < B; b += GT) {
            double m[6];
            leaf_sum<false>(d, sd, b, m);
            cell_record<false>(d, sd.coff + b, 0, dy.step, m);
        }
        cluster_sync();
        for (int t = rank; t < (int)d.T_total; t += nct)
            summarize_tile<false, CL_THREADS>(d, t, 1, false, sm.u.sum.cm, sm.u.sum.chm);
    }
    // ---- the work items, which nothing here waits for
    if (d.stream) cluster_stream_items<true>(d, sm, ig0, ig1, item_base);
    else cluster_walk_items<true>(d, sm, ig0, ig1, item_base);
    if (rank == nct - 1 && tid == 0) (d.stream ? d.sitem_off : d.item_off)[ng] = item_base + (int)sm.items;
}

// ------------------------------------------------------------------ launches
// Launch of k_tree_cluster: 16 CTAs where the device keeps a cluster that large, else 8.
static cudaError_t cluster_config(cudaLaunchConfig_t &c, cudaLaunchAttribute a[2], int ctas, cudaStream_t st) {
    memset(&c, 0, sizeof(c));
    memset(a, 0, 2 * sizeof(a[0]));
    a[0].id = cudaLaunchAttributeClusterDimension;
    a[0].val.clusterDim.x = ctas;
    a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
    a[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (launch_step)
    a[1].val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = dim3(ctas);
    c.blockDim = dim3(CL_THREADS);
    c.dynamicSmemBytes = sizeof(ClusterSmem);
    c.stream = st;
    c.attrs = a;
    c.numAttrs = 2;
    return cudaSuccess;
}
cudaError_t tree_init(int *ctas) {
    cudaError_t e = cudaFuncSetAttribute(k_tree_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClusterSmem));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_tree_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t c;
    cudaLaunchAttribute a[2];
    cluster_config(c, a, 16, nullptr);
    int fit = 0;
    *ctas = cudaOccupancyMaxActiveClusters(&fit, k_tree_cluster, &c) == cudaSuccess && fit > 0 ? 16 : 8;
    cudaGetLastError();
    return cudaSuccess;
}
cudaError_t launch_tree_cluster(const DevPlan &d, bool summary, cudaStream_t st) {
    cudaLaunchConfig_t c;
    cudaLaunchAttribute a[2];
    cluster_config(c, a, d.cl_ctas, st);
    return cudaLaunchKernelEx(&c, k_tree_cluster, d, summary ? 1 : 0);
}
cudaError_t launch_prologue(const DevPlan &d, cudaStream_t st) {
    long long n = d.B_total > d.nsys ? d.B_total : d.nsys;
    launch_step(k_prologue, grid_for(n, TPB, d.nsm * 16LL), TPB, 0, st, d);
    return cudaGetLastError();
}
cudaError_t launch_bbox(const DevPlan &d, cudaStream_t st) {
    if (d.n_total == 0) return cudaSuccess;
    // (a block per 2,048 particles at least: its five atomics meet every other block's)
    launch_step(k_bbox, grid_for(d.n_total, TPB * (d.nsys == 1 ? 8 : 16), d.nsm * (d.nsys == 1 ? 4LL : 8LL)), TPB, 0, st,
                d);
    return cudaGetLastError();
}
cudaError_t launch_place(const DevPlan &d, cudaStream_t st) {
    if (d.n_total == 0) return cudaSuccess;
    launch_step(k_place, grid_for(d.n_total, TPB * PLACE_PP, d.nsm * 8LL), TPB, 0, st, d);
    return cudaGetLastError();
}
cudaError_t launch_scan(const DevPlan &d, cudaStream_t st) {
    return scan_excl(d.qcounts, d.box_start, d.B_total, d.sst_box, d.glob, 0, st, true);
}
// Work items of the walk kernel and the learned correction, or of the pair generator (group, target chunk).
cudaError_t launch_walk_items(const DevPlan &d, cudaStream_t st) {
    unsigned g = grid_for(d.NG_total, TPB, d.nsm * 8LL);
    k_group_items<<<g, TPB, 0, st>>>(d);
    cudaError_t e = scan_excl(d.item_cnt, d.item_off, d.NG_total, d.sst_witem, d.glob, 1, st);
    if (e != cudaSuccess) return e;
    launch_step(k_fill_items, g, TPB, 0, st, d);
    return cudaGetLastError();
}
// The step's work items: the walk items where the walk or the learned correction runs, the
// list-streaming items where the lists are streamed (a streaming plan builds walk items only
// with the learned correction, or on demand for bh_learned_pairs; so does a plan with FP64 pairs
// the generator's).
cudaError_t launch_items(const DevPlan &d, cudaStream_t st) {
    cudaError_t e;
    if (!d.stream || d.learned) {
        e = launch_walk_items(d, st);
        if (e == cudaSuccess && d.learned && d.pchunk != d.chunk) e = launch_walk_items(pair_items(d), st);
        if (e != cudaSuccess) return e;
    }
    if (d.stream && d.NG_total > 0) {
        k_sitems<<<(unsigned)((d.NG_total + SITEM_TILE - 1) / SITEM_TILE), SITEM_WARPS * 32, 0, st>>>(d);
    }
    return cudaGetLastError();
}
// The stream waits for `join` (the work items, on another stream) before the gather, so that whatever
// follows the tree waits for one kernel; the gather itself, which waits for two, is launched plainly.
cudaError_t launch_scatter(const DevPlan &d, cudaEvent_t join, cudaStream_t st) {
    if (d.n_total == 0) return cudaStreamWaitEvent(st, join, 0);
    launch_step(k_perm, grid_for(d.n_total, TPB, d.nsm * 8LL), TPB, 0, st, d);
    launch_step(k_segsort, grid_for(4 * d.B_total, TPB, d.nsm * 8LL), TPB, 0, st, d);
    launch_step(k_segsort_big, (unsigned)(d.nsm * 4), TPB, 0, st, d);
    const cudaError_t e = cudaStreamWaitEvent(st, join, 0);
    if (e != cudaSuccess) return e;
    if (d.learned) k_gather<true><<<grid_for(d.n_total, TPB, d.nsm * 8LL), TPB, 0, st>>>(d);
    else k_gather<false><<<grid_for(d.n_total, TPB, d.nsm * 8LL), TPB, 0, st>>>(d);
    return cudaGetLastError();
}
// leaves: the leaf sums of k_gather were overwritten since (bh_set_leaf_moments): redo them
cudaError_t launch_summarize(const DevPlan &d, bool leaves, cudaStream_t st) {
    if (leaves && d.n_total > 0) {
        const unsigned g = grid_for((d.n_total + 31) / 32, TPB / 32, d.nsm * 8LL);
        if (d.learned) k_leaf<true><<<g, TPB, 0, st>>>(d);
        else k_leaf<false><<<g, TPB, 0, st>>>(d);
    }
    // the second moments of the pyramid cells feed only the learned correction
    const unsigned g = grid_for(d.T_total, 1, d.nsm * 8LL);
    auto k = d.learned ? k_summarize<true> : k_summarize<false>;
    if (d.n_total > 0) launch_step(k, g, SUM_THREADS, 0, st, d, 0);
    else k<<<g, SUM_THREADS, 0, st>>>(d, 0);  // (a tree without particles ends on the join)
    return cudaGetLastError();
}
cudaError_t launch_pyramid(const DevPlan &d, cudaStream_t st, bool second) {
    const unsigned g = grid_for(d.T_total, 1, d.nsm * 8LL);
    if (second && !d.learned) {
        // a plan without the learned correction sums no second moments: the leaves again from
        // the particles with them, then the pyramid
        if (d.n_total > 0) k_leaf<true><<<grid_for((d.n_total + 31) / 32, TPB / 32, d.nsm * 8LL), TPB, 0, st>>>(d);
        k_summarize<true><<<g, SUM_THREADS, 0, st>>>(d, 0);
    } else if (d.learned) {
        k_summarize<true><<<g, SUM_THREADS, 0, st>>>(d, 1);
    } else {
        k_summarize<false><<<g, SUM_THREADS, 0, st>>>(d, 1);
    }
    return cudaGetLastError();
}

}  // namespace bh
