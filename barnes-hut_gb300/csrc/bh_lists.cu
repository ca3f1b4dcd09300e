// bh_lists.cu -- interaction lists of every target group, for the list-streaming force kernel.
//
// The reference evaluates every box against its 3 x 3 neighbourhood and the centre of mass of
// every other box (kernels/grid_decomposition/gpu/grid.py:116-157,
// sequential/evaluation.py:73-109); in theta mode this project replaces the flat far field with
// a walk of the cell pyramid, and this kernel does that walk once per target group instead of
// once per work item.  One warp per group (grid-stride over groups) walks the pyramid level by
// level, each lane testing a frontier cell per round: a cell whose centre of mass lies at distance d
// from the group's box rectangle is accepted when s^2 < theta^2 d^2 (s = cell edge) and goes to the
// far list, a rejected leaf goes to the near list, any other rejected cell opens into its children.
// Ballots (a warp scan where a level's last row or column has fewer children) place the entries in
// frontier order, so list order is deterministic and matches the walking force kernel's; the test is
// the same FP32 arithmetic, so both paths accept the same cells.
//
// Output per group g of system s: far entries (the accepted cell's centre of mass in the group
// frame, as the opening test computed it, and its mass) at lfar[s.lfoff + lg * s.lfcap ..]; near
// descriptors -- (first particle, exclusive prefix of the boxes' particle counts, box-origin shift in
// the group frame) and (box index, mass, centre of mass in the group frame) -- at lnear[s.lnoff + lg *
// 2 * (s.lncap + 1) ..] with the total in descriptor [count]; lcnt[g] = (far count, near count).  The slots are
// sized on the host so that a level's accepted cells never exceed FRONTIER_CAP; the kernel still
// checks and raises BH_DEV_LIST_OVERFLOW.
#include "bh_internal.cuh"
#include "bh_pairs.cuh"

namespace bh {

constexpr int LW = 4;  // warps per list-building CTA; one warp walks one group
// CTAs per SM (56 registers): the walk is bound by its instructions and their latency together.  1,048,576
// particles, four steps: 3,773 us with twelve (40 registers, which spill), 3,749 with ten, 3,717 with eight
constexpr int LISTS_MINB = 8;

__global__ void __launch_bounds__(LW * 32, LISTS_MINB) k_lists(DevPlan d) {
    step_enter();
    __shared__ __align__(16) int front[LW][2][FR_CAP];  // cells as x << 16 | y; near boxes as indices
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int(*fb)[FR_CAP] = front[warp];
    const float theta2 = d.theta2_f;
    const unsigned lt_mask = (1u << lane) - 1u;
    if (blockIdx.x == 0 && threadIdx.x < 2 * ITEM_BUCKETS) d.item_bucket[threadIdx.x] = 0;  // (for the item order)
    for (long long g = (long long)blockIdx.x * LW + warp; g < d.NG_total; g += (long long)gridDim.x * LW) {
        const int s = find_seg(d.goff_tab, d.nsys, g);
        const SysDesc &sd = d.sys[s];
        const SysDyn &dy = d.dyn[s];
        const long long lg = g - sd.goff;
        const int TG = sd.TG;
        const int gi = (int)(lg / sd.NGs), gj = (int)(lg - (long long)gi * sd.NGs);
        const int gx0 = gi * TG, gy0 = gj * TG;
        const int gx1 = min(sd.G, gx0 + TG), gy1 = min(sd.G, gy0 + TG);
        const float step_f = __double2float_rn(dy.step);
        const float W_f = __fmul_rn((float)TG, step_f);
        float4 *far_out = d.lfar + sd.lfoff + lg * sd.lfcap;
        int4 *near_out = d.lnear + sd.lnoff + lg * 2 * (sd.lncap + 1);
        int nfar = 0, nnear = 0, nfr = 1, cur = 0;
        bool ovf = false;
        __syncwarp();  // the previous group is done with front[]
        if (lane == 0) fb[0][0] = 0;
        __syncwarp();
        for (int l = sd.L - 1; l >= 0 && nfr > 0; l--) {
            const int gl = sd.lvg[l];
            const int gc = l > 0 ? sd.lvg[l - 1] : 0;
            const float s_f = ldexpf(step_f, l);
            const float s2 = __fmul_rn(s_f, s_f);
            const int *fr = fb[cur];
            int *fn = fb[cur ^ 1];  // next frontier; at the leaf level, the near boxes
            // the cells over the group's rectangle; and whether every cell has its four children
            const int ox0 = gx0 >> l, ox1 = (gx1 - 1) >> l, oy0 = gy0 >> l, oy1 = (gy1 - 1) >> l;
            const bool full = gc == 2 * gl;
            const float4 *rec = d.rec + sd.coff + sd.lvoff[l];
            int nnext = 0;
            for (int q0 = 0; q0 < nfr; q0 += 32) {
                const int q = q0 + lane;
                int ci = 0, cj = 0, kind = 0;
                float rx = 0.f, ry = 0.f;  // centre of mass in the group frame
                float4 rr = make_float4(0.f, 0.f, 0.f, 0.f);
                if (q < nfr) {
                    const int c = fr[q];
                    ci = c >> 16;
                    cj = c & 0xFFFF;
                    if ((unsigned)ci >= (unsigned)gl || (unsigned)cj >= (unsigned)gl)
                        raise_err(d.glob, 4u /*BH_DEV_BAD_KEY*/);  // never expected: skip it
                    else
                        rr = rec[ci * gl + cj];
                    if (rr.z > 0.f) {
                        bool accept = false;
                        if (ci < ox0 || ci > ox1 || cj < oy0 || cj > oy1) {
                            rx = __fadd_rn(__fmul_rn(small_int_f((ci << l) - gx0), step_f), rr.x);
                            ry = __fadd_rn(__fmul_rn(small_int_f((cj << l) - gy0), step_f), rr.y);
                            const float dxo = fmaxf(0.f, fmaxf(-rx, __fsub_rn(rx, W_f)));
                            const float dyo = fmaxf(0.f, fmaxf(-ry, __fsub_rn(ry, W_f)));
                            const float d2 = __fadd_rn(__fmul_rn(dxo, dxo), __fmul_rn(dyo, dyo));
                            accept = s2 < __fmul_rn(theta2, d2);
                        }
                        kind = accept ? 1 : (l == 0 ? 2 : 3);
                    }
                }
                // append in frontier order
                const unsigned mf = __ballot_sync(0xffffffffu, kind == 1);
                const unsigned mo = __ballot_sync(0xffffffffu, kind >= 2);  // (a level has near boxes or opened cells)
                if (kind == 1) {
                    const int pos = nfar + __popc(mf & lt_mask);
                    if (pos < sd.lfcap) far_out[pos] = make_float4(rx, ry, rr.z, 0.f);
                }
                nfar += __popc(mf);
                if (l == 0) {
                    if (kind == 2) {
                        const int pos = nnear + __popc(mo & lt_mask);
                        if (pos < sd.lncap) fn[pos] = ci * gl + cj;
                    }
                    nnear += __popc(mo);
                } else if (full) {
                    const int pos = nnext + 4 * __popc(mo & lt_mask), c0 = (ci << 17) | (cj << 1);
                    if (kind == 3 && pos + 4 <= FR_CAP)
                        *reinterpret_cast<int4 *>(fn + pos) = make_int4(c0, c0 + 1, c0 + 65536, c0 + 65537);
                    nnext += 4 * __popc(mo);
                } else {
                    const bool bx = 2 * ci + 1 < gc, by = 2 * cj + 1 < gc;  // second children along x, y
                    const int nch = kind == 3 ? (bx ? 2 : 1) * (by ? 2 : 1) : 0;
                    int inc = nch;  // inclusive warp scan of the children counts
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, inc, o);
                        if (lane >= o) inc += y;
                    }
                    int pos = nnext + inc - nch;
                    if (nch && pos + nch <= FR_CAP) {
                        const int c0 = (ci << 17) | (cj << 1);
                        fn[pos++] = c0;
                        if (by) fn[pos++] = c0 + 1;
                        if (bx) fn[pos++] = c0 + 65536;
                        if (bx && by) fn[pos++] = c0 + 65537;
                    }
                    nnext += __shfl_sync(0xffffffffu, inc, 31);
                }
                if (nnext > FR_CAP) ovf = true;
            }
            __syncwarp();  // the next frontier (or the near list) is complete
            cur ^= 1;
            // an overflowed frontier may hold unwritten slots: abandon the walk (flagged)
            nfr = ovf ? 0 : nnext;
        }
        // near descriptors: first particle, exclusive prefix of the particle counts, box shift.
        // The near boxes were appended at the leaf level into the buffer that is now fb[cur]
        // (children in (0, 0), (0, 1), (1, 0), (1, 1) order, so a pair of boxes of one column
        // often follows each other: the force kernel copies such a run at once).
        const int nn = min(nnear, sd.lncap);
        const int *nl = fb[cur];
        int base = 0;
        for (int k0 = 0; k0 <= nn; k0 += 32) {
            const int k = k0 + lane, loc = k < nn ? nl[k] : 0;
            int st = 0, c = 0;
            float4 rr = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < nn) {
                st = d.box_start[sd.boff + loc];
                c = d.box_start[sd.boff + loc + 1] - st;
                rr = d.rec[sd.coff + loc];  // the leaf's record (level 0)
            }
            int inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            const int pre = base + inc - c;
            if (k < nn) {
                const int kx = loc / sd.G, ky = loc - kx * sd.G;
                const float shx = __fmul_rn(small_int_f(kx - gx0), step_f), shy = __fmul_rn(small_int_f(ky - gy0), step_f);
                near_out[2 * k] = make_int4(st, pre, __float_as_int(shx), __float_as_int(shy));
                near_out[2 * k + 1] = make_int4(loc, __float_as_int(rr.z), __float_as_int(__fadd_rn(shx, rr.x)),
                                                __float_as_int(__fadd_rn(shy, rr.y)));
            } else if (k == nn) {
                near_out[2 * k] = make_int4(0, pre, 0, 0);
                near_out[2 * k + 1] = make_int4(0, 0, 0, 0);
            }
            base += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) {
            if (ovf || nfar > sd.lfcap || nnear > sd.lncap) raise_err(d.glob, 2u /*BH_DEV_LIST_OVERFLOW*/);
            d.lcnt[g] = make_int2(min(nfar, sd.lfcap), nn);
        }
    }
}

// ---------------------------------------------------------------- heaviest-first item order
// A warp of the force kernel owns one work item, so an item's duration grows with its pair count
// and the launch ends with its slowest warp.  Items are therefore handed out heaviest first:
// bucket b holds the items whose estimated cost (STREAM_CHUNK / slices) x (near sources + 2 x far
// cells) lies in [2^b, 2^(b+1)); buckets are laid out from the top down.  Order inside a bucket
// follows atomic arrival, which changes only which warp evaluates an item, not its result.
__device__ __forceinline__ int item_cost_bucket(const DevPlan &d, long long item) {
    const long long g = d.sitem_group[item];
    const int sub = d.sitem_sub[item];
    const int2 ck = d.sitem_chunk[item];
    const int s = find_seg(d.goff_tab, d.nsys, g);
    const SysDesc &sd = d.sys[s];
    const long long lg = g - sd.goff;
    const int2 cnt = d.lcnt[g];
    const int near_total = d.lnear[sd.lnoff + lg * 2 * (sd.lncap + 1) + 2 * cnt.y].y;
    const int gi = (int)(lg / sd.NGs), gj = (int)(lg - (long long)gi * sd.NGs);
    const int gx0 = gi * sd.TG, gy0 = gj * sd.TG;
    const int gx1 = min(sd.G, gx0 + sd.TG), gy1 = min(sd.G, gy0 + sd.TG);
    const int nbox = sd.TG * sd.TG;
    int nt = 0;  // the item's target set: a quadrant, one dense box, or the group's sparse boxes
    for (int c = gx0; c < gx1; c++)
        for (int r = gy0; r < gy1; r++) {
            const long long b = sd.boff + (long long)c * sd.G + r;
            const int nb = d.box_start[b + 1] - d.box_start[b];
            const int bi = (c - gx0) * sd.TG + (r - gy0);
            if (sub >= nbox) {
                if (bi == (sub - nbox) >> 2) nt += d.qcounts[4 * b + ((sub - nbox) & 3)];
            } else if (sub >= 0 ? bi == sub : box_item_kind(nb, d.dense_min, d.quad_min) == 0) {
                nt += nb;
            }
        }
    int c0, T;
    sitem_range(nt, ck.x, &c0, &T);
    // a sweep of T targets runs 32 / ceil(T / FORCE_R) slices; cost in full-warp target units
    const int nslice = 32 / max(1, (T + FORCE_R - 1) / FORCE_R);
    const unsigned long long cost =
        (unsigned long long)(STREAM_CHUNK / nslice) * (unsigned long long)(near_total + 2 * cnt.x) + 1ull;
    const int b = 63 - __clzll((long long)cost);
    return min(b, ITEM_BUCKETS - 1);
}

__global__ void __launch_bounds__(256) k_item_hist(DevPlan d) {
    step_enter();
    __shared__ int h[ITEM_BUCKETS];
    if (threadIdx.x < ITEM_BUCKETS) h[threadIdx.x] = 0;
    __syncthreads();
    const long long nitems = d.sitem_off[d.NG_total];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nitems; i += (long long)gridDim.x * blockDim.x) {
        const int b = item_cost_bucket(d, i);
        d.item_cost[i] = (unsigned char)b;  // for k_item_order
        atomicAdd(&h[b], 1);
    }
    __syncthreads();
    if (threadIdx.x < ITEM_BUCKETS && h[threadIdx.x]) atomicAdd(&d.item_bucket[threadIdx.x], h[threadIdx.x]);
}

__global__ void __launch_bounds__(256) k_item_order(DevPlan d) {
    step_enter();
    __shared__ int off[ITEM_BUCKETS], h[ITEM_BUCKETS], base[ITEM_BUCKETS];
    if (threadIdx.x == 0) {
        int o = 0;
        for (int b = ITEM_BUCKETS - 1; b >= 0; b--) {  // heaviest bucket first
            off[b] = o;
            o += d.item_bucket[b];
        }
    }
    if (threadIdx.x < ITEM_BUCKETS) h[threadIdx.x] = 0;
    __syncthreads();
    const long long nitems = d.sitem_off[d.NG_total];
    const long long stride = (long long)gridDim.x * blockDim.x;
    // one pass of the grid per round; each round reserves a range per bucket for its block
    for (long long r0 = (long long)blockIdx.x * blockDim.x; r0 < nitems; r0 += stride) {
        const long long i = r0 + threadIdx.x;
        int b = -1, rank = 0;
        if (i < nitems) {
            b = d.item_cost[i];
            rank = atomicAdd(&h[b], 1);
        }
        __syncthreads();
        if (threadIdx.x < ITEM_BUCKETS) {
            base[threadIdx.x] = h[threadIdx.x] ? atomicAdd(&d.item_bucket[ITEM_BUCKETS + threadIdx.x], h[threadIdx.x]) : 0;
            h[threadIdx.x] = 0;
        }
        __syncthreads();
        if (b >= 0) d.item_order[off[b] + base[b] + rank] = (int)i;
        __syncthreads();
    }
}

// Both of the above for a few items, by one CTA (a launch less; 10,000 particles: 6.1 us against the
// pair's 5.6 and 4.3).
constexpr int ORDER_THREADS = 1024, ORDER_MAX = 8192;

__global__ void __launch_bounds__(ORDER_THREADS) k_item_order_few(DevPlan d) {
    step_enter();
    __shared__ int h[ITEM_BUCKETS], cur[ITEM_BUCKETS];
    __shared__ unsigned char cost[ORDER_MAX];
    const int tid = threadIdx.x;
    if (tid < ITEM_BUCKETS) h[tid] = 0;
    __syncthreads();
    const int nitems = d.sitem_off[d.NG_total];  // <= ORDER_MAX (launch_lists)
    for (int i = tid; i < nitems; i += ORDER_THREADS) {
        const int b = item_cost_bucket(d, i);
        cost[i] = (unsigned char)b;
        atomicAdd(&h[b], 1);
    }
    __syncthreads();
    if (tid < ITEM_BUCKETS) {
        int o = 0;
        for (int b = ITEM_BUCKETS - 1; b > tid; b--) o += h[b];  // heaviest bucket first
        cur[tid] = o;
        d.item_bucket[tid] = h[tid];  // (stream_split)
    }
    __syncthreads();
    for (int i = tid; i < nitems; i += ORDER_THREADS) d.item_order[atomicAdd(&cur[cost[i]], 1)] = i;
}

cudaError_t launch_lists(const DevPlan &d, cudaStream_t st) {
    if (d.NG_total == 0) return cudaSuccess;
    long long grid = (long long)d.nsm * LISTS_MINB;
    if (grid * LW > d.NG_total) grid = (d.NG_total + LW - 1) / LW;
    launch_step(k_lists, (unsigned)grid, LW * 32, 0, st, d);
    const long long items_max = d.NG_total + d.n_total / d.dense_min +
                                (d.quad_min > 0 ? 4 * (d.n_total / d.quad_min) : 0) + d.n_total / STREAM_ITEM_DIV + 1;  // >= items
    if (list_kernels(items_max) == 2) {
        launch_step(k_item_order_few, 1, ORDER_THREADS, 0, st, d);
        return cudaGetLastError();
    }
    long long ig = (items_max + 255) / 256;
    if (ig > (long long)d.nsm * 8) ig = (long long)d.nsm * 8;
    launch_step(k_item_hist, (unsigned)ig, 256, 0, st, d);
    launch_step(k_item_order, (unsigned)ig, 256, 0, st, d);
    return cudaGetLastError();
}

int list_kernels(long long items_max) { return items_max <= ORDER_MAX ? 2 : 3; }

}  // namespace bh
