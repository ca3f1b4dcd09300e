// bh_force.cu -- box-tiled force evaluation by a walk of the cell pyramid per work item.
//
// Replaces g_evaluate_boxes (python-bh/barneshut/kernels/grid_decomposition/gpu/grid.py:116-157,
// with d_self_self_grav / d_self_other_grav / d_self_COM_grav at :211-268); the tick
// (g_tick_particles, gpu/grid.py:159-174) is a kernel of its own here (launch_force).  The
// interaction semantics follow the reference CPU path
// (kernels/grid_decomposition/sequential/evaluation.py:73-109 with
// kernels/gravity/cpu_numba.py:30-92) in flat mode, and this project's opening-angle rule in
// theta mode.
//
// Work decomposition: a target group is TG x TG leaf boxes; its nt targets are split into work
// items of at most TARGET_CHUNK targets (TARGET_CHUNK64 with FP64 pairs; built after the box scan),
// which CTAs pull from a device queue, so dense groups spread over many SMs.  Per item the CTA walks
// the cell pyramid level by level (every thread tests one frontier cell; accepted cells, rejected
// leaves and children are compacted with a block scan, so list order is deterministic), stages far
// entries (centre of mass in the group frame, mass) and near-box particles (shifted into the group
// frame) in shared memory, and evaluates them: each thread owns R targets in registers and sweeps a
// slice of the staged entries (one shared-memory load feeds R pair interactions).  Lists that outgrow
// shared memory are evaluated and emptied on the fly; slice partials are reduced in shared memory.
//
// Pair arithmetic: a += m_j (x_j - x_t) * rcp(r^2 + eps^2) in FP32 (rcp.approx), far-field
// contributions Kahan-compensated when requested; BH_PREC_FP64 runs the same lists in FP64.
// Positions are box-relative offsets rounded once from FP64, so dx keeps ~1e-7 of a box edge.
#include "bh_internal.cuh"
#include "bh_pairs.cuh"
#include "bh_tc.cuh"

namespace bh {

template <typename R> struct Src;
template <> struct Src<float> { using T = float4; };  // (FP32 entries are two records, see below)
template <> struct Src<double> { struct T { double x, y, m; int idx, pad; }; };


__device__ __forceinline__ void src_get(const Src<double>::T &e, double &x, double &y, double &m,
                                        int &idx) {
    x = e.x; y = e.y; m = e.m; idx = e.idx;
}


// bytes per staged far entry: the FP64 record, or (x, x, y, y) + (M, M) in FP32
template <typename R> __host__ __device__ constexpr int far_bytes() {
    return sizeof(typename Src<R>::T) > 24 ? (int)sizeof(typename Src<R>::T) : 24;
}
// bytes per staged near source: the FP64 record, or the 32-byte PD record (x, x, y, y), (m, m, i, box)
template <typename R> __host__ __device__ constexpr int src_bytes() {
    return sizeof(typename Src<R>::T) > 32 ? (int)sizeof(typename Src<R>::T) : 32;
}

// A work item's T targets are dealt to threads in quads, nthr = ceil(T / 4) of them, and the sources
// to nslice = FT / nthr slices: a thread sums one slice's sources for its targets, in order.  NR
// targets per thread: with NR = 4 a CTA serves a whole item; with NR = 2 an item is two CTAs' work,
// each taking half of every quad with the same slices, so every sum runs over the same terms in the
// same order and the results are the same bits.  A plan whose items do not fill the chip takes
// NR = 2 (launch_force).
template <typename R, int NR, bool KAHAN, bool TEST, bool EXACT, int MINB>
__global__ void __launch_bounds__(FT, MINB)
k_force(DevPlan d, int accumulate) {
    step_enter();
    using S = typename Src<R>::T;
    constexpr bool F32 = sizeof(R) == 4;
    constexpr int PARTS = FORCE_R / NR;  // CTAs per item
    static_assert(NR % 2 == 0 && FORCE_R % NR == 0, "targets in packed pairs");
    extern __shared__ __align__(16) unsigned char smem[];
    S *far = reinterpret_cast<S *>(smem);                     // FAR_CAP x far_bytes<R>()
    float2 *farm = reinterpret_cast<float2 *>(reinterpret_cast<float4 *>(far) + FAR_CAP);
    S *src = reinterpret_cast<S *>(smem + FAR_CAP * far_bytes<R>());  // SRC_CAP x src_bytes<R>()
    __shared__ uint64_t s_mbar;  // bulk-copy completion of the near-source staging
    R *red = reinterpret_cast<R *>(smem);                     // aliases far/src at the end
    float2 *nshift = reinterpret_cast<float2 *>(reinterpret_cast<unsigned char *>(src) +
                                                SRC_CAP * src_bytes<R>());  // NEAR_CAP
    int *nbox = reinterpret_cast<int *>(nshift + NEAR_CAP);   // first particle of near box
    int *ncnt = nbox + NEAR_CAP;
    int *npre = ncnt + NEAR_CAP;                              // NEAR_CAP + 4
    int *front0 = npre + NEAR_CAP + 4;                        // FR_CAP
    int *front1 = front0 + FR_CAP;                            // FR_CAP
    __shared__ int sh_scan[32];
    __shared__ int s_item;
    __shared__ int s_col0[MAX_TG + 1], s_colpre[MAX_TG + 1];

    const int tid = threadIdx.x;
    const int nxt = (d.glob->epoch + 1) & 1;
    const double *Xs = d.X[nxt], *Ys = d.Y[nxt], *Ms = d.M[nxt];
    const long long nitems = d.item_off[d.NG_total];
    unsigned long long npairs = 0, fpairs = 0;  // counted by thread 0
    uint32_t tphase = 0;                        // parity of s_mbar's current phase
    bool tma_ok = true;  // block-uniform; cleared (and flagged) when a staging wait times out
    if (F32) {
        if (tid == 0) {
            tc::mbar_init(&s_mbar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
    }

    // Half items are few: a CTA's first one is its own index, so that they spread over all SMs.  Taken from the
    // queue, they went to the CTAs that started first: 100,003 particles on 12 x 12 boxes, flat, 576 of them to
    // 115 of 152 SMs, the round 472 us against 385 without a cutoff, 542 against 460 with one; 131,072 clustered
    // on 16 x 16 boxes, theta 0.5, 2,900 against 1,949.  Not for whole items (130,000 on 24 x 24: 494 and 534).
    constexpr bool SPREAD = PARTS > 1;
    for (bool first = SPREAD;; first = false) {
        if (tid == 0)
            s_item = first ? (int)blockIdx.x : (int)((SPREAD ? gridDim.x : 0u) + atomicAdd(&d.glob->item_next, 1u));
        __syncthreads();
        const int item = s_item / PARTS, part = s_item - item * PARTS;
        if (item >= nitems) break;
        const long long g = d.item_group[item];
        const int chunk = item - d.item_off[g];
        const int s = find_seg(d.goff_tab, d.nsys, g);
        const SysDesc &sd = d.sys[s];
        const SysDyn &dy = d.dyn[s];
        const long long lg = g - sd.goff;
        const int TG = sd.TG, G = sd.G;
        const int gi = (int)(lg / sd.NGs), gj = (int)(lg - (long long)gi * sd.NGs);
        const int gx0 = gi * TG, gy0 = gj * TG;
        const int gx1 = min(G, gx0 + TG), gy1 = min(G, gy0 + TG);
        const int ncol = gx1 - gx0;
        if (tid < ncol) {
            long long b0 = sd.boff + (long long)(gx0 + tid) * G + gy0;
            int st = d.box_start[b0];
            s_col0[tid] = st;
            s_colpre[tid + 1] = d.box_start[b0 + (gy1 - gy0)] - st;
        }
        __syncthreads();
        if (tid == 0) {
            s_colpre[0] = 0;
            for (int c = 1; c <= ncol; c++) s_colpre[c] += s_colpre[c - 1];
        }
        __syncthreads();
        // list counters: block-uniform registers, advanced by every thread from the
        // block scan's totals (no shared counter, no extra barrier)
        int nfar = 0, nnear = 0, nnext = 0;
        bool ovf = false;
        const int nt = s_colpre[ncol];
        int c0, T;
        item_range(nt, d.item_cnt[g], chunk, &c0, &T);
        const float step_f = __double2float_rn(dy.step);
        const float W_f = __fmul_rn((float)TG, step_f);
        const double gox = box_origin(dy.minx, gx0, dy.step), goy = box_origin(dy.miny, gy0, dy.step);
        const R eps2 = (R)(sizeof(R) == 4 ? (double)d.eps2_f : d.eps2);
        const R cut = (R)(sizeof(R) == 4 ? (double)d.cut_f : d.cutoff);

        // ---- thread -> (slice, NR targets)
        const int nthr = (T + FORCE_R - 1) / FORCE_R;
        const int nslice = FT / nthr;
        const bool active = tid < nslice * nthr;
        const int slice = active ? tid / nthr : 0, tl = active ? tid % nthr : 0;
        int ti[NR];
        R tx[NR], ty[NR];
        bool tv[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            int v = tl * FORCE_R + part * NR + r;
            tv[r] = v < T;
            int u = c0 + (tv[r] ? v : 0), c = 0;
            while (c + 1 < ncol && s_colpre[c + 1] <= u) c++;
            ti[r] = s_col0[c] + (u - s_colpre[c]);
            if (sizeof(R) == 4) {
                const float4 p = d.PD[2 * (long long)ti[r]];  // (x, x, y, y) box-relative
                int lb = d.skey[ti[r]] - (int)sd.boff;
                int kx = lb / G, ky = lb - kx * G;
                tx[r] = (R)__fadd_rn(__fmul_rn((float)(kx - gx0), step_f), p.x);
                ty[r] = (R)__fadd_rn(__fmul_rn((float)(ky - gy0), step_f), p.z);
            } else {
                tx[r] = (R)(Xs[ti[r]] - gox);
                ty[r] = (R)(Ys[ti[r]] - goy);
            }
        }
        R anx[NR], any_[NR], afx[NR], afy[NR], acx[NR], acy[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) anx[r] = any_[r] = afx[r] = afy[r] = acx[r] = acy[r] = 0;
        // packed near-field state: negated target coordinates and accumulators, pairs of targets
        f2_t ntx2[NR / 2], nty2[NR / 2], nax2[NR / 2], nay2[NR / 2];
        // packed far-field sums and Kahan compensations
        f2_t fsx2[NR / 2], fsy2[NR / 2], fcx2[NR / 2], fcy2[NR / 2];
        const f2_t eps2x2 = f2_pack((float)eps2, (float)eps2);
        const f2_t m1x2 = f2_pack(-1.f, -1.f);
        if (F32) {
#pragma unroll
            for (int k = 0; k < NR / 2; k++) {
                ntx2[k] = f2_pack(-(float)tx[2 * k], -(float)tx[2 * k + 1]);
                nty2[k] = f2_pack(-(float)ty[2 * k], -(float)ty[2 * k + 1]);
                nax2[k] = nay2[k] = f2_pack(0.f, 0.f);
                fsx2[k] = fsy2[k] = fcx2[k] = fcy2[k] = f2_pack(0.f, 0.f);
            }
        }

        // FP64: 1 / (r^2 + eps^2), zero where the cutoff predicate on the unsoftened r^2 fails
        auto pair_inv64 = [&](double dx, double dyy) -> double {
            if (!TEST) return rcp64(dx * dx + (dyy * dyy + (double)eps2));
            const double r2 = dx * dx + dyy * dyy;
            const double inv = rcp64(r2 + (double)eps2);
            return r2 > (double)cut ? inv : 0.0;
        };
        // FP32, two targets: the same; near a cutoff > 0 (EXACT, sidx >= 0) the predicate is decided
        // on the FP64 positions
        auto pair_inv = [&](f2_t dx, f2_t dyy, int kk, int sidx) -> f2_t {
            if (!TEST) return f2_rcp(f2_fma(dx, dx, f2_fma(dyy, dyy, eps2x2)));
            const f2_t r2 = f2_fma(dx, dx, f2_mul(dyy, dyy));
            float i0, i1, r0, r1;
            f2_unpack(f2_rcp(f2_add(r2, eps2x2)), i0, i1);
            f2_unpack(r2, r0, r1);
            bool k0 = r0 > (float)cut, k1 = r1 > (float)cut;
            if constexpr (EXACT) if (sidx >= 0) {
                const float band = (float)cut * 1e-3f, d0 = fabsf(r0 - (float)cut), d1 = fabsf(r1 - (float)cut);
                if (d0 <= band || d1 <= band) {
                    const double sx = Xs[sidx], sy = Ys[sidx];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int t = ti[2 * kk + h];
                        const double ex = __dsub_rn(Xs[t], sx), ey = __dsub_rn(Ys[t], sy);
                        const bool keep = __dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)) > d.cutoff;
                        if (h == 0 && d0 <= band) k0 = keep;
                        if (h == 1 && d1 <= band) k1 = keep;
                    }
                }
            }
            return f2_pack(k0 ? i0 : 0.f, k1 ? i1 : 0.f);
        };

        // evaluate and empty the far list (entries were written before the last barrier of
        // the block scan that appended them; the next append's scan barriers order the reuse)
        auto flush_far = [&]() {
            __syncthreads();
            const int nf = nfar;
            if (active && F32) {
                const ulonglong2 *fp = reinterpret_cast<const ulonglong2 *>(far);
                const f2_t *fm = reinterpret_cast<const f2_t *>(farm);
#pragma unroll 4
                for (int k = slice; k < nf; k += nslice) {
                    const ulonglong2 rxy = fp[k];  // (rx, rx), (ry, ry)
                    const f2_t mm = fm[k];         // (M, M)
#pragma unroll
                    for (int kk = 0; kk < NR / 2; kk++) {
                        f2_t dx = f2_add(rxy.x, ntx2[kk]), dyy = f2_add(rxy.y, nty2[kk]);
                        f2_t w = f2_mul(mm, pair_inv(dx, dyy, kk, -1));
                        if (KAHAN) {  // y = f - c; t = s + y; c = (t - s) - y; s = t
                            // (with the cutoff test f - c is one fused operation)
                            f2_t yx = TEST ? f2_fma(w, dx, f2_mul(fcx2[kk], m1x2)) : f2_fma(fcx2[kk], m1x2, f2_mul(w, dx));
                            f2_t t1 = f2_add(fsx2[kk], yx);
                            fcx2[kk] = f2_fma(yx, m1x2, f2_fma(fsx2[kk], m1x2, t1));
                            fsx2[kk] = t1;
                            f2_t yy = TEST ? f2_fma(w, dyy, f2_mul(fcy2[kk], m1x2)) : f2_fma(fcy2[kk], m1x2, f2_mul(w, dyy));
                            f2_t t2 = f2_add(fsy2[kk], yy);
                            fcy2[kk] = f2_fma(yy, m1x2, f2_fma(fsy2[kk], m1x2, t2));
                            fsy2[kk] = t2;
                        } else if (TEST) {
                            fsx2[kk] = f2_fma(w, dx, fsx2[kk]);
                            fsy2[kk] = f2_fma(w, dyy, fsy2[kk]);
                        } else {
                            fsx2[kk] = f2_add(fsx2[kk], f2_mul(w, dx));
                            fsy2[kk] = f2_add(fsy2[kk], f2_mul(w, dyy));
                        }
                    }
                }
            } else if (active) {
                for (int k = slice; k < nf; k += nslice) {
                    double sx, sy, sm;
                    int sidx;
                    src_get(reinterpret_cast<const typename Src<double>::T *>(far)[k], sx, sy, sm, sidx);
#pragma unroll
                    for (int r = 0; r < NR; r++) {
                        const double dx = sx - (double)tx[r], dyy = sy - (double)ty[r];
                        const double w = sm * pair_inv64(dx, dyy);
                        afx[r] += (R)(w * dx);
                        afy[r] += (R)(w * dyy);
                    }
                }
            }
            if (part == 0) fpairs += (unsigned long long)T * nf;
            nfar = 0;
        };

        auto flush_near = [&]() {
            __syncthreads();
            const int nn = nnear;
            int total;
            {
                constexpr int IT = NEAR_CAP / FT;
                int v[IT], sum = 0;
#pragma unroll
                for (int k = 0; k < IT; k++) {
                    int e = tid * IT + k;
                    v[k] = e < nn ? ncnt[e] : 0;
                    sum += v[k];
                }
                int pre = block_scan(sum, sh_scan, &total);
#pragma unroll
                for (int k = 0; k < IT; k++) {
                    int e = tid * IT + k;
                    if (e < nn) npre[e] = pre;
                    pre += v[k];
                }
                if (tid == 0) npre[nn] = total;
            }
            __syncthreads();
            for (int s0 = 0; s0 < total && tma_ok; s0 += SRC_CAP) {
                const int ns = min(SRC_CAP, total - s0);
                if (F32 && !TEST) {
                    // Bulk copies (TMA) of the 32-byte PD records of every near-box piece
                    // that falls into [s0, s0 + ns), all completing on one mbarrier phase.
                    if (tid == 0) tc::mbar_expect_tx(&s_mbar, (uint32_t)ns * 32u);
                    tc::fence_async_smem();
                    unsigned char *sbase = reinterpret_cast<unsigned char *>(src);
                    for (int k = tid; k < nn; k += FT) {
                        const int lo = max(npre[k], s0), hi = min(npre[k] + ncnt[k], s0 + ns);
                        if (lo < hi)
                            tc::bulk_g2s(sbase + 32 * (lo - s0), d.PD + 2 * (long long)(nbox[k] + (lo - npre[k])),
                                         (uint32_t)(hi - lo) * 32u, &s_mbar);
                    }
                    const bool ok = tc::mbar_wait(&s_mbar, tphase);
                    tphase ^= 1u;
                    if (!__syncthreads_and(ok ? 1 : 0)) {
                        // flagged; give the copies in flight a second bounded wait, then stage
                        // nothing more in this launch (the barrier phase is no longer known)
                        if (tid == 0) raise_err(d.glob, 8u /*BH_DEV_WAIT_TIMEOUT*/);
                        tc::mbar_wait(&s_mbar, tphase ^ 1u);
                        tma_ok = false;
                        __syncthreads();
                        break;
                    }
                    // a slice takes an equal contiguous range [j0, j1) of the staged sources and
                    // walks the boxes it overlaps; each box's shift is folded into the targets
                    const int per = (ns + nslice - 1) / nslice;
                    const int j0 = min(ns, slice * per), j1 = min(ns, j0 + per);
                    if (active && j0 < j1) {
                        const float4 *s4 = reinterpret_cast<const float4 *>(src);
                        int k = 0;
                        {
                            int hi = nn;  // npre[k] <= s0 + j0 < npre[hi]
                            while (hi - k > 1) {
                                const int mid = (k + hi) >> 1;
                                if (npre[mid] <= s0 + j0) k = mid; else hi = mid;
                            }
                        }
                        for (int lo = j0; lo < j1 && k < nn; k++) {
                            const int hi = min(npre[k] + ncnt[k] - s0, j1);
                            if (lo >= hi) continue;
                            const float2 sh = nshift[k];
                            const f2_t shx = f2_pack(sh.x, sh.x), shy = f2_pack(sh.y, sh.y);
                            f2_t bx[NR / 2], by[NR / 2];
#pragma unroll
                            for (int kk = 0; kk < NR / 2; kk++) {
                                bx[kk] = f2_add(ntx2[kk], shx);
                                by[kk] = f2_add(nty2[kk], shy);
                            }
#pragma unroll 2
                            for (int j = lo; j < hi; j++) {
                                const ulonglong2 sxy = *reinterpret_cast<const ulonglong2 *>(s4 + 2 * j);
                                const f2_t mm = *reinterpret_cast<const f2_t *>(s4 + 2 * j + 1);
#pragma unroll
                                for (int kk = 0; kk < NR / 2; kk++) {
                                    f2_t dx = f2_add(sxy.x, bx[kk]), dyy = f2_add(sxy.y, by[kk]);
                                    f2_t r2 = f2_fma(dx, dx, f2_fma(dyy, dyy, eps2x2));
                                    f2_t w = f2_mul(mm, f2_rcp(r2));
                                    nax2[kk] = f2_fma(w, dx, nax2[kk]);
                                    nay2[kk] = f2_fma(w, dyy, nay2[kk]);
                                }
                            }
                            lo = hi;
                        }
                    }
                    if (part == 0) npairs += (unsigned long long)T * ns;
                    __syncthreads();  // the staging buffer is refilled by the next pass
                    continue;
                }
                for (int j = tid; j < ns; j += FT) {
                    int J = s0 + j;
                    int lo = 0, hi = nn;  // npre[lo] <= J < npre[hi]
                    while (hi - lo > 1) {
                        int mid = (lo + hi) >> 1;
                        if (npre[mid] <= J) lo = mid; else hi = mid;
                    }
                    int idx = nbox[lo] + (J - npre[lo]);
                    if (F32) {  // (x, x, y, y), (m, m, index, -) in the group frame
                        const float4 pxy = d.PD[2 * (long long)idx], pm = d.PD[2 * (long long)idx + 1];
                        const float2 sh = nshift[lo];
                        const float x = __fadd_rn(sh.x, pxy.x), y = __fadd_rn(sh.y, pxy.z);
                        float4 *s4 = reinterpret_cast<float4 *>(src) + 2 * j;
                        s4[0] = make_float4(x, x, y, y);
                        s4[1] = pm;
                    } else {
                        typename Src<double>::T q;
                        q.x = Xs[idx] - gox;
                        q.y = Ys[idx] - goy;
                        q.m = Ms[idx];
                        q.idx = idx;
                        q.pad = 0;
                        reinterpret_cast<typename Src<double>::T *>(src)[j] = q;
                    }
                }
                __syncthreads();
                if (active && F32) {
                    const float4 *s4 = reinterpret_cast<const float4 *>(src);
                    auto sweep1 = [&](int j) {
                        const ulonglong2 sxy = *reinterpret_cast<const ulonglong2 *>(s4 + 2 * j);
                        const ulonglong2 smi = *reinterpret_cast<const ulonglong2 *>(s4 + 2 * j + 1);
                        const int sidx = (int)(unsigned)smi.y;
#pragma unroll
                        for (int kk = 0; kk < NR / 2; kk++) {
                            const f2_t dx = f2_add(sxy.x, ntx2[kk]), dyy = f2_add(sxy.y, nty2[kk]);
                            const f2_t w = f2_mul(smi.x, pair_inv(dx, dyy, kk, sidx));
                            nax2[kk] = f2_fma(w, dx, nax2[kk]);
                            nay2[kk] = f2_fma(w, dyy, nay2[kk]);
                        }
                    };
                    if constexpr (EXACT) {
                        // U sources at a time with the FP32 predicate alone, one branch for all of them:
                        // a group with a pair near the cutoff is swept again, source by source.  A branch
                        // per pair left no two pairs in flight: cutoff 1e-5, flat, 5,000 particles on 3 x 3
                        // boxes 388 -> 202 us, 100,003 on 12 x 12 724 -> 542, 200,000 on 17 x 17 1,320 ->
                        // 787.  (U = 4 | 8 with two targets a thread: 229 | 202 and 581 | 543; 2 | 4 with
                        // four: 788 | 835 at 200,000.)
                        constexpr int U = NR == 2 ? 8 : 2;
                        const float cutf = (float)cut, band = cutf * 1e-3f;
                        int j = slice;
                        for (; j + (U - 1) * nslice < ns; j += U * nslice) {
                            f2_t dx[U][NR / 2], dyy[U][NR / 2], w[U][NR / 2];
                            bool close = false;
#pragma unroll
                            for (int u = 0; u < U; u++) {
                                const float4 *e = s4 + 2 * (j + u * nslice);
                                const ulonglong2 sxy = *reinterpret_cast<const ulonglong2 *>(e);
                                const f2_t mm = *reinterpret_cast<const f2_t *>(e + 1);
#pragma unroll
                                for (int kk = 0; kk < NR / 2; kk++) {
                                    dx[u][kk] = f2_add(sxy.x, ntx2[kk]);
                                    dyy[u][kk] = f2_add(sxy.y, nty2[kk]);
                                    const f2_t r2 = f2_fma(dx[u][kk], dx[u][kk], f2_mul(dyy[u][kk], dyy[u][kk]));
                                    float i0, i1, r0, r1;
                                    f2_unpack(f2_rcp(f2_add(r2, eps2x2)), i0, i1);
                                    f2_unpack(r2, r0, r1);
                                    close |= fabsf(r0 - cutf) <= band;
                                    close |= fabsf(r1 - cutf) <= band;
                                    w[u][kk] = f2_mul(mm, f2_pack(r0 > cutf ? i0 : 0.f, r1 > cutf ? i1 : 0.f));
                                }
                            }
                            if (close) {
#pragma unroll 1
                                for (int u = 0; u < U; u++) sweep1(j + u * nslice);
                                continue;
                            }
#pragma unroll
                            for (int u = 0; u < U; u++)
#pragma unroll
                                for (int kk = 0; kk < NR / 2; kk++) {
                                    nax2[kk] = f2_fma(w[u][kk], dx[u][kk], nax2[kk]);
                                    nay2[kk] = f2_fma(w[u][kk], dyy[u][kk], nay2[kk]);
                                }
                        }
#pragma unroll 1
                        for (; j < ns; j += nslice) sweep1(j);
                    } else {
#pragma unroll 8 / NR
                        for (int j = slice; j < ns; j += nslice) sweep1(j);
                    }
                } else if (active) {
                    for (int j = slice; j < ns; j += nslice) {
                        double sx, sy, sm;
                        int sidx;
                        src_get(reinterpret_cast<const typename Src<double>::T *>(src)[j], sx, sy, sm, sidx);
#pragma unroll
                        for (int r = 0; r < NR; r++) {
                            const double dx = sx - (double)tx[r], dyy = sy - (double)ty[r];
                            const double w = sm * pair_inv64(dx, dyy);
                            anx[r] += (R)(w * dx);
                            any_[r] += (R)(w * dyy);
                        }
                    }
                }
                if (part == 0) npairs += (unsigned long long)T * ns;
                __syncthreads();  // src is restaged by the next pass
            }
            nnear = 0;
        };

        // kind: 0 none, 1 far, 2 near, 3 open (children into front_next).  One block scan
        // places every thread's entries; all threads advance the counters from its total.
        auto emit = [&](int kind, int id, int l, int ci, int cj, float rx, float ry, float M,
                        int *front_next, int gc) {
            int nch = 0;
            if (kind == 3) nch = (2 * ci + 1 < gc ? 2 : 1) * (2 * cj + 1 < gc ? 2 : 1);
            int packed = (kind == 1 ? 1 : 0) | ((kind == 2 ? 1 : 0) << 10) | (nch << 20);
            int tot;
            int pre = block_scan(packed, sh_scan, &tot);
            if (kind == 1) {
                int pos = nfar + (pre & 1023);
                if (sizeof(R) == 4) {
                    reinterpret_cast<float4 *>(far)[pos] = make_float4(rx, rx, ry, ry);
                    farm[pos] = make_float2(M, M);
                } else {
                    const double *q = d.mom + 6 * (long long)id;
                    typename Src<double>::T e;
                    double ox = box_origin(dy.minx, ci << l, dy.step) - gox;
                    double oy = box_origin(dy.miny, cj << l, dy.step) - goy;
                    e.x = ox + q[1] / q[0];
                    e.y = oy + q[2] / q[0];
                    e.m = q[0];
                    e.idx = id;
                    e.pad = 0;
                    reinterpret_cast<typename Src<double>::T *>(far)[pos] = e;
                }
            } else if (kind == 2) {
                int pos = nnear + ((pre >> 10) & 1023);
                int st = d.box_start[id];
                nbox[pos] = st;
                ncnt[pos] = d.box_start[id + 1] - st;
                int lb = id - (int)sd.boff;
                int kx = lb / G, ky = lb - kx * G;
                nshift[pos] = make_float2(__fmul_rn((float)(kx - gx0), step_f),
                                          __fmul_rn((float)(ky - gy0), step_f));
            } else if (kind == 3) {
                int pos = nnext + (pre >> 20);
                if (pos + nch <= FR_CAP) {
                    for (int a = 0; a < 2; a++)
                        for (int b = 0; b < 2; b++)
                            if (2 * ci + a < gc && 2 * cj + b < gc)
                                front_next[pos++] = (2 * ci + a) * gc + (2 * cj + b);
                }
            }
            nfar += tot & 1023;
            nnear += (tot >> 10) & 1023;
            if (nnext + (tot >> 20) > FR_CAP) ovf = true;
            nnext += tot >> 20;
        };

        if (d.flat) {
            const long long B = (long long)G * G;
            for (long long q0 = 0; q0 < B; q0 += FT) {
                if (nfar + FT > FAR_CAP) flush_far();
                if (nnear + FT > NEAR_CAP) flush_near();
                long long b = q0 + tid;
                int kind = 0, bx = 0, byy = 0, id = 0;
                float rx = 0, ry = 0, M = 0;
                if (b < B) {
                    bx = (int)(b / G);
                    byy = (int)(b - (long long)bx * G);
                    long long gb = sd.boff + b;
                    // near boxes by their particles, far boxes by their moments (a plan over one
                    // rank's part of a system holds the other boxes' moments, not their particles)
                    if (abs(bx - gx0) <= 1 && abs(byy - gy0) <= 1) {
                        if (d.box_start[gb + 1] > d.box_start[gb]) {
                            kind = 2;
                            id = (int)gb;
                        }
                    } else {
                        float4 rr = d.rec[sd.coff + b];
                        if (rr.z > 0.f) {
                            rx = __fadd_rn(__fmul_rn((float)(bx - gx0), step_f), rr.x);
                            ry = __fadd_rn(__fmul_rn((float)(byy - gy0), step_f), rr.y);
                            M = rr.z;
                            kind = 1;
                            id = (int)(sd.coff + b);
                        }
                    }
                }
                emit(kind, id, 0, bx, byy, rx, ry, M, front1, 0);
            }
        } else {
            int *fr = front0, *fn = front1;
            if (tid == 0) fr[0] = 0;
            int nfr = 1;
            const float theta2 = d.theta2_f;
            for (int l = sd.L - 1; l >= 0 && nfr > 0; l--) {
                const int gl = sd.lvg[l];
                const int gc = l > 0 ? sd.lvg[l - 1] : 0;
                nnext = 0;
                __syncthreads();  // frontier entries of the previous level are visible
                for (int q0 = 0; q0 < nfr; q0 += FT) {
                    if (nfar + FT > FAR_CAP) flush_far();
                    if (nnear + FT > NEAR_CAP) flush_near();
                    int q = q0 + tid;
                    int kind = 0, ci = 0, cj = 0, id = 0;
                    float rx = 0, ry = 0, M = 0;
                    int loc = q < nfr ? fr[q] : 0;
                    if (q < nfr && (unsigned)loc >= (unsigned)(gl * gl)) {
                        raise_err(d.glob, 4u /*BH_DEV_BAD_KEY*/);  // never expected: skip the cell
                    } else if (q < nfr) {
                        ci = loc / gl;
                        cj = loc - ci * gl;
                        long long cell = sd.coff + sd.lvoff[l] + loc;
                        float4 rr = d.rec[cell];
                        if (rr.z > 0.f) {
                            int lo_x = ci << l, hi_x = (ci + 1) << l;
                            int lo_y = cj << l, hi_y = (cj + 1) << l;
                            bool overlap = lo_x < gx1 && hi_x > gx0 && lo_y < gy1 && hi_y > gy0;
                            bool accept = false;
                            if (!overlap) {
                                rx = __fadd_rn(__fmul_rn((float)(lo_x - gx0), step_f), rr.x);
                                ry = __fadd_rn(__fmul_rn((float)(lo_y - gy0), step_f), rr.y);
                                float dxo = fmaxf(0.f, fmaxf(-rx, __fsub_rn(rx, W_f)));
                                float dyo = fmaxf(0.f, fmaxf(-ry, __fsub_rn(ry, W_f)));
                                float d2 = __fadd_rn(__fmul_rn(dxo, dxo), __fmul_rn(dyo, dyo));
                                float s_f = ldexpf(step_f, l);
                                accept = __fmul_rn(s_f, s_f) < __fmul_rn(theta2, d2);
                            }
                            M = rr.z;
                            if (accept) {
                                kind = 1;
                                id = (int)cell;
                            } else if (l == 0) {
                                kind = 2;
                                id = (int)(sd.boff + loc);
                            } else {
                                kind = 3;
                            }
                        }
                    }
                    emit(kind, id, l, ci, cj, rx, ry, M, fn, gc);
                }
                int *t = fr;
                fr = fn;
                fn = t;
                // an overflowed frontier may hold unwritten slots: abandon the walk
                // (flagged; the host bounds theta and group size so this cannot happen)
                nfr = ovf ? 0 : nnext;
                if (ovf && tid == 0) raise_err(d.glob, 2u /*BH_DEV_LIST_OVERFLOW*/);
            }
        }
        flush_far();
        flush_near();
        __syncthreads();  // the reduction below reuses the staging buffers

        // ---- reduce slice partials and write
        if (F32) {
#pragma unroll
            for (int k = 0; k < NR / 2; k++) {
                float a0, a1, b0, b1;
                f2_unpack(nax2[k], a0, a1);
                f2_unpack(nay2[k], b0, b1);
                anx[2 * k] = (R)a0;
                anx[2 * k + 1] = (R)a1;
                any_[2 * k] = (R)b0;
                any_[2 * k + 1] = (R)b1;
                f2_unpack(fsx2[k], a0, a1);
                f2_unpack(fsy2[k], b0, b1);
                afx[2 * k] = (R)a0;
                afx[2 * k + 1] = (R)a1;
                afy[2 * k] = (R)b0;
                afy[2 * k + 1] = (R)b1;
                f2_unpack(fcx2[k], a0, a1);
                f2_unpack(fcy2[k], b0, b1);
                acx[2 * k] = (R)a0;
                acx[2 * k + 1] = (R)a1;
                acy[2 * k] = (R)b0;
                acy[2 * k + 1] = (R)b1;
            }
        }
        if (active) {
#pragma unroll
            for (int r = 0; r < NR; r++) {
                R *o = red + 2 * ((slice * nthr + tl) * NR + r);
                o[0] = anx[r] + (afx[r] - acx[r]);
                o[1] = any_[r] + (afy[r] - acy[r]);
            }
        }
        __syncthreads();
        // (the sweeps' and this loop's unrolling: 100,003 particles on 12 x 12 boxes, no cutoff, the round 384 us,
        // with far entries by two and near ones by sixteen 397; 200,000 on 24 x 24 with the cutoff 593, with
        // four targets here at once 601)
        if (active && slice == 0) {
#pragma unroll NR == 4 && EXACT ? 1 : NR
            for (int r = 0; r < NR; r++) {
                if (!tv[r]) continue;
                R sx = 0, sy = 0;
#pragma unroll 4
                for (int k = 0; k < nslice; k++) {
                    const R *o = red + 2 * ((k * nthr + tl) * NR + r);
                    sx += o[0];
                    sy += o[1];
                }
                const int t = ti[r];
                double ax = d.gconst * (double)sx, ay = d.gconst * (double)sy;
                if (accumulate) {
                    ax += d.AX[t];
                    ay += d.AY[t];
                }
                d.AX[t] = ax;
                d.AY[t] = ay;
            }
        }
        __syncthreads();  // red and s_item are reused by the next item
    }
    if (tid == 0) {
        atomicAdd(&d.glob->near_pairs, npairs);
        atomicAdd(&d.glob->far_pairs, fpairs);
        // the last CTA leaves the queue as the next launch wants it (no other CTA takes from it now)
        if (atomicAdd(&d.glob->force_done, 1u) == gridDim.x - 1) {
            d.glob->item_next = 0u;
            d.glob->force_done = 0u;
        }
    }
}

template <typename R>
static size_t force_smem() {
    using S = typename Src<R>::T;
    return (size_t)far_bytes<R>() * FAR_CAP + (size_t)src_bytes<R>() * SRC_CAP + sizeof(float2) * NEAR_CAP +
           sizeof(int) * (3 * NEAR_CAP + 4) + sizeof(int) * 2 * FR_CAP;
}

template <typename R, int NR, bool KAHAN, bool TEST, bool EXACT, int MINB>
static cudaError_t launch_force_nr(const DevPlan &d, bool accumulate, cudaStream_t st, long long items_max) {
    static_assert(sizeof(R) * 2 * FT * NR <= (size_t)far_bytes<R>() * FAR_CAP + (size_t)src_bytes<R>() * SRC_CAP,
                  "reduction buffer must fit in the staging buffers");
    static_assert(FT * FORCE_R >= TARGET_CHUNK, "a CTA's quads must cover every target of a work item");
    auto k = k_force<R, NR, KAHAN, TEST, EXACT, MINB>;
    const long long slots = (long long)d.nsm * MINB, grid = items_max * (FORCE_R / NR);
    launch_step(k, (unsigned)(grid < slots ? grid : slots), FT, force_smem<R>(), st, d, accumulate ? 1 : 0);
    return cudaGetLastError();
}

// An item is one CTA's work, or two CTAs' (NR = 2) while the items, doubled, still fit on the chip
// at once: each CTA then repeats the item's walk and staging, which is what its idle neighbours
// would have waited for.  100,003 particles on 12 x 12 boxes, flat, FP32, no cutoff, the round: 958 us with
// one CTA per item and scalar arithmetic, 699 packed, 502 with two.  With the cutoff test four CTAs per SM
// (five of the half ones): 200,000 particles on 24 x 24 boxes 917 us, with six, which spill, 1,135.
template <bool TEST, int MINB> constexpr int HALF_MINB = TEST ? MINB + 1 : MINB;
template <typename R, bool KAHAN, bool TEST, bool EXACT, int MINB = (sizeof(R) == 8 ? 4 : TEST ? 4 : 8)>
struct ForceForm {  // the builds of one plan's walk
    static cudaError_t launch(const DevPlan &d, bool accumulate, cudaStream_t st) {
        const long long items_max = d.NG_total + d.n_total / d.chunk + 1;
        if constexpr (sizeof(R) == 4)
            if (2 * items_max <= (long long)d.nsm * HALF_MINB<TEST, MINB>)
                return launch_force_nr<R, 2, KAHAN, TEST, EXACT, HALF_MINB<TEST, MINB>>(d, accumulate, st, items_max);
        return launch_force_nr<R, FORCE_R, KAHAN, TEST, EXACT, MINB>(d, accumulate, st, items_max);
    }
    static cudaError_t init() {
        const int sm = (int)force_smem<R>();
        if constexpr (sizeof(R) == 4) {
            cudaError_t e = cudaFuncSetAttribute(k_force<R, 2, KAHAN, TEST, EXACT, HALF_MINB<TEST, MINB>>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
            if (e != cudaSuccess) return e;
        }
        return cudaFuncSetAttribute(k_force<R, FORCE_R, KAHAN, TEST, EXACT, MINB>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    }
};

// f(the plan's form)
template <bool KAHAN, typename F> static cudaError_t with_form32(const DevPlan &d, F f) {
    if (d.cutoff > 0.0) return f(ForceForm<float, KAHAN, true, true>());
    if (d.eps2 == 0.0) return f(ForceForm<float, KAHAN, true, false>());
    if (d.tune == 1) return f(ForceForm<float, KAHAN, false, false, 6>());
    return f(ForceForm<float, KAHAN, false, false>());
}
template <typename F> static cudaError_t with_form(const DevPlan &d, F f) {
    if (d.prec != 2) return d.prec == 1 ? with_form32<true>(d, f) : with_form32<false>(d, f);
    if (d.cutoff > 0.0 || d.eps2 == 0.0) return f(ForceForm<double, false, true, false>());
    return f(ForceForm<double, false, false, false>());
}

// Raise the dynamic shared-memory limit of the builds the plan launches (outside any stream capture).
cudaError_t force_init(const DevPlan &d) {
    if (d.stream) return fstream_init(d);
    return with_form(d, [](auto form) { return form.init(); });
}

cudaError_t launch_force(const DevPlan &d, bool tick, bool accumulate, cudaStream_t st,
                         const cudaEvent_t *ev) {
    if (d.n_total == 0) return cudaSuccess;
    if (d.stream) {  // prebuilt interaction lists, streamed (bh_lists.cu, bh_fstream.cu)
        cudaError_t e = launch_lists(d, st);
        if (e != cudaSuccess) return e;
        return launch_fstream(d, tick, accumulate, st, ev);
    }
    // The walk reads source positions from the FP64 state that a fused tick would update in
    // place while other CTAs still read them, so here the tick runs as its own kernel.
    cudaError_t e = cudaSuccess;
    if (ev && (e = cudaEventRecord(ev[0], st)) != cudaSuccess) return e;
    e = with_form(d, [&](auto form) { return form.launch(d, accumulate, st); });
    if (e != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[1], st)) != cudaSuccess) return e;
    return tick ? launch_tick(d, st, true) : cudaSuccess;
}

}  // namespace bh
