// bh_misc.cu -- state upload / download, unfused tick, FP64 direct-sum sampler, diagnostics.
#include "bh_internal.cuh"
#include "bh_split64.cuh"

namespace bh {

constexpr int MT = 256;

static inline unsigned grid_of(long long n, int tpb, int nsm) {
    long long b = (n + tpb - 1) / tpb;
    if (b < 1) b = 1;
    if (b > nsm * 16LL) b = nsm * 16LL;
    return (unsigned)b;
}

// Upload: state buffer (epoch + 1) & 1 receives the particles in the given
// order; pid = concatenated index.  rec_stride = 0: SoA arrays; 10: the
// reference's N x 10 record (internals/particle.py:3-15), x points at row 0.
// The accelerations are not written: until the next evaluation they read as
// zero (the host tracks it; k_store then writes zeros).
__global__ void k_load(DevPlan d, const double *x, const double *y, const double *m,
                       const double *vx, const double *vy, long long rs) {
    step_enter();
    const int b = (d.glob->epoch + 1) & 1;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < d.n_total; i += stride) {
        long long k = rs ? i * rs : i;
        d.X[b][i] = x[k];
        d.Y[b][i] = y[k];
        d.M[b][i] = m[k];
        d.VX[b][i] = vx[k];
        d.VY[b][i] = vy[k];
        d.PID[b][i] = (int)i;
    }
}

// A state whose box order is far from its pid order (more than a quarter of the neighbours, counted
// by k_gather) is downloaded by gathering: random reads of whole sectors, coalesced writes.  The
// scatter writes each 8-byte value to a sector of its own, which only pays where neighbours share
// sectors.  27.3M particles of 512 systems in file order: 4,078 us -> 1,363 us with the inverse; 1,048,576: 66 -> 44 us; 4,194,304 in
// box order stay with the scatter (59 us, the memory's rate).
__device__ __forceinline__ bool store_gathers(const DevPlan &d) {
    return 4ull * d.glob->far_pids > (unsigned long long)d.n_total;
}

// inverse permutation of the current state into the key array, where k_store will gather
__global__ void k_store_inverse(DevPlan d) {
    step_enter();
    if (!store_gathers(d)) return;
    const int b = (d.glob->epoch + 1) & 1;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < d.n_total; i += stride)
        d.key[d.PID[b][i]] = (int)i;
}

// Download in pid order.  rec: N x 10 records (px, py, mass, vx, vy, ax, ay,
// gx, gy, pid) or NULL; SoA outputs may be NULL.  gx/gy come from the box
// keys of the last create_tree (skey), 0 before the first one; ax/ay are 0
// when no evaluation followed the last load (has_acc = 0).  gather: k_store_inverse ran before.
__global__ void k_store(DevPlan d, double *rec, double *x, double *y, double *vx, double *vy,
                        double *ax, double *ay, int has_tree, int has_acc, int gather) {
    step_enter();
    const int b = (d.glob->epoch + 1) & 1;
    long long stride = (long long)gridDim.x * blockDim.x;
    const bool inv = gather && store_gathers(d);
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < d.n_total; k += stride) {
        const long long i = inv ? d.key[k] : k, p = inv ? k : d.PID[b][k];
        double px = d.X[b][i], py = d.Y[b][i], pvx = d.VX[b][i], pvy = d.VY[b][i];
        const double pax = has_acc ? d.AX[i] : 0.0, pay = has_acc ? d.AY[i] : 0.0;
        if (rec) {
            double *r = rec + 10 * p;
            double gx = 0.0, gy = 0.0;
            if (has_tree) {
                int key = d.skey[i];
                int s = find_seg(d.boff_tab, d.nsys, key);
                int lb = (int)(key - d.sys[s].boff);
                gx = (double)(lb / d.sys[s].G);
                gy = (double)(lb % d.sys[s].G);
            }
            r[0] = px; r[1] = py; r[2] = d.M[b][i]; r[3] = pvx; r[4] = pvy;
            r[5] = pax; r[6] = pay; r[7] = gx; r[8] = gy; r[9] = (double)p;
        }
        if (x) x[p] = px;
        if (y) y[p] = py;
        if (vx) vx[p] = pvx;
        if (vy) vy[p] = pvy;
        if (ax) ax[p] = pax;
        if (ay) ay[p] = pay;
    }
}

// v += a dt; a = 0; x += v dt  (gpu/grid.py:159-174)
// keep_acc: leave the accelerations in place (the fused step's tick, which keeps the last
// evaluation's accelerations; the reference's tick, gpu/grid.py:159-174, zeroes them)
__global__ void k_tick(DevPlan d, int keep_acc) {
    step_enter();
    const int b = (d.glob->epoch + 1) & 1;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < d.n_total; i += stride) {
        double ax = d.AX[i], ay = d.AY[i];
        double vx = d.VX[b][i] + ax * d.dt, vy = d.VY[b][i] + ay * d.dt;
        d.VX[b][i] = vx;
        d.VY[b][i] = vy;
        if (!keep_acc) {
            d.AX[i] = 0.f;
            d.AY[i] = 0.f;
        }
        d.X[b][i] = d.X[b][i] + vx * d.dt;
        d.Y[b][i] = d.Y[b][i] + vy * d.dt;
    }
}

// inverse permutation pid -> current index over the particles of one system, written into the key array
__global__ void k_inverse_pid(DevPlan d, long long i0, long long n) {
    const int b = (d.glob->epoch + 1) & 1;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        d.key[d.PID[b][i0 + i]] = (int)(i0 + i);
}

// FP64 direct sum (base.py:16-32; the target itself is skipped by index).  A CTA serves a tile of T
// targets (T a power of two, 4 .. 64) over one chunk of the sources: T / 4 threads per slice of the
// chunk, four targets each, so a source is loaded once per four pairs.  Bound: the FP64 pipe (2
// operations per clock and SM on GB300; 10 per pair, with rcp64 in place of the division's 8), so
// the split over chunks only has to fill it: few targets over many sources run on the whole chip
// (before: one CTA per target, 16.5 operations per pair).  1,500 targets of 400,000: 16.2 ->
// 13.4 ms; 100 of 200,000: 938 -> 536 us; 10 of 100,000: 494 -> 93 us.
// Partial sums of chunk c, target k: px, py[c * nt + k] (the state buffer that is not current, free
// between steps), added in chunk order by k_direct_sum; a single chunk writes the result itself.
constexpr int DT = 128, DR = 4, DRUN = 16;  // threads, targets per thread, sources per run
// k_direct_split from 2^19 sources on: relative error of the sums against quadruple precision, over
// uniform, clustered, generated and far-off systems, softened and not, FP64 kernel / split floats:
// 65,536 sources 0.8-1.1e-16 / 1.6-3.2e-16, 262,144: 1.0-1.2 / 1.0-1.2, 524,288: 1.1-1.5 / 0.8-1.0,
// 1,048,576: 1.3-1.9 / 0.7-1.0, 2,000,000: 1.3-2.3 / 0.7-1.1; and from 2^23 pairs on (two passes over
// the particles first)
constexpr long long SPLIT_MIN_N = 1 << 19, SPLIT_MIN_PAIRS = 1 << 23;

__global__ void __launch_bounds__(DT) k_direct(DevPlan d, int sys, const long long *targets, long long nt, int T,
                                               int nchunk, double *oax, double *oay) {
    const int b = (d.glob->epoch + 1) & 1;
    const SysDesc &sd = d.sys[sys];
    const double *X = d.X[b], *Y = d.Y[b], *M = d.M[b];
    __shared__ double red[2 * DT * DR];
    const int nthr = T / DR, nslice = DT / nthr, slice = threadIdx.x / nthr, tl = threadIdx.x - slice * nthr;
    const long long tile = blockIdx.x / nchunk;
    const int chunk = blockIdx.x - (int)(tile * nchunk);
    const long long k0 = tile * T + (long long)tl * DR;
    long long ti[DR];
    double xt[DR], yt[DR], sx[DR], sy[DR];
#pragma unroll
    for (int r = 0; r < DR; r++) {
        const long long t = k0 + r < nt ? targets[k0 + r] : -1;
        const bool in = t >= sd.poff && t < sd.poff + sd.n;  // a particle of this system
        ti[r] = in ? d.key[t] : -1;
        xt[r] = in ? X[ti[r]] : 0.0;
        yt[r] = in ? Y[ti[r]] : 0.0;
        sx[r] = sy[r] = 0.0;
    }
    const long long j0 = sd.poff + (sd.n * chunk) / nchunk, j1 = sd.poff + (sd.n * (chunk + 1)) / nchunk;
    // runs of DRUN sources are summed by themselves: a thread's share of the sources is one sum's rounding
    // errors long otherwise, where the former kernel had a 256th of them
    for (long long b0 = j0 + slice; b0 < j1; b0 += DRUN * nslice) {
        double rx[DR], ry[DR];
#pragma unroll
        for (int r = 0; r < DR; r++) rx[r] = ry[r] = 0.0;
        const long long b1 = b0 + DRUN * nslice < j1 ? b0 + DRUN * nslice : j1;
#pragma unroll 2
        for (long long j = b0; j < b1; j += nslice) {
            const double x = X[j], y = Y[j], m = M[j];
#pragma unroll
            for (int r = 0; r < DR; r++) {
                const double dx = x - xt[r], dy = y - yt[r];
                const double w = m * rcp64(dx * dx + (dy * dy + d.eps2));
                if (j != ti[r]) {
                    rx[r] += w * dx;
                    ry[r] += w * dy;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < DR; r++) {
            sx[r] += rx[r];
            sy[r] += ry[r];
        }
    }
#pragma unroll
    for (int r = 0; r < DR; r++) {
        red[2 * (threadIdx.x * DR + r)] = sx[r];
        red[2 * (threadIdx.x * DR + r) + 1] = sy[r];
    }
    __syncthreads();
    double *px = d.VX[b ^ 1], *py = d.VY[b ^ 1];
    for (int v = threadIdx.x; v < T && tile * T + v < nt; v += DT) {
        double ax = 0.0, ay = 0.0;
        for (int s0 = 0; s0 < nslice; s0 += DRUN) {
            double rx = 0.0, ry = 0.0;
            for (int s = s0; s < s0 + DRUN && s < nslice; s++) {
                rx += red[2 * (s * T + v)];
                ry += red[2 * (s * T + v) + 1];
            }
            ax += rx;
            ay += ry;
        }
        const long long k = tile * T + v;
        if (nchunk > 1) {
            px[chunk * nt + k] = ax;
            py[chunk * nt + k] = ay;
        } else {
            const bool in = targets[k] >= sd.poff && targets[k] < sd.poff + sd.n;
            const double nan = __longlong_as_double(0x7ff8000000000000ll);
            oax[k] = in ? d.gconst * ax : nan;
            oay[k] = in ? d.gconst * ay : nan;
        }
    }
}

// ---- the same on the FP32 pipe (bh_split64.cuh), for long sums
// Inverse permutation and extents of the system's particles; the last block sets up the frame.
__global__ void __launch_bounds__(MT) k_direct_prep(DevPlan d, long long i0, long long n) {
    const int b = (d.glob->epoch + 1) & 1;
    const double *X = d.X[b], *Y = d.Y[b];
    unsigned long long e[4] = {~0ull, ~0ull, 0ull, 0ull};
    for (long long i = (long long)blockIdx.x * MT + threadIdx.x; i < n; i += (long long)gridDim.x * MT) {
        d.key[d.PID[b][i0 + i]] = (int)(i0 + i);
        const unsigned long long x = ord_bits(X[i0 + i]), y = ord_bits(Y[i0 + i]);
        e[0] = x < e[0] ? x : e[0];
        e[1] = y < e[1] ? y : e[1];
        e[2] = x > e[2] ? x : e[2];
        e[3] = y > e[3] ? y : e[3];
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, e[q], o);
            e[q] = q < 2 ? (v < e[q] ? v : e[q]) : (v > e[q] ? v : e[q]);
        }
        if ((threadIdx.x & 31) == 0) {
            if (q < 2) atomicMin(&d.split->ext[q], e[q]);
            else atomicMax(&d.split->ext[q], e[q]);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&d.split->done, 1u) == gridDim.x - 1) {
        __threadfence();
        Split64 &s = *d.split;
        double v[4];
        for (int q = 0; q < 4; q++) {
            v[q] = unord_bits(__ldcg(&s.ext[q]));
            s.ext[q] = q < 2 ? ~0ull : 0ull;
        }
        s.done = 0u;
        split_setup(s, v[0], v[2], v[1], v[3], d.eps2);
    }
}

// The particles as split floats, into the state buffer that is not current: (a, b) of x and of y, both
// c, the mass.
__global__ void __launch_bounds__(MT) k_direct_convert(DevPlan d, long long i0, long long n) {
    const int b = (d.glob->epoch + 1) & 1;
    const double cx = d.split->cx, cy = d.split->cy, scale = d.split->scale;
    float2 *AX = reinterpret_cast<float2 *>(d.X[b ^ 1]), *AY = reinterpret_cast<float2 *>(d.Y[b ^ 1]);
    float2 *C = reinterpret_cast<float2 *>(d.VX[b ^ 1]), *MM = reinterpret_cast<float2 *>(d.M[b ^ 1]);
    for (long long i = i0 + (long long)blockIdx.x * MT + threadIdx.x; i < i0 + n; i += (long long)gridDim.x * MT) {
        float xa, xb, xc, ya, yb, yc, mh, ml;
        split3((d.X[b][i] - cx) * scale, xa, xb, xc);
        split3((d.Y[b][i] - cy) * scale, ya, yb, yc);
        if (!split_mass(d.M[b][i], mh, ml)) d.split->usable = 0;
        AX[i] = make_float2(xa, xb);
        AY[i] = make_float2(ya, yb);
        C[i] = make_float2(xc, yc);
        MM[i] = make_float2(mh, ml);
    }
}

// As k_direct, with DT sources staged at a time; partial sums interleaved in VY of the other buffer.
// 1,000 targets of 1,048,576: 21.9 ms in FP64 -> 3.3 ms, 100 targets 0.9 ms.
template <bool EPS>
__global__ void __launch_bounds__(DT, 4) k_direct_split(DevPlan d, int sys, const long long *targets, long long nt,
                                                        int T, int nchunk, double *oax, double *oay) {
    __shared__ __align__(16) Src64 src[DT];
    __shared__ double red[2 * DT * DR];
    const int b = (d.glob->epoch + 1) & 1;
    const SysDesc &sd = d.sys[sys];
    const Split64 &fr = *d.split;
    const bool usable = fr.usable != 0;
    const double *X = d.X[b], *Y = d.Y[b], *M = d.M[b];
    const float2 *AX = reinterpret_cast<const float2 *>(d.X[b ^ 1]), *AY = reinterpret_cast<const float2 *>(d.Y[b ^ 1]);
    const float2 *C = reinterpret_cast<const float2 *>(d.VX[b ^ 1]), *MM = reinterpret_cast<const float2 *>(d.M[b ^ 1]);
    const int nthr = T / DR, nslice = DT / nthr, slice = threadIdx.x / nthr, tl = threadIdx.x - slice * nthr;
    const long long tile = blockIdx.x / nchunk;
    const int chunk = blockIdx.x - (int)(tile * nchunk);
    const long long k0 = tile * T + (long long)tl * DR;
    int ti[DR];
    double sx[DR], sy[DR];
    Tgt64 tg[DR / 2];
    Sum64 sum[DR / 2];
#pragma unroll
    for (int r = 0; r < DR; r++) {
        const long long t = k0 + r < nt ? targets[k0 + r] : -1;
        ti[r] = t >= sd.poff && t < sd.poff + sd.n ? d.key[t] : -1;  // a particle of this system
        sx[r] = sy[r] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < DR / 2; k++) {
        const int i0 = ti[2 * k] < 0 ? (int)sd.poff : ti[2 * k], i1 = ti[2 * k + 1] < 0 ? (int)sd.poff : ti[2 * k + 1];
        const float2 x0 = AX[i0], x1 = AX[i1], y0 = AY[i0], y1 = AY[i1], c0 = C[i0], c1 = C[i1];
        tg[k].ax = f2_pack(x0.x, x1.x);
        tg[k].bx = f2_pack(x0.y, x1.y);
        tg[k].cx = f2_pack(c0.x, c1.x);
        tg[k].ay = f2_pack(y0.x, y1.x);
        tg[k].by = f2_pack(y0.y, y1.y);
        tg[k].cy = f2_pack(c0.y, c1.y);
        sum64_zero(sum[k]);
    }
    const f2_t eh = f2_dup(fr.eh), el = f2_dup(fr.el);
    // one pair in FP64 (close ones, and every one of a system that does not fit the floats), into the
    // sums' scaled units
    auto pair_fp64 = [&](int r, long long j) {
        if (ti[r] < 0 || j == ti[r]) return;
        const double dx = X[j] - X[ti[r]], dy = Y[j] - Y[ti[r]];
        const double w = M[j] * rcp64(dx * dx + (dy * dy + d.eps2)) * fr.inv_scale;
        sx[r] += w * dx;
        sy[r] += w * dy;
    };
    const long long j0 = sd.poff + (sd.n * chunk) / nchunk, j1 = sd.poff + (sd.n * (chunk + 1)) / nchunk;
    for (long long p = j0; p < j1; p += DT) {
        const int ns = (int)(j1 - p < DT ? j1 - p : DT);
        __syncthreads();  // the previous stage has been swept
        if (threadIdx.x < ns) {
            const long long j = p + threadIdx.x;
            const float2 ax = AX[j], ay = AY[j], c = C[j], m = MM[j];
            src64_make(src[threadIdx.x], make_float4(ax.x, ax.y, c.x, m.x), make_float4(ay.x, ay.y, c.y, m.y));
        }
        __syncthreads();
        if (usable) {
            for (int q0 = slice; q0 < ns; q0 += SPLIT_RUN * nslice) {
#pragma unroll 1
                for (int u = 0; u < SPLIT_RUN; u++) {
                    const int q = q0 + u * nslice;
                    if (q >= ns) break;
                    const Src64 s = src[q];
#pragma unroll
                    for (int k = 0; k < DR / 2; k++)
                        pair64<EPS>(s, tg[k], eh, el, SPLIT_LIM, sum[k],
                                    [&](int half, float) { pair_fp64(2 * k + half, p + q); });
                }
#pragma unroll
                for (int k = 0; k < DR / 2; k++)
                    sum64_flush(sum[k], sx[2 * k], sx[2 * k + 1], sy[2 * k], sy[2 * k + 1]);
            }
        } else {
            for (int q = slice; q < ns; q += nslice)
                for (int r = 0; r < DR; r++) pair_fp64(r, p + q);
        }
    }
#pragma unroll
    for (int r = 0; r < DR; r++) {
        red[2 * (threadIdx.x * DR + r)] = sx[r];
        red[2 * (threadIdx.x * DR + r) + 1] = sy[r];
    }
    __syncthreads();
    double2 *part = reinterpret_cast<double2 *>(d.VY[b ^ 1]);
    for (int v = threadIdx.x; v < T && tile * T + v < nt; v += DT) {
        double ax = 0.0, ay = 0.0;
        for (int s = 0; s < nslice; s++) {
            ax += red[2 * (s * T + v)];
            ay += red[2 * (s * T + v) + 1];
        }
        part[chunk * nt + tile * T + v] = make_double2(ax * fr.scale, ay * fr.scale);
    }
}

// a warp per target: the chunks' partial sums, lane-strided, then a fixed tree
// (pairs: the partial sums as pairs in VY, else x in VX and y in VY)
__global__ void __launch_bounds__(MT) k_direct_sum(DevPlan d, int sys, const long long *targets, long long nt, int nchunk,
                                                   int pairs, double *oax, double *oay) {
    const int b = (d.glob->epoch + 1) & 1, lane = threadIdx.x & 31;
    const SysDesc &sd = d.sys[sys];
    const long long k = ((long long)blockIdx.x * MT + threadIdx.x) >> 5;
    if (k >= nt) return;
    const double *px = d.VX[b ^ 1], *py = d.VY[b ^ 1];
    double ax = 0.0, ay = 0.0;
    for (int c = lane; c < nchunk; c += 32) {
        if (pairs) {
            const double2 v = reinterpret_cast<const double2 *>(py)[c * nt + k];
            ax += v.x;
            ay += v.y;
        } else {
            ax += px[c * nt + k];
            ay += py[c * nt + k];
        }
    }
    for (int o = 16; o; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
    if (lane == 0) {
        const bool in = targets[k] >= sd.poff && targets[k] < sd.poff + sd.n;
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        oax[k] = in ? d.gconst * ax : nan;
        oay[k] = in ? d.gconst * ay : nan;
    }
}

// out = {kinetic, momentum x, momentum y, potential}; FP64 block reductions.
__global__ void __launch_bounds__(MT) k_diag(DevPlan d, int sys, int want_pot, double *out) {
    const int b = (d.glob->epoch + 1) & 1;
    const SysDesc &sd = d.sys[sys];
    __shared__ double red[4][MT / 32];
    double ke = 0, px = 0, py = 0, pe = 0;
    long long n = sd.n;
    for (long long i = (long long)blockIdx.x * MT + threadIdx.x; i < n; i += (long long)gridDim.x * MT) {
        long long k = sd.poff + i;
        double m = d.M[b][k], vx = d.VX[b][k], vy = d.VY[b][k];
        ke += 0.5 * m * (vx * vx + vy * vy);
        px += m * vx;
        py += m * vy;
        if (want_pot) {
            double xi = d.X[b][k], yi = d.Y[b][k], s = 0.0;
            for (long long j = sd.poff; j < sd.poff + n; j++) {
                if (j == k) continue;
                double dx = d.X[b][j] - xi, dy = d.Y[b][j] - yi;
                s += d.M[b][j] * 0.5 * log(dx * dx + dy * dy + d.eps2);
            }
            pe += 0.5 * m * s;  // each pair counted twice
        }
    }
    double v[4] = {ke, px, py, pe * d.gconst};
    for (int c = 0; c < 4; c++)
        for (int o = 16; o; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
    if ((threadIdx.x & 31) == 0)
        for (int c = 0; c < 4; c++) red[c][threadIdx.x >> 5] = v[c];
    __syncthreads();
    if (threadIdx.x < 4) {
        double a = 0;
        for (int k = 0; k < MT / 32; k++) a += red[threadIdx.x][k];
        atomicAdd(out + threadIdx.x, a);
    }
}

// Leaf centres of mass in the reference layout (G x G x 3: cx, cy, M).
__global__ void k_box_com(DevPlan d, int sys, double *out) {
    const SysDesc &sd = d.sys[sys];
    const SysDyn &dy = d.dyn[sys];
    long long B = (long long)sd.G * sd.G;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x; b < B; b += stride) {
        const double *q = d.mom + 6 * (sd.coff + b);
        double M = q[0];
        double *o = out + 3 * b;
        if (M > 0.0) {
            int kx = (int)(b / sd.G), ky = (int)(b % sd.G);
            o[0] = box_origin(dy.minx, kx, dy.step) + q[1] / M;
            o[1] = box_origin(dy.miny, ky, dy.step) + q[2] / M;
            o[2] = M;
        } else {
            o[0] = o[1] = o[2] = 0.0;
        }
    }
}

cudaError_t launch_box_com(const DevPlan &d, int sys, double *out, cudaStream_t st) {
    k_box_com<<<d.nsm * 4, MT, 0, st>>>(d, sys, out);
    return cudaGetLastError();
}

cudaError_t launch_load(const DevPlan &d, const double *x, const double *y, const double *m,
                        const double *vx, const double *vy, long long rs, cudaStream_t st) {
    if (d.n_total == 0) return cudaSuccess;
    launch_step(k_load, grid_of(d.n_total, MT, d.nsm), MT, 0, st, d, x, y, m, vx, vy, rs);
    return cudaGetLastError();
}

cudaError_t launch_store(const DevPlan &d, int has_tree, bool has_acc, double *rec, double *x, double *y,
                         double *vx, double *vy, double *ax, double *ay, cudaStream_t st) {
    if (d.n_total == 0) return cudaSuccess;
    // (before the first create_tree the state is in pid order)
    const bool gather = has_tree && d.n_total >= STORE_GATHER_MIN;
    if (gather) launch_step(k_store_inverse, grid_of(d.n_total, MT, d.nsm), MT, 0, st, d);
    launch_step(k_store, grid_of(d.n_total, MT, d.nsm), MT, 0, st, d, rec, x, y, vx, vy, ax, ay, has_tree, has_acc ? 1 : 0,
                gather ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_tick(const DevPlan &d, cudaStream_t st, bool keep_acc) {
    if (d.n_total == 0) return cudaSuccess;
    launch_step(k_tick, grid_of(d.n_total, MT, d.nsm), MT, 0, st, d, keep_acc ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_direct(const DevPlan &d, int sys, long long poff, long long n, const long long *targets,
                          long long nt, double *ax, double *ay, cudaStream_t st) {
    if (d.n_total == 0 || nt == 0) return cudaSuccess;
    // split floats: long sums (their accuracy rests on averaging), enough of them to pay for two
    // passes over the particles, and room for the partial sums
    const bool split = n >= SPLIT_MIN_N && nt * n >= SPLIT_MIN_PAIRS && 2 * nt <= d.n_total;
    const long long cap = split ? d.n_total / (2 * nt) : d.n_total / nt;  // chunks the scratch holds
    if (split) {
        k_direct_prep<<<grid_of(n, MT * 4, d.nsm), MT, 0, st>>>(d, poff, n);
        k_direct_convert<<<grid_of(n, MT, d.nsm), MT, 0, st>>>(d, poff, n);
    } else if (n > 0) {
        k_inverse_pid<<<grid_of(n, MT, d.nsm), MT, 0, st>>>(d, poff, n);
    }
    // The largest tile that leaves at most 1/16 of its targets idle (else the one that leaves least),
    // while tiles x chunks fill the chip: the scratch holds n_total / nt chunks, so many targets of
    // few sources need small tiles.  A small tile costs nothing but its slices' longer reduction.
    const long long fill = (long long)d.nsm * 4;
    int T = 64;
    long long least = 0;
    for (int c = 64; c >= DR; c >>= 1) {
        const long long pad = (nt + c - 1) / c * c, room = cap > 1 ? cap : 1;
        if (c == 64 || pad < least || (nt + T - 1) / T * room < fill) {
            least = pad;
            T = c;
        }
        if (16 * pad <= 17 * nt && (nt + T - 1) / T * room >= fill) break;
    }
    for (long long t0 = 0; t0 < nt; t0 += (1LL << 28)) {
        const long long c = nt - t0 < (1LL << 28) ? nt - t0 : (1LL << 28), tiles = (c + T - 1) / T;
        // chunks: 16 CTAs per SM (an SM with one more than another is then a sixteenth behind: 1,500
        // targets of 400,000 15.5 -> 13.4 ms against four), at least two sources for every slice, within
        // the scratch
        long long nchunk = (4 * fill + tiles - 1) / tiles;
        const long long most = n / (2LL * (DT * DR / T));
        nchunk = nchunk < most ? nchunk : most;
        nchunk = nchunk < cap ? nchunk : cap;
        if (nchunk < 1) nchunk = 1;
        if (split) {
            auto k = d.eps2 > 0.0 ? k_direct_split<true> : k_direct_split<false>;
            k<<<(unsigned)(tiles * nchunk), DT, 0, st>>>(d, sys, targets + t0, c, T, (int)nchunk, ax + t0, ay + t0);
            k_direct_sum<<<(unsigned)((c + MT / 32 - 1) / (MT / 32)), MT, 0, st>>>(d, sys, targets + t0, c, (int)nchunk, 1,
                                                                                 ax + t0, ay + t0);
            continue;
        }
        k_direct<<<(unsigned)(tiles * nchunk), DT, 0, st>>>(d, sys, targets + t0, c, T, (int)nchunk, ax + t0, ay + t0);
        if (nchunk > 1)
            k_direct_sum<<<(unsigned)((c + MT / 32 - 1) / (MT / 32)), MT, 0, st>>>(d, sys, targets + t0, c, (int)nchunk, 0,
                                                                                 ax + t0, ay + t0);
    }
    return cudaGetLastError();
}

cudaError_t launch_diag(const DevPlan &d, int sys, int want_pot, double *out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, 4 * sizeof(double), st);
    if (e != cudaSuccess) return e;
    k_diag<<<d.nsm * 2, MT, 0, st>>>(d, sys, want_pot, out);
    return cudaGetLastError();
}

}  // namespace bh
