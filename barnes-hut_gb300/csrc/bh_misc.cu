// bh_misc.cu -- state upload / download, unfused tick, FP64 direct-sum sampler, diagnostics.
#include "bh_internal.cuh"
#include "bh_pairs.cuh"

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

// a warp per target: the chunks' partial sums, lane-strided, then a fixed tree
__global__ void __launch_bounds__(MT) k_direct_sum(DevPlan d, int sys, const long long *targets, long long nt, int nchunk,
                                                   double *oax, double *oay) {
    const int b = (d.glob->epoch + 1) & 1, lane = threadIdx.x & 31;
    const SysDesc &sd = d.sys[sys];
    const long long k = ((long long)blockIdx.x * MT + threadIdx.x) >> 5;
    if (k >= nt) return;
    const double *px = d.VX[b ^ 1], *py = d.VY[b ^ 1];
    double ax = 0.0, ay = 0.0;
    for (int c = lane; c < nchunk; c += 32) {
        ax += px[c * nt + k];
        ay += py[c * nt + k];
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
    const long long cap = d.n_total / nt;  // chunks the scratch holds
    if (n > 0) k_inverse_pid<<<grid_of(n, MT, d.nsm), MT, 0, st>>>(d, poff, n);
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
        k_direct<<<(unsigned)(tiles * nchunk), DT, 0, st>>>(d, sys, targets + t0, c, T, (int)nchunk, ax + t0, ay + t0);
        if (nchunk > 1)
            k_direct_sum<<<(unsigned)((c + MT / 32 - 1) / (MT / 32)), MT, 0, st>>>(d, sys, targets + t0, c, (int)nchunk,
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
