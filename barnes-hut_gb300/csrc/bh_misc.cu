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
// targets (a power of two) over one chunk of the sources: T / DR threads per slice of the chunk, DR
// targets each, so a source is loaded once per DR pairs; the chunks of a tile are the CTAs of one
// cluster, whose sums meet in its first CTA, in chunk order.  Nothing is left in the workspace but
// the inverse permutation, the same from every call: samplers on several streams may overlap, with
// each other and with an evaluation.  Bound: the FP64 pipe (2 operations per clock and SM on GB300;
// 10 per pair, with rcp64 in place of the division's 8), so the split only has to fill it.  One CTA
// per target and the division, then this: 1,000 targets of 1,048,576 29.6 -> 23.4 ms, 100 of them 4.7
// -> 2.2, 10 of them 4.7 -> 0.62; 1,500 of 400,000 16.2 -> 13.4; 10 of 100,000 0.50 -> 0.10.
constexpr int DT = 128, DRUN = 16;  // threads, sources per run
constexpr int DCL = 8;              // most chunks of a tile (the portable cluster size)

template <int DR>
__global__ void __launch_bounds__(DT) k_direct(DevPlan d, int sys, const long long *targets, long long nt, int T,
                                               int nchunk, double *oax, double *oay) {
    const int b = (d.glob->epoch + 1) & 1;
    const SysDesc &sd = d.sys[sys];
    const double *X = d.X[b], *Y = d.Y[b], *M = d.M[b];
    __shared__ double red[2 * DT * DR], part[DT], sum[DT];  // (T <= DT / 2)
    const int nthr = T / DR, nslice = DT / nthr, slice = threadIdx.x / nthr, tl = threadIdx.x - slice * nthr;
    const long long tile = blockIdx.x / nchunk;
    const int chunk = blockIdx.x - (int)(tile * nchunk);  // (its rank in the cluster)
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
                const double w = quot64(m, dx * dx + (dy * dy + d.eps2));
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
    // the slices' sums, again in runs of DRUN, then the runs'; T x runs <= DT / 2 for every T
    for (int e = threadIdx.x; e < T * ((nslice + DRUN - 1) / DRUN); e += DT) {
        const int v = e % T, s0 = e / T * DRUN;
        double rx = 0.0, ry = 0.0;
        for (int s = s0; s < s0 + DRUN && s < nslice; s++) {
            rx += red[2 * (s * T + v)];
            ry += red[2 * (s * T + v) + 1];
        }
        part[2 * e] = rx;
        part[2 * e + 1] = ry;
    }
    __syncthreads();
    const int v = threadIdx.x;
    double ax = 0.0, ay = 0.0;
    if (v < T) {
        for (int s0 = 0; s0 < nslice; s0 += DRUN) {
            ax += part[2 * (s0 / DRUN * T + v)];
            ay += part[2 * (s0 / DRUN * T + v) + 1];
        }
        sum[2 * v] = ax;
        sum[2 * v + 1] = ay;
    }
    if (nchunk > 1) {
        cluster_sync();
        if (chunk == 0 && v < T)
            for (int c = 1; c < nchunk; c++) {
                ax += __longlong_as_double(ld_cluster(reinterpret_cast<unsigned long long *>(sum) + 2 * v, c));
                ay += __longlong_as_double(ld_cluster(reinterpret_cast<unsigned long long *>(sum) + 2 * v + 1, c));
            }
        cluster_sync();  // (the sums have been read)
    }
    const long long k = tile * T + v;
    if (chunk == 0 && v < T && k < nt) {
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
    if (n > 0) k_inverse_pid<<<grid_of(n, MT, d.nsm), MT, 0, st>>>(d, poff, n);
    // Four targets a thread where their tiles, in DCL chunks each, give every SM four CTAs, in the largest
    // tile that leaves at most 1/16 of its targets idle and the chip filled; else one target a thread.
    // Chunks: a power of two of them, 16 CTAs per SM (an SM with one more than another is then a
    // sixteenth behind), two sources or more for every slice.
    const long long fill = (long long)d.nsm * 16;
    const bool four = (nt + 3) / 4 * DCL >= (long long)d.nsm * 4;
    int T = four ? 64 : 1;
    while (T > 4 && (16 * ((nt + T - 1) / T * T) > 17 * nt || (nt + T - 1) / T * DCL < fill)) T >>= 1;
    for (long long t0 = 0; t0 < nt; t0 += (1LL << 26)) {
        const long long c = nt - t0 < (1LL << 26) ? nt - t0 : (1LL << 26), tiles = (c + T - 1) / T;
        const long long most = n / (2LL * (DT * (four ? 4 : 1) / T));
        int nchunk = 1;
        while (nchunk < DCL && tiles * nchunk < fill && 2 * nchunk <= most) nchunk *= 2;
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nchunk;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cf = {};
        cf.gridDim = dim3((unsigned)(tiles * nchunk));
        cf.blockDim = dim3(DT);
        cf.stream = st;
        cf.attrs = &at;
        cf.numAttrs = 1;
        cudaError_t e = cudaLaunchKernelEx(&cf, four ? k_direct<4> : k_direct<1>, d, sys, targets + t0, c, T, nchunk, ax + t0,
                                           ay + t0);
        if (e != cudaSuccess) return e;
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
