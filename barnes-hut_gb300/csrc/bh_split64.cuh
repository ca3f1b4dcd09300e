// bh_split64.cuh -- pair interactions of nearly FP64 accuracy on the FP32 pipe, for long direct sums.
//
// GB300 executes 2 FP64 operations per clock and SM against 128 FP32 ones, and a pair costs 10 FP64
// operations: 4.8e10 pairs/s.  Here two pairs are 75 packed FP32 operations:
//   * a coordinate is a sum of three floats, x = a + b + c, with a on a grid of 2^-22 and b on one of
//     2^-44 of the system's scale, so the differences of the a's and of the b's are exact and that of
//     the c's is rounded at 2^-68 of the scale;
//   * differences, r^2, the weight and the products are unevaluated sums of two floats (error-free
//     transformations: Dekker 1971, Knuth TAOCP 4.2.2, products by fused multiply-add).  A pair's
//     error is 5e-15 rms and, the point of the operations' order, without a systematic part above
//     4e-17: terms of 2^-48 enter by fused operations whose product has bits below them, or they would
//     always be rounded away.  Over half a million terms the random part averages out below the
//     rounding of an FP64 sum, which is where these pairs are used;
//   * eight pairs are summed as two floats and the sum enters the FP64 total of the target (FP64
//     additions, on the otherwise idle FP64 pipe).
// A pair closer than 2^-16 of the scale (or anything not a number) is left to the caller's FP64
// arithmetic, so close pairs and coincident ones keep the full relative precision of their
// difference; so is a whole system whose scale, masses or softening leave the floats' range
// (Split64::usable).
#pragma once
#include "bh_pairs.cuh"

namespace bh {

constexpr float SPLIT_LIM = 2.3283064365386963e-10f;  // 2^-32: (2^-16)^2
constexpr int SPLIT_RUN = 8;                          // pairs summed in floats

__device__ __forceinline__ f2_t f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ f2_t f2_neg1() { return f2_dup(-1.f); }
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) { return f2_fma(b, f2_neg1(), a); }  // a - b, one rounding

// The shift and scale of one coordinate range [mn, mx]: a system far from the origin is moved by its
// minimum, which is exact there (every coordinate lies within a factor of two of it).
__device__ __forceinline__ double split_origin(double mn, double mx) {
    return fmax(fabs(mn), fabs(mx)) >= 2.0 * (mx - mn) ? mn : 0.0;
}

// Scale, origin, softening of a system whose coordinates span [mn, mx] and [my, My].
__device__ inline void split_setup(Split64 &s, double mn, double mx, double my, double My, double eps2) {
    s.cx = split_origin(mn, mx);
    s.cy = split_origin(my, My);
    const double e = fmax(fmax(fabs(mn - s.cx), fabs(mx - s.cx)), fmax(fabs(my - s.cy), fabs(My - s.cy)));
    int k = 0;
    const bool fin = e <= 1e300;  // (false for NaN)
    if (fin && e > 0.0) frexp(e, &k);  // e in [2^(k-1), 2^k)
    const bool ok = fin && k > -400 && k < 400;
    s.scale = ok ? scalbn(1.0, -k) : 1.0;
    s.inv_scale = ok ? scalbn(1.0, k) : 1.0;
    const double es = eps2 * s.scale * s.scale;
    s.usable = ok && es <= 1.0e12 ? 1 : 0;
    s.eh = (float)es;
    s.el = (float)(es - (double)s.eh);
}

// v (|v| <= 1) = a + b + c
__device__ __forceinline__ void split3(double v, float &a, float &b, float &c) {
    const double g1 = 1.5 * 1073741824.0;      // 1.5 x 2^30: additions round to multiples of 2^-22
    const double g2 = 1.5 * 256.0;             // 1.5 x 2^8: to multiples of 2^-44
    const double va = __dsub_rn(__dadd_rn(v, g1), g1);
    const double r = __dsub_rn(v, va);  // exact
    const double vb = __dsub_rn(__dadd_rn(r, g2), g2);
    a = (float)va;
    b = (float)vb;
    c = (float)__dsub_rn(r, vb);
}

// A mass as two floats; false where it leaves their comfortable range.
__device__ __forceinline__ bool split_mass(double m, float &mh, float &ml) {
    mh = (float)m;
    ml = (float)(m - (double)mh);
    const double q = fabs(m);
    return q == 0.0 || (q >= 8.7e-19 && q <= 1.1e18);  // 2^-60 .. 2^60 (false for NaN)
}

struct Src64 {  // a source, every value twice: -a, -b, -c of both coordinates, the mass
    f2_t ax, bx, cx, ay, by, cy, mh, ml;
};
struct Tgt64 {  // two targets
    f2_t ax, bx, cx, ay, by, cy;
};
struct Sum64 {
    f2_t hx, lx, hy, ly;
};

__device__ __forceinline__ void src64_make(Src64 &s, float4 x, float4 y) {  // (a, b, c, mh), (a, b, c, ml)
    s.ax = f2_dup(-x.x);
    s.bx = f2_dup(-x.y);
    s.cx = f2_dup(-x.z);
    s.ay = f2_dup(-y.x);
    s.by = f2_dup(-y.y);
    s.cy = f2_dup(-y.z);
    s.mh = f2_dup(x.w);
    s.ml = f2_dup(y.w);
}

__device__ __forceinline__ void sum64_zero(Sum64 &a) { a.hx = a.lx = a.hy = a.ly = 0ull; }

// (h, l) += p + low with p = -np: the sum's rounding error is kept
__device__ __forceinline__ void sum64_add(f2_t &h, f2_t &l, f2_t np, f2_t low) {
    const f2_t s = f2_sub(h, np), bb = f2_sub(s, h);
    const f2_t e = f2_sub(f2_sub(h, f2_sub(s, bb)), f2_add(np, bb));
    h = s;
    l = f2_add(l, f2_add(e, low));
}

__device__ __forceinline__ f2_t f2_max(f2_t a, f2_t b) {
    float a0, a1, b0, b1;
    f2_unpack(a, a0, a1);
    f2_unpack(b, b0, b1);
    return f2_pack(fmaxf(a0, b0), fmaxf(a1, b1));
}
__device__ __forceinline__ f2_t f2_min(f2_t a, f2_t b) {
    float a0, a1, b0, b1;
    f2_unpack(a, a0, a1);
    f2_unpack(b, b0, b1);
    return f2_pack(fminf(a0, b0), fminf(a1, b1));
}
// -1 / a, approximate
__device__ __forceinline__ f2_t f2_nrcp(f2_t a) {
    float a0, a1;
    f2_unpack(a, a0, a1);
    return f2_pack(rcp_approx(-a0), rcp_approx(-a1));
}

// The pair of one source and two targets: sum += m (x_source - x_target) / (r^2 + eps^2).  Halves
// with r^2 below lim (or NaN) contribute nothing here; `near(half, r2)` is called for them.
template <bool EPS, typename Near>
__device__ __forceinline__ void pair64(const Src64 &s, const Tgt64 &t, f2_t eh, f2_t el, float lim, Sum64 &sum,
                                       Near near) {
    const f2_t m1 = f2_neg1(), one = f2_dup(1.f);
    // d = target - source = xh + xl
    const f2_t ax = f2_add(t.ax, s.ax), bx = f2_add(t.bx, s.bx), cx = f2_add(t.cx, s.cx);
    const f2_t ay = f2_add(t.ay, s.ay), by = f2_add(t.by, s.by), cy = f2_add(t.cy, s.cy);
    const f2_t xh = f2_add(ax, bx), yh = f2_add(ay, by);
    const f2_t xl = f2_add(f2_sub(bx, f2_sub(xh, ax)), cx), yl = f2_add(f2_sub(by, f2_sub(yh, ay)), cy);
    const f2_t nxh = f2_mul(xh, m1), nyh = f2_mul(yh, m1);
    // r^2 + eps^2 = sh + sl: the high parts' sum, and the rounding errors of the squares and of the sums,
    // the cross terms, xl^2 + yl^2 and the rest of eps^2
    const f2_t px = f2_mul(xh, xh), py = f2_mul(yh, yh);
    const f2_t nex = f2_fma(xh, nxh, px), ney = f2_fma(yh, nyh, py);  // -(the squares' rounding errors)
    const f2_t big = f2_max(px, py), sml = f2_min(px, py);
    f2_t sh = f2_add(big, sml);
    const f2_t es = f2_sub(sml, f2_sub(sh, big));
    float r0, r1;
    f2_unpack(sh, r0, r1);
    f2_t lx = f2_add(xl, xl), ly = f2_add(yl, yl);
    if (EPS) {
        const f2_t hi = f2_max(sh, eh), lo = f2_min(sh, eh), u = f2_add(hi, lo);
        ly = f2_fma(yh, ly, f2_sub(lo, f2_sub(u, hi)));
        lx = f2_fma(xh, lx, f2_fma(yl, yl, f2_fma(xl, xl, el)));
        sh = u;
    } else {
        ly = f2_mul(yh, ly);
        lx = f2_fma(xh, lx, f2_fma(yl, yl, f2_mul(xl, xl)));
    }
    const f2_t sl = f2_add(f2_sub(lx, nex), f2_add(f2_sub(ly, ney), es));
    // -w = nq0 + nq1, w = m / (sh + sl)
    const f2_t ny0 = f2_nrcp(sh);
    const f2_t ny = f2_fma(ny0, f2_fma(sh, ny0, one), ny0);
    f2_t nq0 = f2_mul(s.mh, ny);
    const f2_t r = f2_add(f2_fma(nq0, sl, f2_fma(nq0, sh, s.mh)), s.ml);
    f2_t nq1 = f2_mul(r, ny);
    nq1 = f2_fma(nq1, f2_fma(sl, ny, f2_fma(sh, ny, one)), nq1);
    if (!(r0 >= lim) || !(r1 >= lim)) {
        float a0, a1, b0, b1;
        f2_unpack(nq0, a0, a1);
        f2_unpack(nq1, b0, b1);
        if (!(r0 >= lim)) {
            a0 = b0 = 0.f;
            near(0, r0);
        }
        if (!(r1 >= lim)) {
            a1 = b1 = 0.f;
            near(1, r1);
        }
        nq0 = f2_pack(a0, a1);
        nq1 = f2_pack(b0, b1);
    }
    // -w d = w (source - target)
    const f2_t npx = f2_mul(nq0, nxh), npy = f2_mul(nq0, nyh);
    sum64_add(sum.hx, sum.lx, npx, f2_add(f2_fma(nq1, xh, f2_fma(nq0, xl, f2_mul(nq1, xl))), f2_fma(nq0, xh, npx)));
    sum64_add(sum.hy, sum.ly, npy, f2_add(f2_fma(nq1, yh, f2_fma(nq0, yl, f2_mul(nq1, yl))), f2_fma(nq0, yh, npy)));
}

// the run's sums into the two targets' FP64 totals; the run starts again
__device__ __forceinline__ void sum64_flush(Sum64 &a, double &x0, double &x1, double &y0, double &y1) {
    float h0, h1, l0, l1;
    f2_unpack(a.hx, h0, h1);
    f2_unpack(a.lx, l0, l1);
    x0 = (x0 + f32_to_f64(l0)) + f32_to_f64(h0);
    x1 = (x1 + f32_to_f64(l1)) + f32_to_f64(h1);
    f2_unpack(a.hy, h0, h1);
    f2_unpack(a.ly, l0, l1);
    y0 = (y0 + f32_to_f64(l0)) + f32_to_f64(h0);
    y1 = (y1 + f32_to_f64(l1)) + f32_to_f64(h1);
    sum64_zero(a);
}

}  // namespace bh
