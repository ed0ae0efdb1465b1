// FP64 device right-hand sides.
//
// These restate the reference's numba @cfunc bodies operation for operation
// (same operand order, every + - * / separately rounded: this file is only
// compiled with -fmad=false), so that with the same inputs they produce the
// same doubles as the CPU oracle apart from the last-bit differences of the
// transcendental functions.
//
//   double gyre   flows.py:1146-1158
//   Bickley jet   flows.py:1182-1213
//   spline RHS    flows.py:154-254 (interpolation.eval_spline, k=3)
#pragma once

#include "dop853_64.cuh"
#include "nbcs_internal.cuh"

namespace nbcs {

#define NBCS_PI 3.141592653589793

// A right-hand side is called by the two lanes of a particle together, each
// with its own component q of the position, and gives each its own component of
// the velocity.
// FEW: as in dop853_solve64, products on the FP64 pipe.
template <bool FEW = false>
struct FlowDG64 {
    static __device__ __forceinline__ double mul(double a, double b)
    {
        return FEW ? a * b : ip_mul(a, b);
    }
    __device__ __forceinline__ double operator()(double t, double y, int q, const Params& P) const
    {
        const double* p = P.v;
        const double yo = other64(y), X = q ? yo : y, Y = q ? y : yo;
        const double tt = p[0] * t;
        // (products on the FP64 pipe too, as far as it has room beside the sines)
        const double a = p[2] * ip_sin(p[4] * tt + p[5]);
        const double a2 = 2.0 * a, b = 1.0 - a2;
        const double f = mul(a, mul(X, X)) + mul(b, X);
        const double df = mul(a2, X) + b;
        // lane 0 takes sin, cos of pi f, lane 1 of pi Y
        double s, c;
        ip_sincos(NBCS_PI * (q ? Y : f), &s, &c);
        const double co = other64(c);
        // dx = -pi A sin(pi f) cos(pi Y), dy = pi A cos(pi f) sin(pi Y) df
        const double w = (q ? NBCS_PI : -NBCS_PI) * p[1];
        const double v = mul(mul(w, q ? co : s), q ? s : co);
        return p[0] * (v * (q ? df : 1.0) - p[3] * y);
    }
};

struct FlowBickley64 {
    __device__ __forceinline__ double operator()(double t, double y, int q, const Params& P) const
    {
        const double* p = P.v;
        const double yo = other64(y), X = q ? yo : y, Yv = q ? y : yo;
        const double tt = p[0] * t;
        const double Y = ip_div(Yv, ip_reciprocal(p[2]));
        const double ch = cosh(Y), th = tanh(Y);
        const double sech2 = quot64(1.0, ip_mul(ch, ch));
        // lane 0 needs the cosines, lane 1 the sines; of the first two waves each
        // lane evaluates its own (the library's functions: the jet is so chaotic
        // that another last bit leaves 1e-9 of the reference's result within days)
        double tr[3];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int w = k ? 2 : q;
            double s, c;
            sincos(ip_mul(w == 2 ? p[8] : w ? p[7] : p[6],
                          X - ip_mul(w == 2 ? p[11] : w ? p[10] : p[9], tt)), &s, &c);
            if (k == 0) {
                const double theirs = other64(q ? c : s);
                tr[0] = q ? theirs : c;
                tr[1] = q ? s : theirs;
            } else {
                tr[2] = q ? s : c;
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) tr[k] = ip_mul(q ? ip_mul(p[3 + k], p[6 + k]) : p[3 + k], tr[k]);
        const double sum = tr[0] + tr[1] + tr[2];
        // dx = U sech^2 + 2 U tanh sech^2 (sum A cos), dy = -(U L sech^2 (sum A k sin))
        const double us = ip_mul(q ? ip_mul(p[1], p[2]) : p[1], sech2);
        const double r = ip_mul(q ? us : ip_mul(ip_mul(ip_scale(p[1], 1), th), sech2), sum);
        return q ? -p[0] * r : p[0] * (us + r);
    }
};

// Python's float modulo a % 360 (sign of the divisor), as numba evaluates it.
// For |a| < 360 -- every longitude that does not lap the globe within a stage
// -- fmod returns its argument; the range test is on the bit pattern.
__device__ __forceinline__ double py_mod360(double a)
{
    const unsigned hi = (unsigned)(__double_as_longlong(a) >> 32);
    double m = a;
    if ((hi & 0x7fffffffu) >= 0x40768000u) m = fmod(a, 360.0);  // |a| >= 360, inf, NaN
    const long long mb = __double_as_longlong(m);
    if (ip_zero(m)) return 0.0;
    return mb < 0 ? m + 360.0 : m;  // NaN stays NaN
}

// Weights of the four cubic B-spline pieces at offset t:
//   w0 = (-1/6) t^3 + (3/6) t^2 + (-3/6) t + (1/6)
//   w1 =  (3/6) t^3 + (-6/6) t^2 + (0/6) t + (4/6)
//   w2 = (-3/6) t^3 + (3/6) t^2 + (3/6) t + (1/6)
//   w3 =  (1/6) t^3 + 0 + 0 + 0
// in the reference's operation order.  Products with 1/2 and 1 are exact, so
// they ride in the FMA of the sum that follows (one rounding, the sum's), the
// zero terms fall away (t is finite or NaN), and w2's two halvings become one
// of the sum: 8 FP64 operations and 3 (integer) products for 27, the same bits.
template <bool FIT>
__device__ __forceinline__ void bspline_w64(double t, double* w, unsigned* notes)
{
    const double t2 = mul64<FIT>(t, t), t3 = mul64<FIT>(t2, t), s3 = mul64<FIT>(1.0 / 6.0, t3);
    *notes |= note64(t3);  // the smallest of them (t is below 2)
    w[0] = __fma_rn(-0.5, t, __fma_rn(0.5, t2, -s3)) + 1.0 / 6.0;
    w[1] = __fma_rn(0.5, t3, -t2) + 4.0 / 6.0;
    w[2] = __fma_rn(0.5, (t2 - t3) + t, 1.0 / 6.0);
    w[3] = s3;
}

// derivative of the basis with respect to the offset t
__device__ __forceinline__ void bspline_dw64(double t, double* w)
{
    double t2 = t * t;
    w[0] = (-3.0 / 6.0) * t2 + (6.0 / 6.0) * t + (-3.0 / 6.0);
    w[1] = (9.0 / 6.0) * t2 + (-12.0 / 6.0) * t + (0.0 / 6.0);
    w[2] = (-9.0 / 6.0) * t2 + (6.0 / 6.0) * t + (3.0 / 6.0);
    w[3] = (3.0 / 6.0) * t2 + (0.0 / 6.0) * t + (0.0 / 6.0);
}

// One axis of the spline grid (SplineGrid's entries of it)
struct Axis64 {
    double a, b, dinv, top;
    int n;
};

__device__ __forceinline__ Axis64 axis64(const SplineGrid& g, int d)
{
    return {g.a[d], g.b[d], g.dinv[d], g.top[d], g.n[d]};
}

// Cell index and fractional offset of a coordinate x; dx = x - a.  A coordinate
// beyond the far end b sets *outside (it can only lie in the last cell, so the
// other cells skip the compare); a NaN coordinate takes any cell (and a NaN
// offset).  floor() runs beside the FP64 pipe; the cell index comes from the
// bits of its result, where the conversions to int and back and the two range
// compares took four FP64-pipe slots an axis.
__device__ __forceinline__ int spline_locate64(const Axis64& g, double x, double dx, double* t,
                                               bool* outside)
{
    const double u = dx * g.dinv;
    double fu = floor(u);
    if (__double_as_longlong(fu) >= __double_as_longlong(g.top)) {  // fu >= n - 2 >= 0, or NaN
        if (ip_pipe_greater(x, g.b)) *outside = true;
        fu = g.top;
    }
    *t = u - fu;
    const unsigned long long k = (unsigned long long)__double_as_longlong(fu);
    const int sh = 1075 - (int)((k >> 52) & 0x7ff);  // fu = m 2^-sh, m its 53-bit significand
    const unsigned long long m = (k & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const int i = sh > 52 ? 0 : (int)(m >> (sh & 63));
    return min(max(i, 0), g.n - 2);
}

// x < a by dx = x - a, whose sign is exact: a negative number, not -0, not NaN
__device__ __forceinline__ bool negative64(double dx)
{
    return (unsigned long long)__double_as_longlong(dx) - 0x8000000000000001ull <
           0x7ff0000000000000ull;
}

__device__ __forceinline__ double pick4(const double* w, int k)
{
    return k == 0 ? w[0] : k == 1 ? w[1] : k == 2 ? w[2] : w[3];
}

// sum_a w0[a] sum_b w1[b] sum_c w2[c] C[it+a, ix+b, iy+c] of one component (c
// points at it) of the interleaved (u, v) coefficient block, every product and
// sum rounded as the reference rounds it.
//
// FIT: the 84 products on the integer pipe (13 cycles of the SM for 19) beside
// the FP64 pipe's 63 sums; *notes tells whether all operands were in its range.
// A time level is one stretch of code without branches, so that the products of
// one row overlap the sums of another (a range test per row left each warp
// waiting for one sum after another: 1.5 times the time); the levels are a
// rolled loop, all sixteen rows at once would outgrow the instruction caches.
template <bool FIT>
__device__ __forceinline__ double spline_sum64(const double* __restrict__ c, int st, int sx,
                                               int nt, int it, int ix, int iy, const double* w0,
                                               const double* w1, const double* w2,
                                               unsigned* notes)
{
    double au = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) *notes |= note64(w0[k]) | note64(w1[k]) | note64(w2[k]);
#pragma unroll 1
    for (int a = 0; a < 4; ++a) {
        double d[4], su;
        constexpr int kRows = FIT ? 4 : 1;
#pragma unroll kRows
        for (int b = 0; b < 4; ++b) {
            const size_t e = (size_t)(it + a) * st + (size_t)(ix + b) * sx + iy;
            const double* row = c + 2 * e;
            double r[4] = {0.0, 0.0, 0.0, 0.0};
            if (NBCS_CHECKED(e + 3 < (size_t)st * (size_t)(nt + 2), NBCS_CHECK_SPLINE_GATHER)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) r[k] = __ldg(row + 2 * k);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) *notes |= note64(r[k]);
            d[b] = mul64<FIT>(w2[0], r[0]) + mul64<FIT>(w2[1], r[1]) + mul64<FIT>(w2[2], r[2]) +
                   mul64<FIT>(w2[3], r[3]);
            *notes |= note64(d[b]);
            const double p = mul64<FIT>(pick4(w1, b), d[b]);
            su = b ? su + p : FIT ? p : __fma_rn(w1[0], d[0], 0.0);
        }
        *notes |= note64(su);
        const double wa = pick4(w0, a), p = mul64<FIT>(wa, su);
        au = a ? au + p : FIT ? p : __fma_rn(wa, su, 0.0);
    }
    return au;
}

// The evaluation on the FP64 pipe: velocity masked over land (coefficients of
// exactly zero), a point on a grid node (a weight of zero), values beyond the
// integer arithmetic's range.  It comes after the integer one, so a flow with a
// component of exactly zero pays for both: 338 x 126 particles of a zonal flow 30.4
// ms, of a meridional one 32.3, at rest 8.5, with land 19.2 (35.6, 37.6, 10.6 and
// 54.7 with one lane a particle and everything on the FP64 pipe; no zeros: 22.0).
static __device__ __noinline__ double spline_plain64(const double* __restrict__ c, int st, int sx,
                                                     int nt, int it, int ix, int iy, double ft,
                                                     double fx, double fy)
{
    double w0[4], w1[4], w2[4];
    unsigned notes = 0;
    bspline_w64<false>(ft, w0, &notes);
    bspline_w64<false>(fx, w1, &notes);
    bspline_w64<false>(fy, w2, &notes);
    return spline_sum64<false>(c, st, sx, nt, it, ix, iy, w0, w1, w2, &notes);
}

// Tricubic evaluation at (t, x, y) with extrapolation mode XM, the extrap_mode
// of the interpolation package's eval_spline that the reference passes through
// (flows.py:121):
//   0 "constant": 0 strictly outside the grid box;
//   1 "nearest":  each coordinate clamped into its axis' [a, b];
//   2 "linear":   the value at the clamped point plus, for each clamped axis
//                 (t, x, y in that order), the derivative along that axis at
//                 the clamped point times the distance beyond the box.
// Lane q of the particle gives its coordinate v of x, y and gets its component:
// it finds the cell and the weights of its own axis and takes the other axis'
// from the other lane.
template <int XM>
__device__ __forceinline__ double spline_eval64(const SplineGrid& g, const double2* __restrict__ c,
                                                double t, double v, int q)
{
    const Axis64 at = axis64(g, 0);
    const Axis64 ao = {q ? g.a[2] : g.a[1], q ? g.b[2] : g.b[1], q ? g.dinv[2] : g.dinv[1],
                       q ? g.top[2] : g.top[1], q ? g.n[2] : g.n[1]};
    const double* comp = reinterpret_cast<const double*>(c) + q;
    double ct = t, co = v;
    if (XM != 0) {
        ct = t < at.a ? at.a : (t > at.b ? at.b : t);
        co = v < ao.a ? ao.a : (v > ao.b ? ao.b : v);
    }
    const double dt = ct - at.a, dv = co - ao.a;
    bool out = XM == 0 && (negative64(dt) || negative64(dv));
    double ft, fo;
    const int it = spline_locate64(at, ct, dt, &ft, &out);
    const int io = spline_locate64(ao, co, dv, &fo, &out);
    const unsigned pm = pair_mask64();
    if (XM == 0 && __any_sync(pm, out)) return 0.0;
    const int ip = __shfl_xor_sync(pm, io, 1);
    const int ix = q ? ip : io, iy = q ? io : ip;
    double w0[4], wo[4], wx[4], wy[4];
    unsigned notes = 0;
    bspline_w64<true>(ft, w0, &notes);
    bspline_w64<true>(fo, wo, &notes);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double wp = other64(wo[k]);
        wx[k] = q ? wp : wo[k];
        wy[k] = q ? wo[k] : wp;
    }
    const double fp = other64(fo), fx = q ? fp : fo, fy = q ? fo : fp;
    double au = spline_sum64<true>(comp, g.st, g.sx, g.n[0], it, ix, iy, w0, wx, wy, &notes);
    if (!fits64(notes))
        au = spline_plain64(comp, g.st, g.sx, g.n[0], it, ix, iy, ft, fx, fy);
    if (XM == 2) {
        const double dlo = v - co, dlp = other64(dlo);
        const double f[3] = {ft, fx, fy};
        const double dl[3] = {t - ct, q ? dlp : dlo, q ? dlo : dlp};
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            if (dl[d] == 0.0 || isnan(dl[d])) continue;
            double dw[4], p0[4], p1[4], p2[4];
            bspline_dw64(f[d], dw);
            bspline_w64<false>(ft, p0, &notes);
            bspline_w64<false>(fx, p1, &notes);
            bspline_w64<false>(fy, p2, &notes);
            const double gu = spline_sum64<false>(comp, g.st, g.sx, g.n[0], it, ix, iy,
                                                  d == 0 ? dw : p0, d == 1 ? dw : p1,
                                                  d == 2 ? dw : p2, &notes);
            const double s = dl[d] * g.dinv[d];
            au = au + s * gu;
        }
    }
    return au;
}

// XM: extrapolation mode (0 constant, 1 nearest, 2 linear)
template <int SPH, int XM = 0>
struct FlowSpline64 {
    SplineGrid g;
    const double2* __restrict__ c;
    double r;

    __device__ __forceinline__ double operator()(double t, double y, int q, const Params& P) const
    {
        const double* p = P.v;
        const double tt = p[0] * t;
        if (SPH == 0) return p[0] * spline_eval64<XM>(g, c, tt, y, q);
        // lane 0 holds the longitude, lane 1 the latitude
        const double lon = SPH == 1 ? py_mod360(y - 180.0) - 180.0 : py_mod360(y);
        const double w = spline_eval64<XM>(g, c, tt, q ? y : lon, q);
        // u 180 / (pi r cos(lat)) on lane 0, v 180 / (pi r) on lane 1
        const double yo = other64(y), pr = NBCS_PI * r;
        const double den = q ? pr : pr * nbcs_cos_deg(q ? y : yo);
        return ip_div(p[0] * w * 180.0, ip_reciprocal(den));
    }
};

}  // namespace nbcs
