// Flow-map composition (integration.py:609-737): a long-T flow map built from
// nT short ones, each particle carried through the maps by bilinear
// interpolation on the particle grid.  Compiled with -fmad=false (the oracle's
// operation order).
//
// One thread per particle walks the nT maps in sequence: per map it gathers the
// 2 x 2 cell around its current point (two 32-byte rows of double2) and
// interpolates both components.  The maps are read in ring order from
// `first`, so a time series that advances by one short map needs no copy of
// the other nT - 1 (the reference shifts the whole stack every step).
//
// Interpolation is the interpolation package's eval_linear on a UCGrid with
// extrapolation CONSTANT: 0 strictly outside the grid box (pinned by the
// reference's composition fixtures: wall points that a map leaves 1 ulp
// outside [0, 2] compose to 0).  Arithmetic: cell offsets from the host-side
// inverse spacing (n - 1) / (b - a) and three explicit-FMA lerps per component,
// the same operations as the oracle.
//
// What bounds it: the FP64 pipe, 19 cycles of the SM an operation, and the
// integer instructions beside it; the stack is read from HBM once (a tenth of the
// time).  Of the 18 operations a map needs, the two scalings, the two cell offsets
// (the low bits of the scaled coordinate) and five of the six differences run on
// the integer pipe (intfp64.h, the same bits), which evens out the two pipes, and
// the tests of the box, of NaN and the cell's index come from bit patterns.  72
// maps of 676 x 251: 729 us with everything on the FP64 pipe, 302 us as it is
// (305 us with four of the differences on the integer pipe, 329 us with all six).
#include "intfp64.h"
#include "nbcs_internal.cuh"

namespace nbcs {

struct UAxis {
    double a, b, dinv, top;  // dinv = (n - 1) / (b - a), top = n - 2
    int n;
};

struct UGrid2 {
    UAxis x, y;
};

__device__ __forceinline__ bool nan64(double v)
{
    // from the halves: the compiler makes an FP64 compare of the 64-bit test
    return (((unsigned)__double2hiint(v) << 1) | (__double2loint(v) != 0)) > 0xffe00000u;
}

// Cell and offset of the coordinate v; *out when it is outside [a, b].  Below a
// by the sign of v - a (exact), beyond b only in the last cell or behind it.
__device__ __forceinline__ int lin_locate(const UAxis& A, double v, double* lam, bool* out)
{
    const double d = v - A.a;
    if (ip_bits(d) - 0x8000000000000001ull < 0x7ff0000000000000ull) *out = true;
    const double u = ip_mul(d, A.dinv);
    const ip_u64 ub = ip_bits(u);
    // u >= n - 2 (or next below it), or NaN; by the upper halves: the compiler
    // makes an FP64 compare of the 64-bit one
    if (__double2hiint(u) >= __double2hiint(A.top) && ip_pipe_greater(v, A.b)) *out = true;
    // u = M 2^-sh; the cell and what is left of it, exact
    const int sh = 1075 - ip_exponent(ub);
    const ip_u64 M = (ub & IP_FRACTION) | IP_IMPLICIT;
    int i = sh > 52 ? 0 : (int)(M >> (sh & 63));
    i = min(max(i, 0), A.n - 2);
    const ip_u64 m = M - ((ip_u64)i << (sh & 63));
    const int n = ip_clz64(m);
    *lam = sh > 52 ? ip_double(ub & ~IP_SIGN)
           : m     ? ip_pack(0, m << (n - 11), 1086 - n - sh)
                   : 0.0;
    return i;
}

__device__ __forceinline__ double2 bilinear2(const double2* __restrict__ f, const UGrid2& g,
                                             double px, double py)
{
    double l0, l1;
    bool out = false;
    const int i = lin_locate(g.x, px, &l0, &out);
    const int j = lin_locate(g.y, py, &l1, &out);
    if (out) return make_double2(0.0, 0.0);
    if (nan64(px) || nan64(py)) {
        const double n = ip_pipe_sub(px, ip_neg(py));  // NaN in, NaN out
        return make_double2(n, n);
    }
    if (!NBCS_CHECKED(i >= 0 && i <= g.x.n - 2 && j >= 0 && j <= g.y.n - 2,
                      NBCS_CHECK_COMPOSE_GATHER))
        return make_double2(0.0, 0.0);
    const double2* r0 = f + (long)i * g.y.n + j;
    const double2* r1 = r0 + g.y.n;
    const double2 f00 = __ldg(r0), f01 = __ldg(r0 + 1), f10 = __ldg(r1), f11 = __ldg(r1 + 1);
    double2 v;
    const double ax = __fma_rn(l1, ip_sub(f01.x, f00.x), f00.x);
    const double bx = __fma_rn(l1, ip_sub(f11.x, f10.x), f10.x);
    const double ay = __fma_rn(l1, ip_sub(f01.y, f00.y), f00.y);
    const double by = __fma_rn(l1, ip_sub(f11.y, f10.y), f10.y);
    v.x = __fma_rn(l0, bx - ax, ax);
    v.y = __fma_rn(l0, ip_sub(by, ay), ay);
    return v;
}

__global__ void __launch_bounds__(128)
compose_kernel(const double2* __restrict__ fms, int nT, int first, UGrid2 g,
               double2* __restrict__ out)
{
    const long m = (long)g.x.n * g.y.n;
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < m;
         p += (long)gridDim.x * blockDim.x) {
        int map = first % nT;
        double2 pt = fms[(long)map * m + p];
        // the maps after the first; of one map alone, that map again
        int k = 1;
        do {
            map = nT > 1 && map + 1 < nT ? map + 1 : 0;
            pt = bilinear2(fms + (long)map * m, g, pt.x, pt.y);
        } while (++k < nT);
        out[p] = pt;
    }
}

}  // namespace nbcs

using namespace nbcs;

extern "C" int nbcs_flowmap_compose(const double* flowmaps, int32_t nT, int32_t first,
                                    const double* grid, double* out, void* stream)
{
    NBCS_RANGE();
    if (!grid) return set_error(NBCS_ERR_INVALID, "compose: NULL grid");
    const double gnx = grid[2], gny = grid[5];
    if (!(gnx >= 2.0 && gny >= 2.0 && gnx <= 2147483647.0 && gny <= 2147483647.0) ||
        gnx != (double)(long)gnx || gny != (double)(long)gny)
        return set_error(NBCS_ERR_INVALID, "compose: grid needs integer n >= 2 on both axes");
    if (!(grid[1] > grid[0]) || !(grid[4] > grid[3]))
        return set_error(NBCS_ERR_INVALID, "compose: grid needs b > a on both axes");
    if (nT < 1 || first < 0 || first >= nT)
        return set_error(NBCS_ERR_INVALID, "compose: need nT >= 1 and 0 <= first < nT");
    const UGrid2 g = {
        {grid[0], grid[1], (gnx - 1.0) / (grid[1] - grid[0]), gnx - 2.0, (int)gnx},
        {grid[3], grid[4], (gny - 1.0) / (grid[4] - grid[3]), gny - 2.0, (int)gny}};
    const long m = (long)g.x.n * g.y.n;
    if (m > (1L << 40)) return set_error(NBCS_ERR_INVALID, "compose: grid too large");
    if (!flowmaps || !out ||
        ((reinterpret_cast<uintptr_t>(flowmaps) | reinterpret_cast<uintptr_t>(out)) & 15))
        return set_error(NBCS_ERR_INVALID, "compose: NULL or misaligned array");
    long blocks = (m + 127) / 128;
    const long cap = (long)sm_count() * 64;
    if (blocks > cap) blocks = cap;
    compose_kernel<<<(unsigned)blocks, 128, 0, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(flowmaps), nT, first, g, reinterpret_cast<double2*>(out));
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}
