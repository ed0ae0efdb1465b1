// FTLE ridge extraction: exact percentile selection, ridge stencil and
// order-preserving compaction, in one cooperative launch.
//
//   ftle_ridge_pts   extraction/ridges.py:9-76
//   _ftle_ridges     extraction/ridges.py:79-154 (the mask)
//   np.percentile    ridges.py:48-51, evaluated by numba inside the jitted
//                    function: rank = 1 + (n-1)*q/100, value
//                    lower*(1-m) + upper*m of the order statistics around it.
//
// Percentile: radix selection of the k-th smallest double on order-preserving
// 64-bit keys, 11 bits per pass.  A pass histograms the digit of the keys in
// the group chosen so far; after a grid-wide barrier every block finds the digit
// with the rank by itself.  As soon as the group has no more than kCand keys --
// after two or three passes on an FTLE field -- they are gathered and ranked by
// counting; that pass over the field also takes the smallest key above the
// group, in case the (k+1)-th order statistic lies there.
//
// Ridge points: each warp evaluates the stencil on its run of points, writes
// the mask (and, when the caller asks for it, the full point array) and keeps
// its points in shared memory in row-major order; after a barrier the block adds
// up the counts of the blocks before it and writes its points behind theirs.
//
// What bounds it: on the benchmark's 676 x 251 field (1.4 MB) nothing but
// latency -- ten launches with a memset between two of them took 81 us, against
// some 2 us per barrier here; on large fields the passes over f (HBM or L2) and
// the stencil, whose quotients and products run on the integer pipe
// (intfp64.h, the same bits).
// Whole launch, percentile 90, against the ten launches: 676 x 251 81 -> 29 us,
// 2701 x 1001 195 -> 78 us (of which the stencil of the points above the
// threshold about half; of all points, percentile 0, 112 us).
//
// The barriers wait for blocks of the same cooperative launch only, which the
// GPU runs all at once, and give up after a fixed number of polls.  One block
// that gives up fails the launch: the others leave at their next poll, and the
// last block to get past the barriers or to give up writes the number of points,
// or -1 and points that are NaN (an atomic a block).
// Compiled with -fmad=false: the stencil arithmetic is the reference's.
#include <math.h>

#include <atomic>
#include <mutex>

#include "intfp64.h"
#include "nbcs_internal.cuh"

namespace nbcs {

constexpr int kDigitBits = 11;
constexpr int kBins = 1 << kDigitBits;
constexpr int kPasses = 6;        // 64 bits: five of 11, one of 9
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kCand = 512;        // keys ranked by counting (one per thread)
constexpr int kKept = 64;         // ridge points a warp keeps; beyond, it evaluates again
constexpr int kPollLimit = 1 << 20;
constexpr unsigned kGaveUp = 0x80000000u;

// Scratch; the first part starts at zero (one memset).
struct SelScratch {
    unsigned int hist[kPasses][kBins];
    unsigned long long above_inv;  // ~(smallest key above the group); 0: none
    unsigned int nan_count, pinf, ninf;
    unsigned int cand_n;
    unsigned int arrived;          // barrier arrivals; kGaveUp: a block has given up
    unsigned int ended;            // blocks past the last barrier, or given up
    unsigned long long total;      // ridge points, by the last block
    unsigned long long cand[kCand];  // not zeroed
};
constexpr size_t kZeroed = offsetof(SelScratch, cand);

// order-preserving unsigned key of a double's bit pattern
__device__ __forceinline__ unsigned long long dkey(unsigned long long u)
{
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// NaN test on the bit pattern, without an FP64 compare
__device__ __forceinline__ bool bits_nan(unsigned long long u)
{
    return (u & 0x7fffffffffffffffull) > 0x7ff0000000000000ull;
}

__device__ __forceinline__ double dkey_decode(unsigned long long k)
{
    unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)u);
}

struct RidgeIn {
    const double* f;
    const double2* ev;
    const double* x;
    const double* y;
    long n;                  // points
    int nx;
    FastDiv ny;
    double sdd;
    double fmin_val;         // threshold when no percentile is taken
    double dx, dy;           // grid spacing; NaN: x[1] - x[0], y[1] - y[0] (ridges.py:39-40)
    uint8_t* mask;           // or NULL
    double2* full;           // or NULL
    double2* pts;
    int* idx;                // linear indices of the points, or NULL
    int64_t* n_out;
    unsigned int* count;     // ridge points per block
    int polls;               // after which a barrier gives up
};

// How the k-th and (k+1)-th order statistics become the percentile (numba's
// rules, ridges.py:48-51).
struct SelFinish {
    int take;     // 0: no percentile
    int mode;     // 0: interpolate; 1: q == 100 (maximum); 2: q == 0 (minimum)
    long long k;  // rank of the lower statistic
    double m;     // interpolation weight of the upper one
    double* out;  // or NULL
};

// ------------------------------------------------------------ grid barrier

// Every block of the (cooperative) launch has arrived `phase + 1` times.
// False, in all threads of the block, when it has waited too long or another
// block has.
__device__ bool grid_barrier(SelScratch* s, unsigned phase, int polls)
{
    __shared__ bool ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&s->arrived, 1u);
        const unsigned want = (phase + 1) * gridDim.x;
        ok = false;
        for (; polls > 0; --polls) {
            unsigned have;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(have) : "l"(&s->arrived) : "memory");
            if (have >= want) {  // or given up: kGaveUp is above all counts
                ok = have < kGaveUp;
                break;
            }
        }
        if (!ok) atomicOr(&s->arrived, kGaveUp);
    }
    __syncthreads();
    return ok;
}

// ------------------------------------------------------------ percentile

__device__ double percentile_of(const SelFinish& fin, long n, unsigned long long kk,
                                unsigned long long up, long long nan_count, long long pinf,
                                long long ninf)
{
    double lower = dkey_decode(kk), val;
    if (nan_count > 0) {
        val = NAN;
    } else if (n == 1) {
        val = lower;
    } else if (fin.mode == 1) {  // q == 100: maximum
        val = lower;
        if ((pinf + ninf) > 0 && !isfinite(val)) val = NAN;
    } else if (fin.mode == 2) {  // q == 0: minimum, with numba's infinity rules
        val = lower;
        if (pinf + ninf > 0) {
            long long finite = n - (pinf + ninf);
            if (finite == 0) val = NAN;
            if (pinf == 1 && n == 2) val = NAN;
            if (ninf > 1) val = NAN;
            if (finite == 1 && pinf > 1 && ninf != 1) val = NAN;
        }
    } else {
        double upper = (up == ~0ull) ? lower : dkey_decode(up);
        val = lower * (1.0 - fin.m) + upper * fin.m;
    }
    return val;
}

struct SelShared {
    unsigned int h[kBins];
    unsigned long long cand[kCand];
    unsigned long long wmax[kWarps];
    long long wsum[kWarps];
    unsigned int cnt[3];
    int digit;
    unsigned int in_bin;
    long long rank;
    unsigned long long kk, up;
    double result;
};

// The percentile of f[0 .. n) in all threads of all blocks (with *ok false the
// NaN of a launch that gave up); *phase counts the barriers.
__device__ double select_percentile(const double* __restrict__ f, long n, SelScratch* s,
                                    SelShared& sh, const SelFinish& fin, int polls,
                                    unsigned* phase, bool* ok)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long stride = (long)gridDim.x * kThreads;
    unsigned long long prefix = 0, pmask = 0;
    long long rank = fin.k;
    int shift = 64;
    for (int pass = 0; pass < kPasses; ++pass) {
        const int bits = shift >= kDigitBits ? kDigitBits : shift;
        shift -= bits;
        const unsigned dmask = (1u << bits) - 1u;
        for (int b = tid; b < kBins; b += kThreads) sh.h[b] = 0;
        if (tid < 3) sh.cnt[tid] = 0;
        __syncthreads();
        unsigned nn = 0, np = 0, nm = 0;
        // whole warps go round together: the lanes whose digit is the first
        // active lane's (most of them, in the first pass: the exponent) are
        // counted by one atomic
        for (long base = (long)blockIdx.x * kThreads + warp * 32; base < n; base += 4 * stride) {
            unsigned long long u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const long i = base + j * stride + lane;
                u[j] = i < n ? (unsigned long long)__double_as_longlong(__ldg(f + i))
                             : 0x7ff8000000000001ull;  // past the end: like a NaN, not counted
                if (i >= n) nn -= pass == 0;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bool in = !bits_nan(u[j]);
                if (pass == 0) {
                    nn += !in;
                    np += u[j] == 0x7ff0000000000000ull;
                    nm += u[j] == 0xfff0000000000000ull;
                }
                const unsigned long long key = dkey(u[j]);
                in = in && (key & pmask) == prefix;
                const unsigned d = (unsigned)(key >> shift) & dmask;
                const unsigned active = __ballot_sync(0xffffffffu, in);
                if (!active) continue;
                const unsigned d0 = __shfl_sync(0xffffffffu, d, __ffs(active) - 1);
                const unsigned same = __ballot_sync(0xffffffffu, in && d == d0);
                if (lane == 0) atomicAdd(&sh.h[d0], (unsigned)__popc(same));
                if (in && d != d0) atomicAdd(&sh.h[d], 1u);
            }
        }
        if (pass == 0) {
            if (nn) atomicAdd(&sh.cnt[0], nn);
            if (np) atomicAdd(&sh.cnt[1], np);
            if (nm) atomicAdd(&sh.cnt[2], nm);
        }
        __syncthreads();
        for (int b = tid; b <= (int)dmask; b += kThreads)
            if (sh.h[b]) atomicAdd(&s->hist[pass][b], sh.h[b]);
        if (pass == 0 && tid == 0) {
            if (sh.cnt[0]) atomicAdd(&s->nan_count, sh.cnt[0]);
            if (sh.cnt[1]) atomicAdd(&s->pinf, sh.cnt[1]);
            if (sh.cnt[2]) atomicAdd(&s->ninf, sh.cnt[2]);
        }
        if (!grid_barrier(s, (*phase)++, polls)) {
            *ok = false;
            return __longlong_as_double((long long)NBCS_PERCENTILE_FAILED);
        }
        // every block: the digit whose cumulative count passes the rank.  Each
        // thread sums four consecutive bins, a block-wide scan of those sums finds
        // the one whose range holds the rank, and it walks its own bins.
        constexpr int kPer = kBins / kThreads;
        const int nb = (int)dmask + 1;
        unsigned hb[kPer];
        long long local = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int b = tid * kPer + q;
            hb[q] = b < nb ? __ldcg(&s->hist[pass][b]) : 0u;
            local += hb[q];
        }
        long long incl = local;
        for (int o = 1; o < 32; o <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) sh.wsum[warp] = incl;
        __syncthreads();
        for (int w = 0; w < warp; ++w) incl += sh.wsum[w];
        const long long excl = incl - local;
        long long total = 0;
        for (int w = 0; w < kWarps; ++w) total += sh.wsum[w];
        // (a rank beyond all keys, with NaN among them: any digit will do)
        if ((excl <= rank && rank < incl) || (rank >= total && tid == kThreads - 1)) {
            long long cum = excl;
            int q = 0;
            for (; q < kPer - 1; ++q) {
                if (cum + (long long)hb[q] > rank) break;
                cum += hb[q];
            }
            sh.digit = min(tid * kPer + q, nb - 1);
            sh.in_bin = hb[q];
            sh.rank = rank - cum;
        }
        __syncthreads();
        prefix |= (unsigned long long)sh.digit << shift;
        pmask |= (unsigned long long)dmask << shift;
        rank = sh.rank;
        const unsigned in_bin = sh.in_bin;
        __syncthreads();
        if (in_bin <= kCand || shift == 0) break;
    }
    const long long nan_count = __ldcg(&s->nan_count), pinf = __ldcg(&s->pinf),
                    ninf = __ldcg(&s->ninf);
    const unsigned in_bin = sh.in_bin;
    // gather the group's keys (all equal when every bit is chosen) and take the
    // smallest key above it
    const bool whole = shift == 0;
    unsigned long long ainv = 0ull;
    if (fin.mode == 0 || !whole) {
        for (long base = (long)blockIdx.x * kThreads + warp * 32; base < n; base += 4 * stride) {
            unsigned long long u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const long i = base + j * stride + lane;
                u[j] = i < n ? (unsigned long long)__double_as_longlong(__ldg(f + i))
                             : 0x7ff8000000000001ull;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (bits_nan(u[j])) continue;
                const unsigned long long key = dkey(u[j]);
                if ((key & pmask) > prefix) {
                    if (~key > ainv) ainv = ~key;
                } else if (!whole && (key & pmask) == prefix) {
                    const unsigned at = atomicAdd(&s->cand_n, 1u);
                    if (at < kCand) s->cand[at] = key;
                }
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, ainv, o);
            ainv = other > ainv ? other : ainv;
        }
        if (lane == 0) sh.wmax[warp] = ainv;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kWarps; ++w) ainv = sh.wmax[w] > ainv ? sh.wmax[w] : ainv;
            if (ainv) atomicMax(&s->above_inv, ainv);
        }
        if (!grid_barrier(s, (*phase)++, polls)) {
            *ok = false;
            return __longlong_as_double((long long)NBCS_PERCENTILE_FAILED);
        }
    }
    const unsigned long long above = __ldcg(&s->above_inv);
    if (tid == 0) {
        sh.kk = prefix;
        sh.up = above ? ~above : ~0ull;
        if (whole && rank + 1 < (long long)in_bin) sh.up = prefix;
    }
    if (!whole) {
        // rank by counting: one candidate a thread (kCand = kThreads)
        if (tid < (int)in_bin) sh.cand[tid] = __ldcg(&s->cand[tid]);
        __syncthreads();
        if (tid < (int)in_bin) {
            const unsigned long long mine = sh.cand[tid];
            unsigned less = 0, equal = 0;
            unsigned long long next = ~0ull;
            for (unsigned c = 0; c < in_bin; ++c) {
                const unsigned long long v = sh.cand[c];
                less += v < mine;
                equal += v == mine;
                if (v > mine && v < next) next = v;
            }
            if ((long long)less <= rank && rank < (long long)(less + equal)) {
                // threads with equal keys write the same values
                sh.kk = mine;
                if (rank + 1 < (long long)(less + equal)) sh.up = mine;
                else if (next != ~0ull) sh.up = next;
            }
        }
    }
    __syncthreads();
    if (tid == 0) sh.result = percentile_of(fin, n, sh.kk, sh.up, nan_count, pinf, ninf);
    __syncthreads();
    return sh.result;
}

// ------------------------------------------------------------ ridges

// a > b for doubles given as bit patterns, by integer comparison (IEEE
// semantics: false when either is NaN, -0 == +0); the ridge threshold test runs
// on every point and an FP64 compare would issue on the narrow FP64 pipe
__device__ __forceinline__ bool gt_bits(unsigned long long a, unsigned long long b)
{
    if (bits_nan(a) || bits_nan(b)) return false;
    if ((a << 1) == 0) a = 0;  // -0 -> +0
    if ((b << 1) == 0) b = 0;
    return dkey(a) > dkey(b);
}

// The stencil's divisors 2 dx, 2 dy, dx^2, dy^2 and 4 dx dy
struct RidgeSpacing {
    double hx, hy;  // dx / 2, dy / 2; below 0 where nothing is within them
    ip_divisor x2, y2, xx, yy, xy;
};

__device__ void ridge_spacing(const RidgeIn& R, RidgeSpacing* S)
{
    const double dx = R.dx == R.dx ? R.dx : R.x[1] - R.x[0];
    const double dy = R.dy == R.dy ? R.dy : R.y[1] - R.y[0];
    S->hx = dx / 2.0 >= 0.0 ? dx / 2.0 : -1.0;
    S->hy = dy / 2.0 >= 0.0 ? dy / 2.0 : -1.0;
    S->x2 = ip_reciprocal(2.0 * dx);
    S->y2 = ip_reciprocal(2.0 * dy);
    S->xx = ip_reciprocal(dx * dx);
    S->yy = ip_reciprocal(dy * dy);
    S->xy = ip_reciprocal(4.0 * dx * dy);
}

// |a| <= h by bit patterns; false for NaN and for h < 0.  Halves: of the 64-bit
// comparison the compiler makes an FP64 one that is true for NaN.
__device__ __forceinline__ bool within(double a, double h)
{
    const int ah = __double2hiint(a) & 0x7fffffff, hh = __double2hiint(h);
    return ah < hh || (ah == hh && (unsigned)__double2loint(a) <= (unsigned)__double2loint(h));
}

// Ridge test at the interior point k = i*ny + j above the threshold
// (ridges.py:52-74).  Returns true and the sub-pixel point when it is a ridge
// point.
__device__ __forceinline__ bool ridge_at(const RidgeIn& R, const RidgeSpacing& S, long k,
                                         double* px, double* py)
{
    const int ny = (int)R.ny.d;
    const double* f = R.f;
    int i, j;
    row_col(k, R.ny, &i, &j);
    const double f0 = __ldg(f + k);
    const double fip = __ldg(f + k + ny), fim = __ldg(f + k - ny), fjp = __ldg(f + k + 1),
                 fjm = __ldg(f + k - 1);
    const double fx = ip_div(fip - fim, S.x2);
    const double fy = ip_div(fjp - fjm, S.y2);
    const double f2 = 2.0 * f0;
    const double fxx = ip_div(fip - f2 + fim, S.xx);
    const double fyy = ip_div(fjp - f2 + fjm, S.yy);
    const double fxy = ip_div(__ldg(f + k + ny + 1) - __ldg(f + k + ny - 1) -
                                  __ldg(f + k - ny + 1) + __ldg(f + k - ny - 1), S.xy);
    const double2 e = R.ev[k];
    const double ex = e.x, ey = e.y;
    const double c2 = ip_mul(ex, ip_mul(fxx, ex) + ip_mul(fxy, ey)) +
                      ip_mul(ey, ip_mul(fxy, ex) + ip_mul(fyy, ey));
    if (!(c2 < -R.sdd)) return false;
    const double t = ip_div(ip_neg(ip_mul(fx, ex) + ip_mul(fy, ey)), ip_reciprocal(c2));
    const double tx = ip_mul(t, ex), ty = ip_mul(t, ey);
    if (within(tx, S.hx) && within(ty, S.hy)) {
        *px = R.x[i] + tx;
        *py = R.y[j] + ty;
        return true;
    }
    return false;
}

// A warp's candidates waiting for the stencil and the ridge points it keeps
struct RidgeWarp {
    double2 pt[kKept];
    int at[kKept];       // their places in the warp's run
    int queue[160];      // candidates, as places in the warp's run
};

struct RidgeShared {
    RidgeWarp w[kWarps];
    RidgeSpacing S;
    unsigned int wcount[kWarps];
    unsigned long long wpre[kWarps];
};

// One warp's run of points [base, base + len): the points above the threshold
// are queued, and the stencil runs on 32 queued points at a time -- a tenth of
// the points are above the 90th percentile, scattered over most warps' rounds,
// and a warp pays for a stencil whether one of its lanes needs it or all.
// Calls take(rank in the run, place in the run, point) for every ridge point, in
// order, and returns their number.  store: also writes the mask and the full
// array.
template <class Take>
__device__ __forceinline__ unsigned ridge_run_of(const RidgeIn& R, const RidgeSpacing& S,
                                                 double fmin, long base, int len, bool store,
                                                 int* queue, Take take)
{
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const unsigned long long fm = (unsigned long long)__double_as_longlong(fmin);
    unsigned found = 0;
    int waiting = 0;
    for (int c0 = 0; c0 < len; c0 += 128) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = c0 + 32 * q + lane;
            v[q] = c < len ? __ldg(R.f + base + c) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = c0 + 32 * q + lane;
            if (store && c < len) {
                if (R.mask) R.mask[base + c] = 0;
                if (R.full) R.full[base + c] = make_double2(0.0, 0.0);
            }
            bool cand = c < len && gt_bits((unsigned long long)__double_as_longlong(v[q]), fm);
            if (cand) {
                int i, j;
                row_col(base + c, R.ny, &i, &j);
                cand = i >= 2 && i < R.nx - 2 && j >= 2 && j < (int)R.ny.d - 2;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, cand);
            if (cand) queue[waiting + __popc(bal & below)] = c;
            waiting += __popc(bal);
        }
        __syncwarp();
        // full warps of queued points, and at the run's end the rest of them
        int done = 0;
        const bool end = c0 + 128 >= len;
#pragma unroll 1
        while (waiting - done >= 32 || (end && waiting > done)) {
            const int m = min(32, waiting - done);
            double px = 0.0, py = 0.0;
            const int place = lane < m ? queue[done + lane] : 0;
            const long k = base + place;
            const bool on = lane < m && ridge_at(R, S, k, &px, &py);
            const unsigned bal = __ballot_sync(0xffffffffu, on);
            if (on) {
                if (store && R.mask) R.mask[k] = 1;
                if (store && R.full) R.full[k] = make_double2(px, py);
                take(found + __popc(bal & below), place, make_double2(px, py));
            }
            found += __popc(bal);
            done += m;
        }
        const int rest = done + lane < waiting ? queue[done + lane] : 0;
        __syncwarp();
        queue[lane] = rest;
        waiting -= done;
        __syncwarp();
    }
    return found;
}

// Ridge flags, points and their compaction by a block; false when a barrier gave
// up.
__device__ __forceinline__ bool ridge_block(const RidgeIn& R, SelScratch* s, RidgeShared& g,
                                            double fmin, unsigned phase)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) ridge_spacing(R, &g.S);
    __syncthreads();
    // this warp's run of points (whole rounds of 32)
    const long runs = (long)gridDim.x * kWarps;
    const long len_all = ((R.n + runs - 1) / runs + 31) / 32 * 32;
    const long base = ((long)blockIdx.x * kWarps + warp) * len_all;
    const int len = base >= R.n ? 0 : (int)(R.n - base < len_all ? R.n - base : len_all);
    RidgeWarp& own = g.w[warp];
    unsigned long long first = 0;
    // once for the counts; again, to write, only where a warp has found more
    // points than it keeps (one copy of the code for both)
#pragma unroll 1
    for (int again = 0; again < 2; ++again) {
        const unsigned found = ridge_run_of(
            R, g.S, fmin, base, len, !again, own.queue,
            [&](unsigned rank, int place, double2 p) {
                if (again) {
                    R.pts[first + rank] = p;
                    if (R.idx) R.idx[first + rank] = (int)(base + place);
                } else if (rank < kKept) {
                    own.pt[rank] = p;
                    own.at[rank] = place;
                }
            });
        if (again) break;
        if (lane == 0) g.wcount[warp] = found;
        __syncthreads();
        unsigned total = 0, before = 0;
        for (int w = 0; w < kWarps; ++w) {
            if (w < warp) before += g.wcount[w];
            total += g.wcount[w];
        }
        if (tid == 0) R.count[blockIdx.x] = total;
        if (!grid_barrier(s, phase, R.polls)) return false;
        // the points of the blocks before this one
        unsigned long long pre = 0;
        for (unsigned b = tid; b < blockIdx.x; b += kThreads) pre += __ldcg(R.count + b);
        for (int o = 16; o > 0; o >>= 1) pre += __shfl_xor_sync(0xffffffffu, pre, o);
        if (lane == 0) g.wpre[warp] = pre;
        __syncthreads();
        for (int w = 0; w < kWarps; ++w) first += g.wpre[w];
        if (blockIdx.x == gridDim.x - 1 && tid == 0) s->total = first + total;
        first += before;
        if (found <= kKept) {
            for (unsigned q = lane; q < found; q += 32) {
                R.pts[first + q] = own.pt[q];
                if (R.idx) R.idx[first + q] = (int)(base + own.at[q]);
            }
            break;
        }
    }
    return true;
}

// A block's warp 0, past the last barrier or after the block has given up: the
// last of them to come writes the outcome.  (What the blocks write to the mask and
// the full array they write before that barrier.)
__device__ __forceinline__ void ridge_end(const RidgeIn& R, SelScratch* s)
{
    const int lane = threadIdx.x & 31;
    unsigned failed = 0;
    if (lane == 0) {
        unsigned before;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(&s->ended) : "memory");
        if (before + 1 == gridDim.x) {
            failed = __ldcg(&s->arrived) >= kGaveUp;
            *R.n_out = failed ? -1 : (int64_t)__ldcg(&s->total);
        }
    }
    if (!__shfl_sync(0xffffffffu, failed, 0)) return;
    __syncwarp();
    for (long k = lane; k < R.n; k += 32) {
        if (R.mask) R.mask[k] = 1;
        if (R.full) R.full[k] = make_double2(NAN, NAN);
    }
}

// One cooperative launch: percentile (when asked for), ridge flags, compaction.
// RIDGES false: the percentile alone.
template <bool RIDGES>
__global__ void __launch_bounds__(kThreads, 2)
ridge_kernel(RidgeIn R, SelScratch* s, SelFinish fin)
{
    __shared__ union {
        SelShared sel;
        RidgeShared ridge;
    } sh;
    const int tid = threadIdx.x;
    unsigned phase = 0;
    bool ok = true;
    double fmin = R.fmin_val;
    if (fin.take) {
        fmin = select_percentile(R.f, R.n, s, sh.sel, fin, R.polls, &phase, &ok);
        // (a block that has passed the last barrier has the value, whatever
        // becomes of the others)
        if (fin.out && blockIdx.x == 0 && tid == 0) *fin.out = fmin;
        __syncthreads();  // the shared memory changes hands
    }
    if constexpr (RIDGES) {
        if (ok) ridge_block(R, s, sh.ridge, fmin, phase);
        if (tid < 32) ridge_end(R, s);
    }
}

// ------------------------------------------------------------ components

// The 8-connected components of the ridge points (the scipy.ndimage.label call
// of ftle_ridges, ridges.py:219-222) from the points themselves: pt_index holds
// their linear grid indices in row-major order, so a neighbour is found by
// binary search.  Components by hooking and pointer jumping in shared memory,
// numbered by their first point, then a sort by (component, point) for the order
// in which ftle_ridges returns them.
//
// One block: a field's ridges are thin, a few thousand points of some millions.
// Labelling the whole grid (seven launches) and sorting with library calls took
// 530 us of the 720 us of a 2701 x 1001 field's ftle_ridges call; this kernel
// 26 us (1500 points).  More than kCompMax points are left to the grid labelling.
constexpr int kCompMax = NBCS_RIDGE_COMPONENTS_MAX;
constexpr int kCompThreads = 1024;
static_assert(kCompMax == 8192, "the sort key holds 13 bits of point index");

__global__ void __launch_bounds__(kCompThreads)
ridge_components_kernel(const double2* __restrict__ pts, const int* __restrict__ pt_index,
                        const int64_t* __restrict__ n_pts, int ny, double2* __restrict__ out,
                        int* __restrict__ head)
{
    extern __shared__ int csh[];
    int* idx = csh;
    int* parent = csh + kCompMax;
    unsigned* key = reinterpret_cast<unsigned*>(csh + 2 * kCompMax);
    int* cnt = csh + 3 * kCompMax;
    __shared__ int wsum[kCompThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t np = *n_pts;
    if (np < 0 || np > kCompMax) {
        if (tid == 0) {
            head[0] = np > 0x7fffffff ? 0x7fffffff : (int)np;
            head[1] = -1;
        }
        return;
    }
    const int n = (int)np;
    for (int q = tid; q < n; q += kCompThreads) {
        idx[q] = pt_index[q];
        cnt[q] = 0;
    }
    __syncthreads();
    // a point's earlier neighbours: the one to its left (1 bit) and up to three
    // above it (the first one's number, their count); it links to the first
    for (int q = tid; q < n; q += kCompThreads) {
        const int k = idx[q], j = k % ny;
        const int left = q > 0 && j > 0 && idx[q - 1] == k - 1;
        int a = 0, up = 0;
        if (k >= ny) {
            const int lo = k - ny - (j > 0), hi = k - ny + (j < ny - 1);
            int b = q;  // the first point at or behind lo
            while (a < b) {
                const int mid = (a + b) >> 1;
                if (idx[mid] < lo) a = mid + 1;
                else b = mid;
            }
            while (a + up < q && idx[a + up] <= hi) ++up;
        }
        key[q] = ((unsigned)a << 3) | ((unsigned)up << 1) | (unsigned)left;
        parent[q] = up ? a : left ? q - 1 : q;
    }
    __syncthreads();
    // Shiloach & Vishkin (1982): shorten all paths to stars by pointer jumping,
    // hook the larger of two touching stars' roots to the smaller, until no two
    // touch.  Of touching stars at least one root a round is hooked, so the rounds
    // end; a star that nothing hooks to and that stays in one round (its neighbours
    // found smaller ones) is hooked itself in the next, so two rounds leave at most
    // half of a component's stars; a handful of rounds do for ridges, up to 11 for
    // combs of 8192 points.  A path of 8192 links is short after 13 jumps.
    for (int round = 0; round < kCompMax; ++round) {
        for (int jump = 0; jump < 14; ++jump) {
            int moved = 0;
            for (int q = tid; q < n; q += kCompThreads) {
                const int p = parent[q], g = parent[p];
                if (g != p) {
                    parent[q] = g;
                    moved = 1;
                }
            }
            if (!__syncthreads_or(moved)) break;
        }
        int hooked = 0;
        for (int q = tid; q < n; q += kCompThreads) {
            const unsigned e = key[q];
            const int rq = parent[q];
            for (int c = 0; c < 4; ++c) {
                int a = -1;
                if (c < 3 && c < (int)((e >> 1) & 3u)) a = (int)(e >> 3) + c;
                if (c == 3 && (e & 1u)) a = q - 1;
                if (a < 0) continue;
                const int ra = parent[a];
                if (ra != rq) {
                    atomicMin(&parent[max(ra, rq)], min(ra, rq));
                    hooked = 1;
                }
            }
        }
        if (!__syncthreads_or(hooked)) break;
    }
    for (int q = tid; q < n; q += kCompThreads) key[q] = (unsigned)parent[q];
    __syncthreads();
    // number the roots in index order: each thread a run of eight points
    constexpr int kPer = kCompMax / kCompThreads;
    int mine = 0;
    for (int e = 0; e < kPer; ++e) {
        const int q = tid * kPer + e;
        mine += q < n && key[q] == (unsigned)q;
    }
    int incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int total = 0;
    for (int w = 0; w < kCompThreads / 32; ++w) {
        if (w < warp) incl += wsum[w];
        total += wsum[w];
    }
    int label = incl - mine;
    for (int e = 0; e < kPer; ++e) {
        const int q = tid * kPer + e;
        if (q < n && key[q] == (unsigned)q) parent[q] = label++;
    }
    __syncthreads();
    int size = 1;  // a power of two for the sort
    while (size < n) size <<= 1;
    for (int q = tid; q < size; q += kCompThreads) {
        if (q < n) {
            const int lab = parent[key[q]];
            atomicAdd(&cnt[lab], 1);
            key[q] = ((unsigned)lab << 13) | (unsigned)q;
        } else {
            key[q] = 0xffffffffu;
        }
    }
    __syncthreads();
    // bitonic sort
    for (int k = 2; k <= size; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int t = tid; t < size / 2; t += kCompThreads) {
                const int a = ((t & ~(j - 1)) << 1) | (t & (j - 1)), b = a | j;
                const unsigned x = key[a], y = key[b];
                if ((x > y) == ((a & k) == 0)) {
                    key[a] = y;
                    key[b] = x;
                }
            }
            __syncthreads();
        }
    }
    for (int q = tid; q < n; q += kCompThreads) out[q] = pts[key[q] & (kCompMax - 1)];
    for (int q = tid; q < total; q += kCompThreads) head[2 + q] = cnt[q];
    if (tid == 0) {
        head[0] = n;
        head[1] = total;
    }
}

// Blocks of a launch: two per SM, all resident at once -- on the SMs that the
// stream's context owns -- and on small fields as few as give every thread four
// points (a barrier costs by the block: 41, 37 and 29 us at one, two and four
// points a thread on 676 x 251).
static unsigned ridge_grid(long n, cudaStream_t st)
{
    long b = (n + 4 * kThreads - 1) / (4 * kThreads);
    const long cap = 2L * stream_sm_count(st);
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

constexpr int kMaxBlocks = 1024;  // block counts in the scratch

// the rank, rule and weight of the q-th percentile of n values
static SelFinish finish_rule(long n, double q, double* out)
{
    SelFinish fin = {1, 0, 0, 0.0, out};
    if (n == 1) {
        fin.k = 0;
    } else if (q == 100.0) {
        fin.mode = 1;
        fin.k = n - 1;
    } else if (q == 0.0) {
        fin.mode = 2;
        fin.k = 0;
    } else {
        double rank = 1.0 + (double)(n - 1) * (q / 100.0);
        double fl = floor(rank);
        fin.m = rank - fl;
        fin.k = (long long)(fl - 1.0);
    }
    return fin;
}

#ifdef NBCS_CHECK
// the debug library's tests let the barriers give up
static std::atomic<int> g_polls{kPollLimit};
static int poll_limit() { return g_polls.load(); }
#else
static int poll_limit() { return kPollLimit; }
#endif

static int launch_ridges(bool ridges, RidgeIn R, SelScratch* s, SelFinish fin, cudaStream_t st)
{
    unsigned g = ridge_grid(R.n, st);
    if (g > kMaxBlocks) g = kMaxBlocks;
    R.polls = poll_limit();
    NBCS_CUDA_TRY(cudaMemsetAsync(s, 0, kZeroed, st));
    void* args[] = {&R, &s, &fin};
    // fewer blocks where that many do not fit at once after all (any number will do)
    cudaError_t e;
    do {
        e = cudaLaunchCooperativeKernel(
            ridges ? (const void*)ridge_kernel<true> : (const void*)ridge_kernel<false>, dim3(g),
            dim3(kThreads), args, 0, st);
        g /= 2;
        if (e == cudaErrorCooperativeLaunchTooLarge) cudaGetLastError();  // not the next call's
    } while (e == cudaErrorCooperativeLaunchTooLarge && g > 0);
    NBCS_CUDA_TRY(e);
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

}  // namespace nbcs

using namespace nbcs;

extern "C" int nbcs_check_ridge_polls(int32_t polls)
{
#ifdef NBCS_CHECK
    g_polls.store(polls < 0 ? kPollLimit : polls);
    return NBCS_OK;
#else
    (void)polls;
    return set_error(NBCS_ERR_UNSUPPORTED, "check_ridge_polls: the bounds-checked build only");
#endif
}

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

extern "C" size_t nbcs_percentile_scratch_bytes(int64_t n)
{
    (void)n;
    return align256(sizeof(SelScratch));
}

extern "C" int nbcs_percentile(const double* f, int64_t n, double q, double* out, void* scratch,
                               size_t scratch_bytes, void* stream)
{
    NBCS_RANGE();
    if (n < 1 || !f || !out) return set_error(NBCS_ERR_INVALID, "percentile: empty input or NULL");
    if (!(q >= 0.0 && q <= 100.0)) return set_error(NBCS_ERR_INVALID, "percentile: q outside [0, 100]");
    if (!scratch || scratch_bytes < sizeof(SelScratch))
        return set_error(NBCS_ERR_SCRATCH, "percentile: scratch needs %zu bytes", sizeof(SelScratch));
    RidgeIn R = {};
    R.f = f;
    R.n = (long)n;
    return launch_ridges(false, R, static_cast<SelScratch*>(scratch), finish_rule((long)n, q, out),
                         as_stream(stream));
}

// selection state, block counts and (as callers have sized it) a byte per point
extern "C" size_t nbcs_ridge_scratch_bytes(int32_t nx, int32_t ny)
{
    if (nx < 0 || ny < 0) return 0;
    return align256(sizeof(SelScratch)) + align256(sizeof(unsigned int) * kMaxBlocks) +
           align256((size_t)nx * ny);
}

// Ridge flags, points and compaction with the threshold f_min either taken
// from the percentile selection (use_percentile, percentile != 0) or given.
static int ridge_run(const double* f, const double* evec_max, const double* x, int32_t nx,
                     const double* y, int32_t ny, double dx, double dy, double sdd_thresh,
                     bool use_percentile, double percentile, double f_min, uint8_t* mask_out,
                     double* rpts_full, double* pts_out, int32_t* pt_index, int64_t* n_out,
                     void* scratch, size_t scratch_bytes, void* stream)
{
    if (nx < 2 || ny < 2) return set_error(NBCS_ERR_INVALID, "ridge_pts: need nx, ny >= 2");
    if (!f || !evec_max || !x || !y || !pts_out || !n_out)
        return set_error(NBCS_ERR_INVALID, "ridge_pts: NULL array");
    if ((reinterpret_cast<uintptr_t>(evec_max) | reinterpret_cast<uintptr_t>(pts_out) |
         reinterpret_cast<uintptr_t>(rpts_full)) & 15)
        return set_error(NBCS_ERR_INVALID, "ridge_pts: evec/pts arrays must be 16-byte aligned");
    if (use_percentile && !(percentile >= 0.0 && percentile <= 100.0))
        return set_error(NBCS_ERR_INVALID, "ridge_pts: percentile outside [0, 100]");
    size_t need = nbcs_ridge_scratch_bytes(nx, ny);
    if (!scratch || scratch_bytes < need)
        return set_error(NBCS_ERR_SCRATCH, "ridge_pts: scratch needs %zu bytes", need);
    const long n = (long)nx * ny;
    if (pt_index && n > 0x7fffffffL)
        return set_error(NBCS_ERR_INVALID, "ridge_pts: 32-bit point indices on a larger grid");
    char* p = static_cast<char*>(scratch);
    SelScratch* sel = reinterpret_cast<SelScratch*>(p);
    p += align256(sizeof(SelScratch));
    RidgeIn R = {};
    R.f = f;
    R.ev = reinterpret_cast<const double2*>(evec_max);
    R.x = x;
    R.y = y;
    R.n = n;
    R.nx = nx;
    R.ny = fast_div(ny);
    R.sdd = sdd_thresh;
    R.dx = dx;
    R.dy = dy;
    R.fmin_val = use_percentile ? 0.0 : f_min;
    R.mask = mask_out;
    R.full = reinterpret_cast<double2*>(rpts_full);
    R.pts = reinterpret_cast<double2*>(pts_out);
    R.idx = pt_index;
    R.n_out = n_out;
    R.count = reinterpret_cast<unsigned int*>(p);
    SelFinish fin = {};
    if (use_percentile && percentile != 0.0) fin = finish_rule(n, percentile, nullptr);  // ridges.py:48-51
    return launch_ridges(true, R, sel, fin, as_stream(stream));
}

extern "C" int nbcs_ridge_pts(const double* f, const double* evec_max, const double* x, int32_t nx,
                              const double* y, int32_t ny, double sdd_thresh, double percentile,
                              uint8_t* mask_out, double* rpts_full, double* pts_out,
                              int64_t* n_out, void* scratch, size_t scratch_bytes, void* stream)
{
    NBCS_RANGE();
    return ridge_run(f, evec_max, x, nx, y, ny, NAN, NAN, sdd_thresh, true, percentile, 0.0,
                     mask_out, rpts_full, pts_out, nullptr, n_out, scratch, scratch_bytes, stream);
}

extern "C" int nbcs_ridge_pts_fmin(const double* f, const double* evec_max, const double* x,
                                   int32_t nx, const double* y, int32_t ny, double dx, double dy,
                                   double sdd_thresh, double f_min, uint8_t* mask_out,
                                   double* rpts_full, double* pts_out, int64_t* n_out,
                                   void* scratch, size_t scratch_bytes, void* stream)
{
    NBCS_RANGE();
    if (!(dx > 0.0 || dx < 0.0) || !(dy > 0.0 || dy < 0.0))
        return set_error(NBCS_ERR_INVALID, "ridge_pts_fmin: dx, dy must be nonzero");
    return ridge_run(f, evec_max, x, nx, y, ny, dx, dy, sdd_thresh, false, 0.0, f_min, mask_out,
                     rpts_full, pts_out, nullptr, n_out, scratch, scratch_bytes, stream);
}

extern "C" int nbcs_ridge_components(const double* f, const double* evec_max, const double* x,
                                     int32_t nx, const double* y, int32_t ny, double sdd_thresh,
                                     double percentile, uint8_t* mask_out, double* pts_out,
                                     int32_t* pt_index, int64_t* n_out, double* comp_pts,
                                     int32_t* head, void* scratch, size_t scratch_bytes,
                                     void* stream)
{
    NBCS_RANGE();
    if (!pt_index || !comp_pts || !head)
        return set_error(NBCS_ERR_INVALID, "ridge_components: NULL array");
    if (reinterpret_cast<uintptr_t>(comp_pts) & 15)
        return set_error(NBCS_ERR_INVALID, "ridge_components: comp_pts must be 16-byte aligned");
    int rc = ridge_run(f, evec_max, x, nx, y, ny, NAN, NAN, sdd_thresh, true, percentile, 0.0,
                       mask_out, nullptr, pts_out, pt_index, n_out, scratch, scratch_bytes, stream);
    if (rc) return rc;
    constexpr int kBytes = 4 * kCompMax * (int)sizeof(int);
    NBCS_CUDA_TRY(cudaFuncSetAttribute(ridge_components_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes));
    ridge_components_kernel<<<1, kCompThreads, kBytes, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(pts_out), pt_index, n_out, ny,
        reinterpret_cast<double2*>(comp_pts), head);
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free ridge extraction.
//
// Some callers cannot allocate device memory: a plugin whose host program
// keeps every cudaMalloc to itself (for example inside its time-step loop), or
// a caller that binds this library through a thin FFI and has no device
// allocator of its own.  nbcs_ridge_pts_noalloc gives them ridge extraction
// without a scratch argument: its scratch is the file-scope array below,
// sized for grids of up to NBCS_RIDGE_NOALLOC_MAX_POINTS points (about 8.4 MB,
// held by every GPU that loads the library until the process exits).
//
// The array's name is only a host-side stand-in, so the device address is
// looked up with cudaGetSymbolAddress, once per device, on the first call made
// with that device current (make that first call before any stream capture).
// The address is cached per device ordinal, i.e. for the runtime's primary
// context; it is not refreshed after cudaDeviceReset.
// Every call shares the array and leaves its contents behind; the kernels
// re-initialise everything they read (the selection state, the histograms, the
// barrier and the block counts), and calls whose work overlaps
// on the GPU race on it.

namespace nbcs {

constexpr size_t align256c(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t kNoallocScratchBytes = align256c(sizeof(SelScratch)) +
                                        align256c(sizeof(unsigned int) * kMaxBlocks) +
                                        align256c((size_t)NBCS_RIDGE_NOALLOC_MAX_POINTS);

static __device__ __align__(256) unsigned char g_ridge_noalloc_scratch[kNoallocScratchBytes];

static int noalloc_scratch(void** out)
{
    static std::mutex mu;
    static void* addr[64] = {nullptr};
    int dev = 0;
    NBCS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_error(NBCS_ERR_INVALID, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        NBCS_CUDA_TRY(cudaGetSymbolAddress(&p, g_ridge_noalloc_scratch));
        addr[dev] = p;
    }
    *out = addr[dev];
    return NBCS_OK;
}

}  // namespace nbcs

extern "C" size_t nbcs_ridge_noalloc_scratch_bytes(void) { return nbcs::kNoallocScratchBytes; }

extern "C" int nbcs_ridge_pts_noalloc(const double* f, const double* evec_max, const double* x,
                                      int32_t nx, const double* y, int32_t ny, double sdd_thresh,
                                      double percentile, uint8_t* mask_out, double* rpts_full,
                                      double* pts_out, int64_t* n_out, void* stream)
{
    NBCS_RANGE();
    if (nx < 0 || ny < 0 || (long)nx * ny > NBCS_RIDGE_NOALLOC_MAX_POINTS)
        return set_error(NBCS_ERR_INVALID,
                         "ridge_pts_noalloc: %d x %d grid exceeds the fixed scratch limit of %ld "
                         "points; use nbcs_ridge_pts with caller scratch",
                         nx, ny, (long)NBCS_RIDGE_NOALLOC_MAX_POINTS);
    void* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    return nbcs_ridge_pts(f, evec_max, x, nx, y, ny, sdd_thresh, percentile, mask_out, rpts_full,
                          pts_out, n_out, scratch, kNoallocScratchBytes, stream);
}
