/*
 * Larger eigenvalue and its unit vector of a Cauchy-Green tensor in 64-bit fixed
 * point, from the FP64 gradients of a flow map.  Plain C++ on both sides, so
 * that the host can check it against wider arithmetic.
 *
 * Fixed point holds what is measured against the tensor's largest entry: the
 * diagonal, its difference, the root and the eigenvalue, with errors below 2^-57
 * of that entry (a 53-bit sum's rounding: 2^-53).  The off-diagonal entry keeps
 * its own exponent, as the double that the reference's operations give: the
 * vector's smaller component is a multiple of it, and is as good as it is
 * however far the two columns of the gradient, or its two diagonals, lie apart.
 */
#ifndef NBCS_EIG2_FIXED_H
#define NBCS_EIG2_FIXED_H

#include "intfp64.h"

/* a >> n; 0 for n of 64 and more (as the instruction has it) */
NBCS_IHD ip_u64 ip_shifted_right(ip_u64 a, int n)
{
#ifdef __CUDA_ARCH__
    ip_u64 r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
    return r;
#else
    return n < 64 ? a >> n : 0ull;
#endif
}

/* a b 2^-64 less the low halves' product: at most two units too small */
NBCS_IHD ip_u64 ip_high_product(ip_u64 a, ip_u64 b)
{
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b,
                   bh = (uint32_t)(b >> 32);
    return (ip_u64)ah * bh + (uint32_t)(((ip_u64)al * bh) >> 32) +
           (uint32_t)(((ip_u64)ah * bl) >> 32);
}

/* the square of a below 2^63, the same way */
NBCS_IHD ip_u64 ip_high_square63(ip_u64 a)
{
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32);
    return (ip_u64)ah * ah + (uint32_t)(((ip_u64)ah * al) >> 31);
}

/* Gradients dxdx, dxdy, dydx, dydy -- normal, their exponents within 200 of 0 --
 * and the tensor's off-diagonal entry b (any value, zero too).  The eigenvalue
 * within an ulp, the vector's components within two of their own, apart from
 * what b and the tensor's own roundings bring.  False where the difference of
 * the diagonal and b are both lost in the fixed point (an isotropic tensor).
 *
 * e = lambda - (smaller diagonal entry) = (|a - d| + disc) / 2 with disc^2 =
 * (a - d)^2 + 4 b^2; the vector is along (e, b) (or (b, e)), whose square length
 * is e disc. */
NBCS_IHD bool eig2_max_fixed(double dxdx, double dxdy, double dydx, double dydy, double b,
                             double* lambda, double* vx, double* vy)
{
    const ip_u64 ux = ip_bits(dxdx), uq = ip_bits(dxdy), ur = ip_bits(dydx), us = ip_bits(dydy),
                 ub = ip_bits(b);
    /* in units of 2^(top - 1086), below 2^63 */
    const int e0 = ip_exponent(ux), e1 = ip_exponent(ur), e2 = ip_exponent(uq),
              e3 = ip_exponent(us);
    const int e01 = e0 > e1 ? e0 : e1, e23 = e2 > e3 ? e2 : e3;
    const int top = (e01 > e23 ? e01 : e23) + 1;
    const ip_u64 p = ip_shifted_right(ip_left(ux), top - e0),
                 r = ip_shifted_right(ip_left(ur), top - e1),
                 q = ip_shifted_right(ip_left(uq), top - e2),
                 s = ip_shifted_right(ip_left(us), top - e3);
    /* a, d and |b| in units of 2^(2 top - 2108) */
    const ip_u64 a = ip_high_square63(p) + ip_high_square63(r);
    const ip_u64 d = ip_high_square63(q) + ip_high_square63(s);
    const bool age = a >= d, zero = ip_zero(b);
    const ip_u64 m = age ? a - d : d - a;
    const ip_u64 Mb = ip_left(ub);
    const int sb = 2 * top - 1022 - ip_exponent(ub);
    const ip_u64 b2 = zero ? 0ull : ip_shifted_right(Mb, sb - 1);
    if (!(m | b2) && !zero) return false;
    /* disc 2^(z - 1 + h) = root, h 0 or 1 */
    const int z = ip_clz64(m | b2 | 1ull);
    /* (from b itself: a root and a vector of the same b give a unit vector) */
    const ip_u64 P = m << z, Q = zero ? 0ull : ip_shifted_right(Mb, sb - 1 - z);
    ip_u64 W = ip_high_square63(P >> 1) + ip_high_square63(Q >> 1);
    const int h = (W >> 62) ? 0 : 1;
    W <<= 2 * h;
    const ip_u64 root = ip_root64(W, ip_root_estimate(W));
    const ip_u64 e = (P >> 2) + (root >> (1 + h));  /* e 2^(z - 1) */
    const ip_u64 l = ((age ? d : a) >> 1) + (e >> z);
    /* 1 / sqrt(e disc) = rr 2^(z + h + g - 128) */
    ip_u64 T = ip_high_product(e, root) << h;
    const int g = (T >> 62) ? 0 : 1;
    T <<= 2 * g;
    const ip_u64 rr = ip_rroot64(T, ip_root_estimate(T));
    double major = 1.0, minor = 0.0;
    ip_u64 sign = 0;
    if (!zero) {
        const ip_u64 c = ip_high_product(e, rr) << (h + g);  /* units of 2^-63 */
        major = ip_double(((c + 0x200ull) >> 10) + (1021ull << 52));
        /* 2 |b| 2^z = Mb 2^(z + 1 - sb); t in units of 2^(z + 1 - sb + h + g - 65) */
        ip_u64 t = ip_high_product(Mb, rr);
        const int up = (int)(t >> 63);
        t <<= 1 - up;
        minor = ip_pack(0, (t >> 11) + ((t >> 10) & 1u), 1023 - 2 + z - sb + h + g + up);
        sign = ub & IP_SIGN;
    }
    const ip_u64 x = ip_bits(age ? major : minor), y = ip_bits(age ? minor : major);
    *vx = ip_double(x);
    *vy = ip_double(y | sign);
    const int n = ip_clz64(l);
    const ip_u64 L = l << n;
    *lambda = ip_pack(0, (L >> 11) + ((L >> 10) & 1u), 2 * top - 1021 - n);
    return true;
}

#endif /* NBCS_EIG2_FIXED_H */
