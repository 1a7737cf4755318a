// Correctly rounded square root and divisions that share one reciprocal.
//
// A softened interaction takes sqrt(s), m / sqrt(s), (..) / s twice and 1 / (s s sqrt(s)), each
// rounded as IEEE division and square root round (the reference's).  Evaluated one by one each
// starts from its own reciprocal estimate; here they share the one of 1 / sqrt(s):
//   * y ~ 1/sqrt(s) from a 20-bit estimate by one third-order step (Householder's iteration);
//   * sqrt(s): g = RN(s y), then RN(g + (s - g^2) y / 2), the residual exact in an fma
//     (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
//     processor", IBM J. Res. Dev. 34 (1990) 111-119);
//   * the correctly rounded reciprocal of b from an approximation within an ulp: RN(y + y (1 - b
//     y)) (the same paper's theorem on reciprocals, with the all-ones significand as the
//     exception it names: nb_near_ones);
//   * a / b: q = RN(a y), then RN(q + (a - b q) y): the correctly rounded quotient when y is the
//     correctly rounded reciprocal of b (Markstein's theorem on quotients).
// No step may overflow, underflow or meet a NaN: the callers hold the operands to exponent
// ranges (nb_exp_in) and leave everything else to the IEEE operators.  Only fma, * and integer
// operations appear, so a host build computes what the device computes from the same estimate.
#pragma once

#include <math.h>
#include <string.h>

#if defined(__CUDACC__)
#define NB_RD __host__ __device__ __forceinline__
#else
#define NB_RD static inline
#endif

NB_RD unsigned nb_hi32(double x)
{
#if defined(__CUDA_ARCH__)
    return (unsigned) __double2hiint(x);
#else
    unsigned long long u;
    memcpy(&u, &x, 8);
    return (unsigned) (u >> 32);
#endif
}

// 2^LO <= |x| < 2^HI (false for zeros, infinities and NaN; -1022 <= LO < HI <= 1023)
template <int LO, int HI>
NB_RD bool nb_exp_in(double x)
{
    return (nb_hi32(x) & 0x7fffffffu) - ((unsigned) (LO + 1023) << 20) <
           (unsigned) (HI - LO) << 20;
}

// 2^LO <= x < 2^HI (false also for every negative x)
template <int LO, int HI>
NB_RD bool nb_pos_exp_in(double x)
{
    return nb_hi32(x) - ((unsigned) (LO + 1023) << 20) < (unsigned) (HI - LO) << 20;
}

// The first 20 bits of the significand are ones: a superset of the divisors whose reciprocal
// the step below does not round correctly (and of the squares of such divisors)
NB_RD bool nb_near_ones(double x) { return (nb_hi32(x) & 0xfffffu) == 0xfffffu; }

// 1/sqrt(s) to about 20 bits, s a positive normal number
NB_RD double nb_rsqrt_estimate(double s)
{
#if defined(__CUDA_ARCH__)
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    return y;
#else
    const double y = 1.0 / sqrt(s);
    unsigned long long u;
    memcpy(&u, &y, 8);
    u &= 0xffffffff00000000ull;
    double r;
    memcpy(&r, &u, 8);
    return r;
#endif
}

// The correctly rounded reciprocal of b from y within an ulp of it (one step also brings an
// approximation good to a few ulps within an ulp).
NB_RD double nb_recip_step(double b, double y) { return fma(y, fma(-b, y, 1.0), y); }

// a / b with y the correctly rounded reciprocal of b
NB_RD double nb_quot(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// sqrt(s) and the correctly rounded reciprocal of that root, from an estimate y0 of 1/sqrt(s)
// good to 2^-19: 2^-100 <= s < 2^100
NB_RD double nb_sqrt_recip(double s, double y0, double& recip)
{
    const double e = fma(-(s * y0), y0, 1.0);
    const double y = fma(y0, e * fma(e, 0.375, 0.5), y0);
    const double g = s * y;
    const double root = fma(fma(-g, g, s), 0.5 * y, g);
    recip = nb_recip_step(root, y);
    return root;
}
