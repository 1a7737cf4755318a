// Correctly rounded square root and divisions that share one reciprocal.
//
// A softened interaction takes sqrt(s), m / sqrt(s), (..) / s twice and 1 / (s s sqrt(s)), each
// rounded as IEEE division and square root round (the reference's).  Evaluated one by one each
// starts from its own reciprocal estimate; here they share the one of 1 / sqrt(s):
//   * y ~ 1/sqrt(s) from a 20-bit estimate by one third-order step (Householder's iteration);
//   * sqrt(s): g = RN(s y), then RN(g + (s - g^2) y / 2);
//   * 1 / b from an approximation y0: RN(y0 + y0 (1 - b y0));
//   * a / b from an approximation y of 1 / b: q = RN(a y), then RN(q + (a - b q) y).
// The steps are those of P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990) 111-119.  His theorem on quotients asks for
// the rounded reciprocal; what is had here after one step is the rounded reciprocal but for a few
// dozen divisors next to a midpoint, so the bounds are proved anew.  Call y "nearly rounded" if
// |y - 1/b| <= (1/2 + 2^-40) ulp(1/b), and let b be scaled to 1 <= b <= 2 - 2^-21 (nb_near_ones
// takes the rest out), d = y - 1/b, so |d| <= (1 + 2^-39) 2^-54; b = 1 is exact throughout.
//   (1) One step from y0 = (1 + e)/b, |e| <= 2^-48, is nearly rounded: before its last rounding
//       it is off by e^2 and the rounding of 1 - b y0, below 2^-95 relative.
//   (2) One step from a nearly rounded y0 is the rounded reciprocal: 1 - b y0 is exact, so the sum
//       before rounding is (1 - e^2)/b with |e| = b|d|, and a midpoint m of doubles lies
//       |1 - b m|/b >= 2^-106/b from 1/b (b m is a multiple of 2^-106 other than 1), farther than
//       e^2/b <= b^2 (1 + 2^-37) 2^-108/b, since b^2 < 4 - 2^-20.
//   (3) A quotient Q = a/b (1 <= a < 2, u = ulp(Q)) from a nearly rounded y is the rounded quotient.
//       The sum before rounding differs from Q by b|Q - q||d|; a midpoint lies at least 2^-53 u/b
//       from Q, as a - b m is a multiple of 2^-53 u other than 0.  If |Q - q| <= (1/2 + 2^-30) u,
//       a - b q is exact and b|Q - q||d| <= b u (1 + 2^-28) 2^-55 is less than that, as b^2 (1 + 2^-28)
//       < 4.  Else no midpoint is within 2^-31 u of Q, and the difference is below 2^-49 u: a
//       midpoint that near would have Q's two neighbours within (1/2 + 2^-31) u, so q would be neither,
//       and |a d| at least u - 2^-31 u (3/4 u - 2^-31 u where Q's lower neighbour is 1; it never is
//       1/2, as Q >= 1/b > 1/2 + 2^-23); but |a d| <= (1 + 2^-39) u/2 for Q >= 1, and for Q < 1, where
//       a < b, |a d| <= (1 - 2^-22)(1 + 2^-39) u.
//   (4) The root: with y = (1 + e)/sqrt(s), |e| <= 1.66 x 2^-53 (the estimate good to 2^-19), 1 <= s <
//       4 and a midpoint m so near that it matters, g is m +- 2^-53 or m +- 3 x 2^-53, and the sum
//       before rounding is off by less than 40 units of 2^-106/(2 sqrt(s)).  s - m^2 is -c x 2^-106 with
//       c = 1 mod 8, so m lies |c| such units away: every s is rounded right but perhaps those with
//       |c| < 40, which are two or fewer for each c: M^2 = c mod 2^54 (s < 2) or 2^55 with M = 2^53 m.
//       tests/test_rdiv.py and tests/test_gpu_exact.py go through all of them.
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

// +0 or -0
NB_RD bool nb_is_zero(double x)
{
#if defined(__CUDA_ARCH__)
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
#else
    return x == 0.0;
#endif
}

// The first 20 bits of the fraction are ones: holds the divisors above 2 - 2^-21 (scaled), for which
// the bounds do not stand, and their squares
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

// The reciprocal of b: nearly rounded from y good to 2^-48 (1), rounded from a nearly rounded y (2).
NB_RD double nb_recip_step(double b, double y) { return fma(y, fma(-b, y, 1.0), y); }

// a / b, rounded, with y the nearly rounded reciprocal of b (3)
NB_RD double nb_quot(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// sqrt(s), rounded, and the nearly rounded reciprocal of that root, from an estimate y0 of
// 1/sqrt(s) good to 2^-19 (4, 1): s and its root's products normal numbers
NB_RD double nb_sqrt_recip(double s, double y0, double& recip)
{
    const double e = fma(-(s * y0), y0, 1.0);
    const double y = fma(y0, e * fma(e, 0.375, 0.5), y0);
    const double g = s * y;
    const double root = fma(fma(-g, g, s), 0.5 * y, g);
    recip = nb_recip_step(root, y);
    return root;
}
